"""The graph engine's force phase in each of its shapes (an i-group's warps
sharing every j tile four, two and one ways; one slice and many) against the
team engine, which sums every step in its own order: the same block steps, and
positions, velocities, accelerations and jerks that differ by summation-order
rounding carried over a short run.
"""
import numpy as np
import pytest

import hermite_b200 as hb
from hermite_b200.ic import plummer, records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,n,eta,dtmax", [
    (4, 33, 0.01, 1 / 32),       # two chunks, a single i-tile
    (4, 12001, 0.02, 1 / 256),   # steps from a few to all particles: every shape
    (6, 7000, 0.1, 1 / 128),
    (8, 5000, 0.3, 1 / 64),
])
def test_graph_shapes_against_team(order, n, eta, dtmax):
    out = []
    for engine in ("graph", "team"):
        with hb.Gravity(order, n) as g:
            g.set_engine(engine)
            g.set_jp_records(records(plummer(n, 5), order))
            g.integrator_init(0.0, (4 / n) ** 2, eta, eta / 4, dtmax)
            g.integrator_run(dtmax)
            out.append((g.integrator_stats(), g.get_records()))
    assert out[0][0] == out[1][0]
    a, b = out[0][1][:, :14], out[1][1][:, :14]
    for k in (slice(0, 3), slice(4, 7), slice(8, 11), slice(11, 14)):
        num = np.linalg.norm(a[:, k] - b[:, k], axis=1)
        assert (num <= 1e-9 * np.linalg.norm(b[:, k], axis=1)).all()
