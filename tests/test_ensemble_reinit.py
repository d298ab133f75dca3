"""An ensemble initialised again, with other records, softenings and time, gives what
a fresh one gives, bit for bit: the tables and scheduler state that init uploads
are the ones its kernels read, in the first init and in later ones, on both
engines."""
import numpy as np
import pytest

from hermite_b200 import Ensemble
from hermite_b200.ic import plummer, records

pytestmark = pytest.mark.gpu
SIZES = [40, 300, 700, 1500]


def _set(e, seed, t0):
    for c, n in enumerate(SIZES):
        e.set_cluster(c, records(plummer(n, seed + c), 6), (seed / n) ** 2)
    e.init(t0, 0.1, 0.02, 1 / 64)


@pytest.mark.parametrize("engine", ["team", "graph"])
def test_second_init_matches_fresh(engine):
    def recs(e):
        start = [e.get_cluster(c) for c in range(len(SIZES))]
        e.run(0.5 + 1 / 64)
        ke, pe = e.energy()
        return start + [e.get_cluster(c) for c in range(len(SIZES))] + [ke, pe]

    with Ensemble(6, SIZES, "fp64") as e:
        e.set_engine(engine)
        _set(e, 11, 0.0)
        e.run(1 / 64)
        _set(e, 3, 0.5)
        again = recs(e)
    with Ensemble(6, SIZES, "fp64") as e:
        e.set_engine(engine)
        _set(e, 3, 0.5)
        fresh = recs(e)
    assert all(np.all(r[:, 7] == 0.5) for r in fresh[:len(SIZES)])
    for a, b in zip(again, fresh):
        assert np.array_equal(a, b)
