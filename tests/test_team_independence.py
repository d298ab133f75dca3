"""A cluster's run on the team engine is a function of that cluster alone: beside
a larger cluster that shares its team size, hence its launch, its records and
steps are those of a run of its own, bit for bit.  The pairs stand where shared
memory decides how many active states a step takes at once: 6th order at 3 CTAs,
8th order at 1 and 3, 4th and 6th at 16, where the larger of the last pair leaves
its records in global memory.
"""
import numpy as np
import pytest

from hermite_b200 import Ensemble
from hermite_b200.ic import plummer, records

pytestmark = pytest.mark.gpu
ETA = {4: 0.02, 6: 0.1, 8: 0.3}


def _run(order, sizes, t=1 / 256):
    with Ensemble(order, sizes, "fp64") as e:
        e.set_engine("team")
        for c, n in enumerate(sizes):
            e.set_cluster(c, records(plummer(n, n), order), (4 / n) ** 2)
        e.init(0.0, ETA[order], ETA[order] / 4, t)
        teams = [e.cluster_engine(c) for c in range(len(sizes))]
        e.run(t)
        return teams, [e.get_cluster(c) for c in range(len(sizes))], [e.cluster_stats(c) for c in range(len(sizes))]


@pytest.mark.parametrize("order,sizes", [
    (6, [850, 1152]), (6, [1000, 1100]), (8, [300, 384]), (8, [850, 1152]),
    (4, [6200, 11000]), (6, [9000, 20000]),
])
def test_same_as_alone(order, sizes):
    teams, recs, stats = _run(order, sizes)
    assert teams[0] == teams[1] and teams[0][0] == "team"
    for c, n in enumerate(sizes):
        _, one, st = _run(order, [n])
        assert np.array_equal(one[0], recs[c]) and st[0] == stats[c], n
