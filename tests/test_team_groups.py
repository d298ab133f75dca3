"""Ensembles on the team engine with team sizes from one CTA to sixteen, their
groups beside one another: a cluster's records are those of the same cluster in
an ensemble of its own, bit for bit, and a block-step budget stops every group.
"""
import numpy as np
import pytest

from hermite_b200 import Ensemble, HermiteError
from hermite_b200.ic import plummer, records

pytestmark = pytest.mark.gpu
SIZES = [40, 384, 385, 1000, 1537, 2700, 5000]


def _run(sizes, seeds, order=4, t=1 / 256, budget=0):
    with Ensemble(order, sizes, "fp64") as e:
        e.set_engine("team")
        for c, (n, s) in enumerate(zip(sizes, seeds)):
            e.set_cluster(c, records(plummer(n, s), order), (4 / n) ** 2)
        e.init(0.0, 0.02, 0.005, t)
        teams = [e.cluster_engine(c) for c in range(len(sizes))]
        if budget:
            with pytest.raises(HermiteError):
                e.run(t, budget)
            return [e.cluster_stats(c) for c in range(len(sizes))]
        e.run(t)
        return teams, [e.get_cluster(c) for c in range(len(sizes))], [e.cluster_stats(c) for c in range(len(sizes))]


def test_groups_match_single_clusters():
    teams, recs, stats = _run(SIZES, range(len(SIZES)))
    assert [t[1] for t in teams] == [1, 1, 2, 3, 5, 8, 14]
    for c, n in enumerate(SIZES):
        _, one, st = _run([n], [c])
        assert np.array_equal(one[0], recs[c]) and st[0] == stats[c], n


def test_budget_stops_every_group():
    for ps, bs, t in _run(SIZES, range(len(SIZES)), budget=3):
        assert bs == 3 and 0 < t < 1 / 256 and ps >= 3
