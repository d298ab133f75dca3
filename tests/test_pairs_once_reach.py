"""The each-pair-once force where its rule and its bands have their edges, with
the path itself asserted: by the rule and the scratch (CPU), and by the launches
of a call (GPU): two for each band, against one for the pairs and one for the sum
of the slices with ordered pairs.

Against the oracle, rows spread over every band of large calls: the oracle's sums
over all particles, with the wanted ones moved to the front.  Relative tolerance
1e-12 per particle and derivative as tests/test_gpu_parity.py: summation order
only (65536 to 262144 terms; the oracle adds them one after another, about
sqrt(n) 2^-53 = 6e-14 of the terms' size).
"""
import numpy as np
import pytest

import hermite_b200 as hb
from hermite_b200 import Gravity
from inputs import make_records, rel_err

EPS2 = (1.0 / 256) ** 2
SLICES = 2 * 148 * 10 * 256         # force records: the scratch of calls below 2^30 pairs
LARGE = 64 << 20                    # doubles: at most this for the others


def padded(n):
    return (n + 255) // 256 * 256


def scratch(order, n, nact):
    words, npad = 3 * (order // 2), padded(n)
    return max(SLICES * words, min(64 * npad * words, LARGE)) if nact * npad >= 1 << 30 else SLICES * words


def bands(order, n, nact, cap=None):
    return hb.load_library().hb_force_pairs_once_bands(order, n, nact,
                                                       scratch(order, n, nact) if cap is None else cap)


def taken(order, n, nact):
    least = 5462 if order == 4 else 4096
    return (nact >= least and nact >= padded(n) * 4 // 10) or (nact >= 8192 and nact >= padded(n) // 5)


@pytest.mark.parametrize("order", [4, 6])
def test_every_scratch_of_two_rows_holds_a_band(order):
    """Taken exactly where the rule says and the scratch has two rows; a band whose
    rows and slice sums left the scratch would give -1."""
    words = 3 * (order // 2)
    seen = 0
    for n in [4096, 5462, 8192, 12289, 15000, 40961, 65536, 131072, 200001, 262144, 300001, 1 << 20, 3 << 20]:
        edges = {4096, 5461, 5462, 8191, 8192, padded(n) * 4 // 10 - 1, padded(n) * 4 // 10, padded(n) // 5 - 1,
                 padded(n) // 5, n // 3, n}
        for nact in sorted(e for e in edges if 1 <= e <= n):
            two = 2 * padded(n) * words
            for cap in (SLICES * words, two - 1, two, 3 * padded(n) * words, LARGE):
                got = bands(order, n, nact, cap)
                if taken(order, n, nact) and cap >= two:
                    assert got > 0, (n, nact, cap)
                    seen += 1
                else:
                    assert got == 0, (n, nact, cap)
    assert seen > 100


LAUNCH_CASES = [(4, 15000, 6041), (6, 15000, 6041),         # 0.4 of the padded slots
                (4, 40900, 8193), (6, 40900, 8193),         # a fifth of them
                (6, 12289, 12000), (4, 32897, 32897)]


@pytest.mark.gpu
@pytest.mark.parametrize("order,n,nact", LAUNCH_CASES)
def test_path_by_launches(order, n, nact, oracle):
    rec = make_records(order, n, seed=74)
    k = bands(order, n, nact)
    assert k >= 2                       # so that its launches are more than the other path's
    ref = oracle.predict_force(order, rec, 0.0, nact, EPS2)
    with Gravity(order, n) as g:
        g.set_jp_records(rec)
        g.predict_all(0.0)
        g.predict_pass()
        before = g.launch_count()
        got = g.calc_force_on_first_nact(nact, EPS2)
        assert g.launch_count() - before == 2 * k
        if padded(n) * 4 // 10 == nact:
            before = g.launch_count()
            g.calc_force_on_first_nact(nact - 1, EPS2)
            assert g.launch_count() - before == 2
    assert rel_err(got, ref).max() <= 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("order,n,nact", [(4, 131072, 131072), (6, 65536, 65536), (6, 131072, 131072),
                                          (6, 131071, 30000), (6, 262144, 262144)])
def test_rows_of_every_band(order, n, nact, oracle):
    rec = make_records(order, n, seed=75)
    group = 32 * (16 if order == 4 else 12)
    last = (nact - 1) // group * group
    rows = np.unique(np.r_[np.linspace(0, nact - 1, 250).astype(int), 0:3, group - 1:group + 1,
                           last - 1:last + 2, nact - 3:nact])
    rest = np.setdiff1d(np.arange(n), rows)
    ref = oracle.predict_force(order, np.ascontiguousarray(rec[np.r_[rows, rest]]), 0.0, rows.size, EPS2)
    with Gravity(order, n) as g:
        g.set_jp_records(rec)
        g.predict_all(0.0)
        g.predict_pass()
        before = g.launch_count()
        got = g.calc_force_on_first_nact(nact, EPS2)
        assert g.launch_count() - before == 2 * bands(order, n, nact)
    assert rel_err(got[rows], ref).max() <= 1e-12
