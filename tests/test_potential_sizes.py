"""The potential against the oracle where its decomposition changes: one slice
and several, the first size at which each pair is taken once, one slot past a
group of 1024, a last group of one chunk row, and several bands of groups
(8th order has the widest scratch rows, 4th the narrowest).  Relative tolerance
1e-13 as tests/test_gpu_parity.py: summation order only.
"""
import numpy as np
import pytest

from hermite_b200 import Gravity
from inputs import make_records

pytestmark = pytest.mark.gpu

EPS2 = (1.0 / 256) ** 2


@pytest.mark.parametrize("order,n", [(4, 1), (6, 257), (8, 8191), (9, 3000), (4, 14335), (6, 14336),
                                     (8, 15361), (4, 16640), (6, 20011)])
def test_potential_against_oracle(order, n, oracle):
    rec = make_records(order, n, seed=61)
    ref = oracle.potential(order, rec, EPS2)
    with Gravity(8 if order == 9 else order, n, "dd" if order == 9 else "fp64") as g:
        g.set_jp_records(rec)
        got = g.calc_potential(EPS2)
        again = g.calc_potential(EPS2)
    assert np.array_equal(got, again)
    np.testing.assert_allclose(got, ref, rtol=1e-13, atol=0)


def test_potential_bands():
    """N = 600000 at 4th order: the scratch holds six rows at most, so the
    groups go in about a hundred bands.  Half the mass-weighted sum is the
    potential energy whichever way pairs are taken; rows of the smaller problem
    made of the first slots, the rest massless, must not change."""
    n, k = 600000, 1500
    rec = make_records(4, n, seed=62)
    rec[k:, 3] = 0.0
    with Gravity(4, n) as g:
        g.set_jp_records(rec)
        got = g.calc_potential(EPS2)
    with Gravity(4, k) as g:
        g.set_jp_records(rec[:k])
        small = g.calc_potential(EPS2)
    np.testing.assert_allclose(got[:k], small, rtol=1e-13, atol=0)
    # every other slot against the k massive ones
    d = np.arange(k, n, 7919)
    r2 = ((rec[d, None, 0:3] - rec[None, :k, 0:3]) ** 2).sum(axis=2) + EPS2
    np.testing.assert_allclose(got[d], -(rec[:k, 3] / np.sqrt(r2)).sum(axis=1), rtol=1e-12, atol=0)


@pytest.mark.parametrize("n", [1000, 14336])
def test_potential_without_softening(n, oracle):
    """The self pair is skipped by index, so eps2 = 0 is finite either way."""
    rec = make_records(4, n, seed=63)
    with Gravity(4, n) as g:
        g.set_jp_records(rec)
        got = g.calc_potential(0.0)
    np.testing.assert_allclose(got, oracle.potential(4, rec, 0.0), rtol=1e-13, atol=0)
