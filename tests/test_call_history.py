"""A force call's bits are a function of the records, N, the active count and
the context's settings, not of the calls made before it: a call below the size
at which the each-pair-once force makes its larger scratch gives the same bits
before and after one above it.
"""
import numpy as np
import pytest

from hermite_b200 import Gravity
from inputs import make_records

pytestmark = pytest.mark.gpu
EPS2 = (1.0 / 256) ** 2


@pytest.mark.parametrize("order", [4, 6])
def test_large_call_between(order):
    n, nact = 65536, 14000              # each pair once, 0.9e9 pairs of slots
    rec = make_records(order, n, seed=81)
    with Gravity(order, n) as g:
        g.set_jp_records(rec)
        g.predict_all(0.0)
        before = g.calc_force_on_first_nact(nact, EPS2)
        g.calc_force_on_first_nact(n, EPS2)
        after = g.calc_force_on_first_nact(nact, EPS2)
    assert np.array_equal(before, after)
