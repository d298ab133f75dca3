"""The potential's self pair is left out by index, in the one chunk of one slice that
holds it, so it does not matter that its separation is zero: without softening
and with, first, last and only chunk, one slice and many, both kinds of positions.
Relative tolerance 1e-13 as tests/test_gpu_parity.py: summation order only.
"""
import numpy as np
import pytest

from hermite_b200 import Gravity
from inputs import make_records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps2", [0.0, (1.0 / 256) ** 2])
@pytest.mark.parametrize("order,n", [(4, 2), (4, 31), (6, 33), (8, 256), (4, 257), (6, 1025), (4, 9001),
                                     (9, 2), (9, 100), (9, 257), (9, 9001)])
def test_against_oracle(order, n, eps2, oracle):
    rec = make_records(order, n, seed=64)
    with Gravity(8 if order == 9 else order, n, "dd" if order == 9 else "fp64") as g:
        g.set_jp_records(rec)
        got = g.calc_potential(eps2)
    assert np.all(np.isfinite(got))
    np.testing.assert_allclose(got, oracle.potential(order, rec, eps2), rtol=1e-13, atol=0)
