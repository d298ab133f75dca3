"""The each-pair-once force (4th and 6th order, FP64, most particles active)
against the oracle at the sizes where its decomposition changes: the smallest it
takes, one slot past a group (512 / 384), a last group partly active, inactive
particles after the active ones, and several bands of groups.  Relative
tolerance 1e-12 per particle and derivative as tests/test_gpu_parity.py:
summation order only.
"""
import numpy as np
import pytest

from hermite_b200 import Gravity, HermiteError
from inputs import make_records, rel_err

pytestmark = pytest.mark.gpu
EPS2 = (1.0 / 256) ** 2


@pytest.mark.parametrize("order,n,nact", [
    (4, 8193, 8193), (6, 8065, 8065),        # one slot past a group
    (6, 4096, 4096),                         # the smallest
    (4, 16384, 16384), (6, 12289, 12000),
    (4, 15000, 6001), (6, 15000, 6001),      # the smallest active part, ragged
    (4, 40900, 8193), (6, 40900, 8193),      # and of a large system
    (4, 32897, 32897),                       # with the larger scratch
])
def test_pairs_once_against_oracle(order, n, nact, oracle):
    rec = make_records(order, n, seed=71)
    ref = oracle.predict_force(order, rec, 0.0, nact, EPS2)
    with Gravity(order, n) as g:
        g.set_jp_records(rec)
        g.predict_all(0.0)
        got = g.calc_force_on_first_nact(nact, EPS2)
        again = g.calc_force_on_first_nact(nact, EPS2)
        g.set_force_shape(8, 4)              # ordered pairs, everything else alike
        ordered = g.calc_force_on_first_nact(nact, EPS2)
    assert np.array_equal(got, again)
    assert not np.array_equal(got, ordered)  # the other path did run
    assert rel_err(got, ref).max() <= 1e-12


def test_massless_and_coincident_particles():
    """Massless particles pull nobody, and particles at one place (separation
    exactly zero) add nothing to each other."""
    n = 6000
    rec = make_records(6, n, seed=72)
    rec[::7, 3] = 0.0
    rec[1::50] = rec[0]
    with Gravity(6, n) as g:
        g.set_jp_records(rec)
        g.predict_all(0.0)
        got = g.calc_force_on_first_nact(n, EPS2)
        g.set_force_shape(8, 4)
        ordered = g.calc_force_on_first_nact(n, EPS2)
    assert np.all(np.isfinite(got))
    assert rel_err(got, ordered).max() <= 1e-12


def test_wait_timeout(oracle):
    n = 5000
    rec = make_records(6, n, seed=73)
    ref = oracle.predict_force(6, rec, 0.0, n, EPS2)
    with Gravity(6, n) as g:
        g.set_jp_records(rec)
        g.predict_all(0.0)
        g.set_wait_limit(0)
        with pytest.raises(HermiteError) as ei:
            g.calc_force_on_first_nact(n, EPS2)
        assert ei.value.status == 4
        g.set_wait_limit(-1)
        assert rel_err(g.calc_force_on_first_nact(n, EPS2), ref).max() <= 1e-12
