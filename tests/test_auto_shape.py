"""The automatic launch shape (two-warp CTAs, many j-slices, a separate sum of
the slices) against the oracle at the sizes where its tiling changes: one i
past a tile, one chunk, slices that do not divide the chunks, and each shape
(fused up to 3072 slots, narrow up to 64 active particles and for small
problems, wide past them).
Tolerances as tests/test_gpu_parity.py: summation order only in FP64.
"""
import numpy as np
import pytest

from hermite_b200 import Gravity, HermiteError
from inputs import make_records, rel_err

pytestmark = pytest.mark.gpu

EPS2 = (1.0 / 256) ** 2
TOL = {"fp64": [1e-12] * 4, "mixed": [1e-6, 1e-5, 1e-4, 1e-2]}


@pytest.mark.parametrize("order,precision", [(4, "fp64"), (6, "fp64"), (8, "fp64"), (9, "fp64"),
                                             (4, "mixed"), (6, "mixed"), (8, "mixed")])
@pytest.mark.parametrize("n,nacts", [
    (17, [17]),                       # one chunk group, one slice
    (300, [17, 33, 64, 65, 300]),     # fewer chunks than slices are wanted
    (8200, [17, 65, 129, 600]),       # the padded tail in the last slice
    (70000, [31, 64, 65, 700]),       # the wide shape past 64
])
def test_auto_shape_against_oracle(order, precision, n, nacts, oracle):
    rec = make_records(order, n, seed=51)
    with Gravity(8 if order == 9 else order, n, "dd" if order == 9 else precision) as g:
        g.set_jp_records(rec)
        g.predict_all(0.0)
        ref = oracle.predict_force(order, rec, 0.0, max(nacts), EPS2)
        for nact in nacts:
            got = g.calc_force_on_first_nact(nact, EPS2)
            again = g.calc_force_on_first_nact(nact, EPS2)
            assert np.array_equal(got, again), nact
            err = rel_err(got, ref[:nact]).max(axis=0)
            assert np.all(err <= TOL[precision][:err.size]), (nact, err)


@pytest.mark.parametrize("order,precision", [(4, "fp64"), (6, "fp64"), (8, "fp64"), (9, "fp64"),
                                             (4, "mixed"), (6, "mixed"), (8, "mixed")])
@pytest.mark.parametrize("n,nacts", [
    (3072, [17, 100, 3072]),          # the last size that predicts as it streams
    (3073, [17, 65, 3073]),           # the first with a predictor pass
])
def test_fused_edge(order, precision, n, nacts, oracle):
    """FP64 against the oracle; mixed against the tiled kernel in an explicit
    shape, whose FP32 pair sums are the same, so that only the FP64 sums' order
    differs.  (Against the oracle one of 3073 particles is ill-conditioned past
    the mixed tolerance, in every shape alike.)"""
    rec = make_records(order, n, seed=51)
    with Gravity(8 if order == 9 else order, n, "dd" if order == 9 else precision) as g:
        g.set_jp_records(rec)
        g.predict_all(0.0)
        got = {nact: g.calc_force_on_first_nact(nact, EPS2) for nact in nacts}
        g.set_force_shape(0, 1)
        ref = (oracle.predict_force(order, rec, 0.0, n, EPS2) if precision == "fp64"
               else g.calc_force_on_first_nact(n, EPS2))
    for nact, f in got.items():
        assert rel_err(f, ref[:nact]).max() <= 1e-12, nact


def test_auto_shape_wait_timeout(oracle):
    """The bounded waits of a force launch whose slices a second launch adds:
    the call reports the timeout and the context then gives the oracle's
    forces."""
    order, n, nact = 6, 20000, 900
    rec = make_records(order, n, seed=53)
    ref = oracle.predict_force(order, rec, 0.0, nact, EPS2)
    with Gravity(order, n) as g:
        g.set_jp_records(rec)
        g.predict_all(0.0)
        g.set_wait_limit(0)
        with pytest.raises(HermiteError) as ei:
            g.calc_force_on_first_nact(nact, EPS2)
        assert ei.value.status == 4
        g.set_wait_limit(-1)
        got = g.calc_force_on_first_nact(nact, EPS2)
    assert rel_err(got, ref).max() <= 1e-12
