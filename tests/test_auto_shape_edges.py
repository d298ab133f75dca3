"""The automatic launch shape at the edges of its rule past 3072 slots: 160 active
particles, the last that are predicted as they are streamed, 161, the first with a
predictor pass; one tile and several, slices of one wave; in double-double the
shapes of 64 and 128 particles, at 8th order that of 64 up to 8192 slots.  FP64
against the oracle, mixed against the tiled kernel in an explicit shape, whose FP32
pair sums are the same, so that only the FP64 sums' order differs; 1e-12 as
tests/test_gpu_parity.py.
"""
import numpy as np
import pytest

from hermite_b200 import Gravity
from inputs import make_records, rel_err

pytestmark = pytest.mark.gpu
EPS2 = (1.0 / 256) ** 2
DD = [(9, "fp64", 12000, [1100, 2049, 2200]), (9, "fp64", 33000, [700, 770, 900]),
      (8, "fp64", 8192, [200, 2700, 3200]), (8, "fp64", 8193, [200, 2700])]


@pytest.mark.parametrize("order,precision,n,nacts",
                         [(o, p, n, [1, 17, 32, 33, 160, 161]) for o, p in
                          ((4, "fp64"), (6, "fp64"), (8, "fp64"), (9, "fp64"), (4, "mixed"), (6, "mixed"), (8, "mixed"))
                          for n in (3073, 20000, 140001)] + DD)
def test_edges(order, precision, n, nacts, oracle):
    rec = make_records(order, n, seed=52)
    with Gravity(8 if order == 9 else order, n, "dd" if order == 9 else precision) as g:
        g.set_jp_records(rec)
        g.predict_all(0.0)
        got = {k: g.calc_force_on_first_nact(k, EPS2) for k in nacts}
        again = {k: g.calc_force_on_first_nact(k, EPS2) for k in nacts}
        g.set_force_shape(0, 1)
        ref = (oracle.predict_force(order, rec, 0.0, max(nacts), EPS2) if precision == "fp64"
               else g.calc_force_on_first_nact(max(nacts), EPS2))
    for k in nacts:
        assert np.array_equal(got[k], again[k]), k
        assert rel_err(got[k], ref[:k]).max() <= 1e-12, k
