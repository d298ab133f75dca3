"""calc_force_on_first_nact and force_device + download_forces give the same
bits for the same call: which kernel runs does not depend on where the results
go.  The active counts stand at both sides of 256 KiB of force records (5461 at
4th order, 3640 at 6th, where small results are written straight to the host) and at
the smallest counts that take every pair once.
"""
import numpy as np
import pytest

from hermite_b200 import Gravity
from inputs import make_records

pytestmark = pytest.mark.gpu
EPS2 = (1.0 / 256) ** 2


@pytest.mark.parametrize("order,n,nact", [
    (4, 4096, 4096), (4, 6000, 4095), (4, 6000, 4096), (4, 13000, 5461), (4, 13000, 5462),
    (6, 4096, 3640), (6, 4096, 4096), (8, 4096, 4096), (4, 3000, 20), (6, 3000, 5),
])
def test_same_bits(order, n, nact):
    rec = make_records(order, n, seed=82)
    with Gravity(order, n) as g:
        g.set_jp_records(rec)
        g.predict_all(0.0)
        host = g.calc_force_on_first_nact(nact, EPS2)
        g.force_device(nact, EPS2)
        device = g.download_forces(nact)
    assert np.array_equal(host, device)
