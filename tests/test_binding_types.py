"""The Python binding takes `double *` arguments as pointers to doubles and
refuses everything else with an ArgumentError before the library is entered (CPU)."""
import ctypes

import numpy as np
import pytest

import hermite_b200 as hb

DP = ctypes.POINTER(ctypes.c_double)


@pytest.mark.parametrize("bad", [
    1234, "text", b"bytes", ctypes.c_void_p(8), ctypes.byref(ctypes.c_int(3)),
    (ctypes.c_float * 4)(), ctypes.pointer(ctypes.c_longlong(1)),
])
def test_wrong_pointers_are_refused(bad):
    lib = hb.load_library()
    with pytest.raises(ctypes.ArgumentError):
        lib.hb_force_first_nact(None, 1, 0.0, bad)
    with pytest.raises(ctypes.ArgumentError):
        lib.hb_set_jp_records(None, 0, 1, bad)
    with pytest.raises(ctypes.ArgumentError):
        lib.hb_energy(None, 0.0, bad, None)


def test_pointers_to_doubles_are_taken():
    lib = hb.load_library()
    a = np.arange(4.0)
    ro = a.copy()
    ro.flags.writeable = False
    for good in (hb._dptr(a), hb._dptr(ro), hb._dptr(np.empty(0)), hb._dptr(a[::2].copy()),
                 a.ctypes.data_as(DP), (ctypes.c_double * 4)(), ctypes.byref(ctypes.c_double(1.0)), None):
        assert lib.hb_set_jp_records(None, 0, 1, good) == 1      # HB_ERR_INVALID: the null context


def test_pointer_is_the_array():
    a = np.arange(6.0).reshape(2, 3)
    p = ctypes.cast(hb._dptr(a), DP)
    assert ctypes.addressof(p.contents) == a.ctypes.data and p[5] == 5.0
