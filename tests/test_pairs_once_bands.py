"""The each-pair-once force finds bands of groups for every scratch it is taken
with: the j-slices' partial sums (2 x 148 x 10 x 256 force records), which smaller
calls use and larger ones where little GPU memory is left, just enough for two
rows, and 512 MiB (CPU)."""
import pytest

import hermite_b200 as hb

SLICES = 2 * 148 * 10 * 256         # force records


@pytest.mark.parametrize("order", [4, 6])
def test_every_scratch_holds_a_band(order):
    bands = hb.load_library().hb_force_pairs_once_bands
    words = 3 * (order // 2)
    for n in [4096, 8192, 12289, 40961, 65536, 131072, 200001, 262144, 300001, 1 << 20, 3 << 20]:
        npad = (n + 127) // 128 * 128
        for nact in sorted({4096, 8192, n // 5 + 1, n // 3, n // 2, n}):
            if nact > n:
                continue
            for cap in (SLICES * words, 2 * npad * words, 3 * npad * words, 64 << 20):
                assert bands(order, n, nact, cap) >= 0, (n, nact, cap)


def test_taken_and_not():
    bands = hb.load_library().hb_force_pairs_once_bands
    assert bands(6, 262144, 262144, SLICES * 9) > bands(6, 262144, 262144, 64 << 20) > 0
    assert bands(6, 262144, 262144, 2 * 262144 * 9 - 1) == 0    # no room for two rows
    assert bands(6, 262144, 40000, 64 << 20) == 0               # too few active
    assert bands(8, 262144, 262144, 64 << 20) == 0
