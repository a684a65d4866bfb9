"""The tensor-core Gram's instruction shapes, decoded on the host: no launch, no GPU."""
import ctypes

import pytest


@pytest.mark.parametrize("m", range(1, 65))
def test_tensor_core_gram_shape_is_defined(ks, m):
    """tcgen05.mma kind::tf32 on one CTA defines N in steps of 16 (16 .. 256) at M = 128, and every block the kernel takes
    (m <= 64) must fit its rows, its TMEM (two slots of N columns per buffer, two buffers at least of 512 columns) and
    the tile (round8(m) rows of S and at least 8 of T)."""
    f = ks.lib()["_ZN2ks13gram_tc_idescEi"]  # ks::gram_tc_idesc(int)
    f.restype, f.argtypes = ctypes.c_uint, [ctypes.c_int]
    d = f(m)
    n, rows = (d >> 17 & 63) * 8, (d >> 24 & 31) * 16
    assert rows == 128 and n % 16 == 0 and 16 <= n <= 256, (n, rows)
    assert m <= n <= (m + 7) // 8 * 8 + 8 and 2 * (2 * n) <= 512
    assert (d >> 4 & 3, d >> 7 & 7, d >> 10 & 7) == (1, 2, 2)  # f32 accumulator, tf32 operands
