"""Which steps launch their kernels to follow one another: not the long
memory-bound ones, nor FP64 grids of one to four blocks an SM."""
import ctypes

import pytest


@pytest.mark.parametrize("size,f64,iord,limited,want", [
    ((24, 24, 24), True, 2, True, True), ((64, 64, 32), True, 2, True, True), ((512, 512, 128), True, 3, True, True),
    ((32, 32, 32), True, 2, True, False),    # 40.4 us plain, 48.7 chained
    ((33, 33, 33), True, 2, True, False),
    ((32, 32, 32), True, 2, False, True), ((32, 32, 32), True, 1, True, True), ((32, 32, 32), False, 2, True, True),
    ((255, 193, 65), False, 1, False, False),  # 51.7 us plain, 59.4 chained
    ((512, 512, 64), False, 2, False, False), ((128, 128, 64), False, 1, False, True)])
def test_chained_where_it_pays(native_lib, size, f64, iord, limited, want):
    n, m, l = size
    f = native_lib["_ZN6mpdata10chain_paysElbibb"]
    f.restype = ctypes.c_bool
    blocks = (n + 31) // 32 * ((m + 3) // 4) * l
    assert f(ctypes.c_long(blocks), ctypes.c_bool(f64), iord, ctypes.c_bool(limited), ctypes.c_bool(False)) == want
    if not f64 and iord > 1:  # the FP32 density step stays chained
        assert f(ctypes.c_long(blocks), ctypes.c_bool(f64), iord, ctypes.c_bool(limited), ctypes.c_bool(True))
