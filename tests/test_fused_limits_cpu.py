"""Size limits of the fused FP32 kernels, checked before a call touches the GPU:
the 16-bit tile index of a batch's work items, and the 32-bit plane strides of
the fused arena, whose halo is wider than the caller's; and which problems of a
velocity group are held to one grid."""
import ctypes

import pytest

from advectionhpctester_gb300 import _native

E_DIMS = -1


def create(lib, probs, iord=2, precision=32):
    arr = (_native.MpdataProblem * len(probs))(*[_native.MpdataProblem(*p) for p in probs])
    h = ctypes.c_void_p()
    rc = lib.mpdata_batch_create(len(probs), arr, 1, iord, 1, precision, h)
    if h.value:
        lib.mpdata_batch_destroy(h)
    return rc


@pytest.mark.parametrize("ibc,gauge,most", [((0, 0, 0), 1, 32 * 65536), ((0, 1, 1), 0, 32 * 65536),
                                            ((1, 1, 1), 0, 32 * 65536), ((1, 1, 1), 1, 64 * 65536)])
def test_batch_refuses_rows_beyond_the_tile_index(native_lib, ibc, gauge, most):
    """A row of more tiles than a work item can name is refused, not wrapped
    into the y index; the longest row that fits is not refused for its size."""
    assert create(native_lib, [(most + 1, 2, 2, *ibc, gauge, 0)]) == E_DIMS
    assert create(native_lib, [(most, 2, 2, *ibc, gauge, 0)]) != E_DIMS


@pytest.mark.parametrize("a,b,refused", [
    ((8, 8, 8, 1, 1, 1, 1, 0), (9, 8, 8, 1, 1, 1, 1, 0), True),    # two fields on one velocity
    ((8, 8, 8, 0, 0, 0, 1, 0), (9, 8, 8, 0, 0, 0, 0, 0), True),
    ((8, 8, 8, 1, 1, 1, 1, 0), (9, 8, 8, 1, 1, 1, 0, 0), False),   # periodic gauge fields keep their own
    ((8, 8, 8, 0, 0, 0, 1, 0), (8, 8, 8, 1, 1, 1, 1, 0), False)])
def test_velocity_group_of_periodic_gauge_and_other_problems(native_lib, a, b, refused):
    assert (create(native_lib, [a, b]) == E_DIMS) == refused


class Geo(ctypes.Structure):
    _fields_ = [(n, ctypes.c_int) for n in ("np", "mp", "lp", "ih", "bx", "by", "bz")]


@pytest.mark.parametrize("np_,mp,fits", [(512, 512, True), (300000000, 2, True), (357913932, 2, True),
                                         (357913933, 2, False), (400000000, 2, False)])
def test_arena_planes_stay_below_32_bit_strides(native_lib, np_, mp, fits):
    """Grids whose own planes have 32-bit strides but whose arena planes (rows
    of np+8, mp+4 rows) do not keep the stage kernels."""
    assert (np_ + 3) * (mp + 3) < 1 << 31
    assert ((np_ + 3) // 4 * 4 + 8) * (mp + 4) < 1 << 31 or not fits
    ok = native_lib["_ZN6mpdata14fused_eligibleERKNS_3GeoEiiiii"]
    ok.restype = ctypes.c_bool
    g = Geo(np_, mp, 4, 1, 1, 1, 1)
    assert ok(ctypes.byref(g), 32, 1, 1, 2, 0) == fits
