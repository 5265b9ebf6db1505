"""Which kernels an FP32 step takes and how many planes a block marches: a grid
that fills the 64x12 tiles badly is not sent to them, a list of equal grids counts
rounds of resident blocks."""
import ctypes

import pytest

NONE, PERIODIC, NARROW, WALL, STD = -1, 0, 1, 2, 3
PER, OPEN = (1, 1, 1), (0, 0, 0)


class Geo(ctypes.Structure):
    _fields_ = [(n, ctypes.c_int) for n in ("np", "mp", "lp", "ih", "bx", "by", "bz")]


def geos(sizes, ibc):
    return (Geo * len(sizes))(*[Geo(*s, 1, *ibc) for s in sizes])


def classes(lib, sizes, ibc, gauge):
    n = len(sizes)
    out = (ctypes.c_int * n)()
    f = lib["_ZN6mpdata13fused_classesEPKNS_3GeoEPKiiiiiPNS_10FusedClassE"]
    f.restype = None
    f(geos(sizes, ibc), (ctypes.c_int * n)(*[gauge] * n), n, 32, 1, 2, out)
    return list(out)


@pytest.mark.parametrize("count,size,ibc,gauge,want", [
    (1, (512, 512, 128), PER, 1, PERIODIC),
    (1, (255, 193, 65), PER, 1, PERIODIC),
    (64, (128, 128, 64), PER, 1, PERIODIC),
    (64, (32, 32, 32), PER, 1, NARROW),       # 242 us a step on 64x12 tiles, 117 on narrow ones
    (256, (16, 16, 16), PER, 1, NARROW),      # 349 : 119
    (1, (4, 512, 64), PER, 1, NARROW),        # 130 : 75
    (1, (160, 200, 64), PER, 1, NARROW),      # 139 : 112
    (1, (1, 64, 64), PER, 1, NARROW),         # the wide arena needs two cells an axis
    (1, (255, 193, 65), OPEN, 1, WALL),
    (12, (127, 95, 48), OPEN, 0, STD),
    (1, (2, 2, 2), OPEN, 1, WALL),            # a launch's latency alone: fewer kernels
    (1, (1000, 2, 100), OPEN, 1, NONE),       # 73 : 45 by the stage kernels
    (1, (32, 32, 512), PER, 0, NONE),         # 127 : 90
    (256, (16, 16, 16), OPEN, 1, NONE),       # 394 : 281 by the tile kernels
    (2, (80, 32, 32), OPEN, 1, NONE),         # 60 : 37
])
def test_kernels_by_how_a_grid_fills_their_tiles(native_lib, monkeypatch, count, size, ibc, gauge, want):
    monkeypatch.delenv("MPDATA_FUSED", raising=False)
    assert classes(native_lib, [size] * count, ibc, gauge) == [want] * count


@pytest.mark.parametrize("size,ibc,gauge,want", [
    ((2, 100000, 5000), OPEN, 1, NONE),     # a wide arena of 312 GB, 76 GB of stage scratch
    ((2, 100000, 5000), PER, 1, NARROW),
    ((8, 200000, 300), PER, 0, NONE),
    ((4096, 4096, 100), OPEN, 0, STD)])
def test_an_arena_takes_no_more_than_the_stage_scratch(native_lib, monkeypatch, size, ibc, gauge, want):
    monkeypatch.delenv("MPDATA_FUSED", raising=False)
    assert classes(native_lib, [size], ibc, gauge) == [want]


def test_a_mixed_batch_is_judged_by_all_its_cells(native_lib, monkeypatch):
    """A few narrow domains among large ones share the large ones' launch."""
    monkeypatch.delenv("MPDATA_FUSED", raising=False)
    sizes = [(32, 32, 32)] * 3 + [(256, 256, 64)] * 5
    assert classes(native_lib, sizes, PER, 1) == [PERIODIC] * 8
    assert classes(native_lib, [(32, 32, 32)] * 60 + [(64, 48, 32)], PER, 1) == [NARROW] * 61
    # a row whose tiles a batch's work items cannot name stays on the wide ones
    assert classes(native_lib, [(32 * 65536 + 1, 2, 2)] * 2, PER, 1) == [PERIODIC] * 2


def chunks(lib, sizes, cls, ibc=PER):
    n = len(sizes)
    out = (ctypes.c_int * n)()
    f = lib["_ZN6mpdata12fused_kchunkEPKNS_3GeoEPKNS_10FusedClassEiPi"]
    f.restype = None
    f(geos(sizes, ibc), (ctypes.c_int * n)(*cls), n, out)
    return list(out)


@pytest.mark.parametrize("count,size,cls,want", [
    (1, (128, 128, 64), PERIODIC, 5), (1, (512, 512, 128), PERIODIC, 19),
    (2, (80, 32, 32), WALL, 3),        # 47 us, 61 with the 1 plane of the rule for uneven lists
    (6, (80, 32, 32), PERIODIC, 4),    # 56 : 76
    (24, (48, 48, 48), STD, 16),       # 246 : 303
    (200, (40, 40, 40), PERIODIC, 20),  # 1.02 ms; a long launch keeps the average
    (64, (32, 32, 32), NARROW, 16), (6, (32, 32, 32), NARROW, 3)])
def test_equal_grids_count_rounds(native_lib, monkeypatch, count, size, cls, want):
    monkeypatch.delenv("MPDATA_FUSED_KCHUNK", raising=False)
    assert chunks(native_lib, [size] * count, [cls] * count) == [want] * count


def test_both_forms_on_one_grid_keep_the_average(native_lib, monkeypatch):
    monkeypatch.delenv("MPDATA_FUSED_KCHUNK", raising=False)
    assert chunks(native_lib, [(127, 95, 48)] * 12, [STD] + [WALL] * 5 + [STD] * 6, OPEN) == [8] * 12
