"""The FP32 quotients of the fused step (mpdata_quot32.cuh) against IEEE division,
bit for bit: every significand's reciprocal, quotients beside the middle of two
numbers for every odd divisor, the ends of the ranges the fast path takes; and
fused steps whose operands leave those ranges, so that every branch with the
division itself runs, against the FP32 oracle."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from advectionhpctester_gb300 import build as B
from advectionhpctester_gb300 import workloads as W
from tests.test_gpu_fused_kinds import device, oracle_steps
from tests.test_gpu_fused import env

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def quot(native_lib, tmp_path_factory):
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "quot32_check.cu")
    out = str(tmp_path_factory.mktemp("quot32") / "libquot32.so")
    subprocess.run([B.nvcc(), *B.NVCC_FLAGS, "-shared", src, "-o", out, "-lcudart"], check=True)
    lib = ctypes.CDLL(out)

    def call(name, *args):
        c = (ctypes.c_ulonglong * 2)()
        assert getattr(lib, name)(*args, c) == 0
        return c[0], c[1]

    return call


@pytest.mark.parametrize("e", [0, 1, -33, -60, 59])
def test_every_reciprocal(quot, e):
    assert quot("check_reciprocals", e) == (0, 1 << 23)


@pytest.mark.parametrize("ed,eq", [(0, 0), (-33, 20), (-60, -60), (59, -59), (-2, -122), (5, 55)])
def test_quotients_beside_the_middles(quot, ed, eq):
    taken = 0
    for r in (1, -1, 3, -3, 5, -7, 9, -11):
        wrong, fast = quot("check_middles", r, ed, eq)
        assert wrong == 0, (r, wrong)
        taken += fast
    assert taken > 1 << 22


@pytest.mark.parametrize("n0,n1,d0,d1", [(-30, 30, -30, 30), (-149, -120, -60, 20), (-140, -60, -5, 60),
                                         (-10, 70, -64, -50), (40, 63, -20, 64), (-128, 127, -126, 127)])
def test_ends_of_the_ranges(quot, n0, n1, d0, d1):
    wrong, fast = quot("check_randoms", 1234 + n0, n0, n1, d0, d1)
    assert wrong == 0 and fast > 1 << 16, (wrong, fast)


def scaled(kind, size, ibc):
    """Fields that leave the fast ranges: tiny ones, and densities (with their mass
    fluxes) beyond 2^60 either way in part of the grid."""
    f = W.random_fields(*size, ibc=ibc, seed=31, courant=0.3, dtype=np.float32, sign_change=kind == "tails")
    if kind == "tails":  # magnitudes from 1e-30 down to the smallest subnormals
        e = np.linspace(-45.0, -30.0, size[0])[:, None, None]
        W.interior(f.x)[...] = (W.interior(f.x) * 10.0 ** e).astype(np.float32)
        f.bcx[...] *= np.float32(1e-38)
        f.bcy[...] *= np.float32(1e-38)
    else:  # one power of two for h and u together keeps the Courant numbers
        s = np.float32(2.0) ** (-70 if kind == "thin" else 61)
        if kind == "dense":  # a later pass's velocities are of the size of u*x*rhr: their squares stay finite
            for k in ("x", "bcx", "bcy"):
                getattr(f, k)[...] *= np.float32(2.0) ** -61
        for k in ("u1", "u2", "u3", "h"):
            getattr(f, k)[...] *= s
        W.interior(f.rhr)[:, : size[1] // 2] *= np.float32(2.0) ** (-64 if kind == "thin" else 61)
    return f


@pytest.mark.parametrize("gauge", [1, 0], ids=["gauge", "std"])
@pytest.mark.parametrize("ibc", [(1, 1, 1), (0, 0, 0)], ids=["periodic", "walls"])
@pytest.mark.parametrize("kind", ["tails", "thin", "dense"])
def test_steps_beyond_the_fast_ranges(native_lib, oracle, kind, ibc, gauge):
    from advectionhpctester_gb300 import mpdata as M
    f = scaled(kind, (70, 26, 7), ibc)
    d = device(M, f)
    with env(MPDATA_FUSED="wide"):
        ws = M.Workspace(f.np, f.mp, f.lp, f.ih, *ibc, iord=3, nonos=1, gauge=gauge, precision=32)
    l0 = M.launch_count()
    ws.step(d["x"], d["u1"], d["u2"], d["u3"], d["h"], d["rhr"], d["bcx"], d["bcy"])
    assert M.launch_count() - l0 == 4
    got = W.interior(M.to_numpy(d["x"]))
    ws.close()
    want = oracle_steps(oracle, f, gauge, 3, 1)
    assert np.isfinite(want).all() and (want != 0).any()
    np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
