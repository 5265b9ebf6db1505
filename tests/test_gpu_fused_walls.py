"""The fused single-precision step on open and wall axes and in the standard
form, against the FP32 oracle and the stage path, bit for bit, psi's halo
included.

The sizes put the walls everywhere a tile of 64x12 cells and a z chunk can meet
them: inside a tile, on its edge, one column or row past it, tiles
whose boxes come in by TMA between wall tiles, grids of two cells, and z
chunks of one plane.
"""

import numpy as np
import pytest

from advectionhpctester_gb300 import workloads as W
from tests.test_gpu_fused import env

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def M(native_lib):
    from advectionhpctester_gb300 import mpdata
    return mpdata


def gpu(M, f, gauge, iord, steps, **kv):
    d = {k: M.fortran_device(getattr(f, k), dtype=f.dtype) for k in ("x", "u1", "u2", "u3", "h", "rhr", "bcx", "bcy")}
    with env(**kv):
        ws = M.Workspace(f.np, f.mp, f.lp, f.ih, f.ibcx, f.ibcy, f.ibcz, iord=iord, nonos=1, gauge=gauge, precision=32)
    l0 = M.launch_count()
    for _ in range(steps):
        ws.step(d["x"], d["u1"], d["u2"], d["u3"], d["h"], d["rhr"], d["bcx"], d["bcy"])
    launches = M.launch_count() - l0
    out = M.to_numpy(d["x"])
    ws.close()
    return out, launches


def oracle_steps(O, f, gauge, iord, steps):
    g = f.copy()
    O.advec_dwarf(O.grid(g.np, g.mp, g.lp, g.ih, g.ibcx, g.ibcy, g.ibcz), g.x, g.bcx, g.bcy, g.u1, g.u2, g.u3, g.rhr,
                  g.h, legacyoptmode=4, t_adv=1 if gauge else 2, iord=iord, nonos=1, nsteps=steps)
    return g.x


def same_bits(a, b):
    np.testing.assert_array_equal(a.view(np.uint32), b.view(np.uint32))


SIZES = [(200, 96, 24), (33, 17, 9), (37, 23, 5), (64, 12, 3), (65, 13, 2), (129, 25, 3), (127, 24, 2), (2, 2, 2),
         (32, 8, 1)]
BCS = [(0, 0, 0), (0, 1, 1), (1, 0, 1), (1, 1, 0), (1, 1, 1)]


@pytest.mark.parametrize("gauge", [1, 0], ids=["gauge", "std"])
@pytest.mark.parametrize("ibc", BCS, ids=lambda b: "bc%d%d%d" % b)
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "%dx%dx%d" % s)
def test_walls_and_forms(M, oracle, size, ibc, gauge):
    if size[2] < 2 and not ibc[2]:
        pytest.skip("a z wall needs two planes")
    iord = 2 + (size[0] + ibc[0] + gauge) % 3
    f = W.random_fields(*size, ih=1 + ibc[1], ibc=ibc, seed=sum(size) + ibc[2], courant=0.3, dtype=np.float32,
                        sign_change=bool((size[1] + ibc[0]) % 2))
    got, launches = gpu(M, f, gauge, iord, 2)
    assert launches == 2 * (2 * iord - 2)
    same_bits(got, oracle_steps(oracle, f, gauge, iord, 2))


@pytest.mark.parametrize("gauge", [1, 0], ids=["gauge", "std"])
@pytest.mark.parametrize("kchunk", [1, 4])
def test_chunks_meet_walls(M, oracle, kchunk, gauge):
    f = W.random_fields(70, 40, 9, ibc=(0, 0, 0), seed=4, courant=0.3, dtype=np.float32)
    got, _ = gpu(M, f, gauge, 3, 2, MPDATA_FUSED_KCHUNK=kchunk)
    same_bits(got, oracle_steps(oracle, f, gauge, 3, 2))


@pytest.mark.parametrize("gauge", [1, 0], ids=["gauge", "std"])
@pytest.mark.parametrize("ibc", [(0, 0, 0), (1, 1, 1)], ids=["walls", "periodic"])
def test_zeros_and_mixed_density(M, oracle, ibc, gauge):
    """Blocks of +0 and -0 beside a wall, a sign change, and a field of unit
    densities with a perturbed box: the stage path gives the same bits too."""
    f = W.random_fields(104, 56, 12, ibc=ibc, seed=5, courant=0.3, dtype=np.float32)
    x, h, r = W.interior(f.x), W.interior(f.h), W.interior(f.rhr)
    x[:40, 5:30, :7] = 0.0
    x[60:, 20:40, 4:] = -0.0
    x[30:40, 40:50, :] *= -1.0
    keep = h[80:, :30, 6:].copy(), r[80:, :30, 6:].copy()
    h[...], r[...] = 1.0, 1.0
    h[80:, :30, 6:], r[80:, :30, 6:] = keep
    f.bcx[:, :, 0] = 0.0
    got, _ = gpu(M, f, gauge, 3, 2)
    same_bits(got, oracle_steps(oracle, f, gauge, 3, 2))
    same_bits(got, gpu(M, f, gauge, 3, 2, MPDATA_FUSED="0")[0])


def test_batch_of_every_class(M, oracle):
    """One batch with periodic, walled and standard-form problems, two of them
    on one velocity: each as its own step."""
    probs, fields = [], []
    for n, (size, ibc, gauge) in enumerate([((40, 24, 8), (1, 1, 1), 1), ((33, 17, 9), (0, 0, 0), 1),
                                            ((33, 17, 9), (0, 0, 0), 0), ((70, 9, 4), (1, 0, 0), 0)]):
        f = W.random_fields(*size, ibc=ibc, seed=20 + n, courant=0.3, dtype=np.float32)
        if n == 2:  # shares problem 1's velocity and densities
            for k in ("u1", "u2", "u3", "h", "rhr"):
                getattr(f, k)[...] = getattr(fields[1], k)
        fields.append(f)
        probs.append(dict(np=f.np, mp=f.mp, lp=f.lp, ibcx=ibc[0], ibcy=ibc[1], ibcz=ibc[2], gauge=gauge,
                          velocity_group=1 if n == 2 else n))
    b = M.Batch(probs, ih=1, iord=3, nonos=1, precision=32)
    dev = [{k: M.fortran_device(getattr(f, k), dtype=np.float32) for k in
            ("x", "u1", "u2", "u3", "h", "rhr", "bcx", "bcy")} for f in fields]
    for p, d in enumerate(dev):
        v = dev[1] if p == 2 else d
        b.set(p, d["x"], v["u1"], v["u2"], v["u3"], v["h"], v["rhr"], d["bcx"], d["bcy"])
    b.graph(True)
    for _ in range(2):
        b.step()
    for p, f in enumerate(fields):
        same_bits(M.to_numpy(dev[p]["x"]), oracle_steps(oracle, f, probs[p]["gauge"], 3, 2))
    b.close()
