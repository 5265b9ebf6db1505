"""Both kinds of the fused FP32 kernels, 64x12 tiles and narrow ones, on grids
that either may take (MPDATA_FUSED=wide, =narrow), against the FP32 oracle bit
for bit: tiles partly outside the grid, seams inside a tile, axes of one and two
cells, chunk edges, several passes; and a batch that holds narrow, wide and
tile-kernel problems."""
import numpy as np
import pytest

from advectionhpctester_gb300 import workloads as W
from tests.test_gpu_fused import env
from tests.test_gpu_fused_walls import same_bits

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def M(native_lib):
    from advectionhpctester_gb300 import mpdata
    return mpdata


def device(M, f):
    return {k: M.fortran_device(getattr(f, k), dtype=f.dtype) for k in ("x", "u1", "u2", "u3", "h", "rhr", "bcx", "bcy")}


def run(M, f, gauge, iord, steps, **kv):
    d = device(M, f)
    prec = 64 if f.dtype == np.float64 else 32
    with env(**kv):
        ws = M.Workspace(f.np, f.mp, f.lp, f.ih, f.ibcx, f.ibcy, f.ibcz, iord=iord, nonos=int(iord > 1), gauge=gauge,
                         precision=prec)
    l0 = M.launch_count()
    for _ in range(steps):
        ws.step(d["x"], d["u1"], d["u2"], d["u3"], d["h"], d["rhr"], d["bcx"], d["bcy"])
    n = M.launch_count() - l0
    out = M.to_numpy(d["x"])
    viol = ws.bound_violations(d["x"], 1e-6) if iord > 2 else 0
    ws.close()
    return out, n, viol


def oracle_steps(O, f, gauge, iord, steps):
    g = f.copy()
    O.advec_dwarf(O.grid(g.np, g.mp, g.lp, g.ih, g.ibcx, g.ibcy, g.ibcz), g.x, g.bcx, g.bcy, g.u1, g.u2, g.u3, g.rhr,
                  g.h, legacyoptmode=4 if iord > 1 else 6, t_adv=1 if gauge else 2, iord=iord, nonos=1, nsteps=steps)
    return W.interior(g.x)


SIZES = [(37, 23, 9), (5, 3, 2), (33, 9, 4), (64, 16, 3), (65, 17, 2), (31, 8, 5), (2, 40, 6), (100, 25, 7)]


@pytest.mark.parametrize("kind", ["wide", "narrow"])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "%dx%dx%d" % s)
def test_periodic_gauge(M, oracle, size, kind):
    iord = 2 + sum(size) % 3
    f = W.random_fields(*size, ibc=(1, 1, 1), seed=sum(size), courant=0.3, dtype=np.float32,
                        sign_change=bool(size[1] % 2))
    got, n, viol = run(M, f, 1, iord, 2, MPDATA_FUSED=kind)
    assert n == 2 * (2 * iord - 2)
    same_bits(W.interior(got), oracle_steps(oracle, f, 1, iord, 2))
    assert viol == run(M, f, 1, iord, 2, MPDATA_FUSED="0")[2]


@pytest.mark.parametrize("size", [(1, 7, 3), (9, 1, 4), (1, 1, 6)], ids=lambda s: "%dx%dx%d" % s)
def test_one_cell_axes(M, oracle, size):
    """An axis of one cell: narrow tiles alone can take it."""
    f = W.random_fields(*size, ibc=(1, 1, 1), seed=3, courant=0.2, dtype=np.float32)
    got, n, _ = run(M, f, 1, 3, 2)
    assert n == 2 * 4
    same_bits(W.interior(got), oracle_steps(oracle, f, 1, 3, 2))


@pytest.mark.parametrize("kchunk", [1, 4, 64])
def test_narrow_chunks(M, oracle, kchunk):
    f = W.random_fields(40, 24, 21, ibc=(1, 1, 1), seed=11, courant=0.3, dtype=np.float32)
    got, _, _ = run(M, f, 1, 3, 2, MPDATA_FUSED="narrow", MPDATA_FUSED_KCHUNK=kchunk)
    same_bits(W.interior(got), oracle_steps(oracle, f, 1, 3, 2))


def test_batch_of_every_kind(M, oracle):
    """Narrow periodic gauge problems beside walled ones on the tile kernels, then a
    batch whose walled problems stay on the fused kernels."""
    for walled in ((9, 6, 5), (70, 25, 5)):
        cases = [((32, 16, 9), (1, 1, 1), 1), (walled, (0, 0, 0), 1), ((20, 9, 12), (1, 1, 1), 1), (walled, (0, 0, 0), 0)]
        probs, fields, dev = [], [], []
        for n, (size, ibc, gauge) in enumerate(cases):
            f = W.random_fields(*size, ibc=ibc, seed=40 + n, courant=0.3, dtype=np.float32)
            fields.append(f)
            dev.append(device(M, f))
            probs.append(dict(np=f.np, mp=f.mp, lp=f.lp, ibcx=ibc[0], ibcy=ibc[1], ibcz=ibc[2], gauge=gauge))
        b = M.Batch(probs, iord=3, precision=32)
        for p, d in enumerate(dev):
            b.set(p, d["x"], d["u1"], d["u2"], d["u3"], d["h"], d["rhr"], d["bcx"], d["bcy"])
        b.graph(True)
        b.step()
        b.step()
        for p, f in enumerate(fields):
            same_bits(W.interior(M.to_numpy(dev[p]["x"])), oracle_steps(oracle, f, probs[p]["gauge"], 3, 2))
        b.close()


def test_thin_walls_take_the_stage_kernels(M, oracle):
    f = W.random_fields(256, 4, 64, ibc=(0, 0, 0), seed=5, courant=0.3, dtype=np.float32)
    for gauge in (1, 0):
        got, n, _ = run(M, f, gauge, 2, 2)
        assert n == 2 * 5  # upwind, pseudo, bounds, limit, update
        same_bits(W.interior(got), oracle_steps(oracle, f, gauge, 2, 2))


def test_fused_batch_takes_no_velocity_scratch(M):
    """A batch on the fused kernels needs its fields' scratch alone (15 fields each),
    not the tile kernels' velocity terms (4 more)."""
    import torch
    n, m, l = 256, 256, 64
    free0 = torch.cuda.mem_get_info()[0]
    b = M.Batch([dict(np=n, mp=m, lp=l)], iord=2, precision=32)
    fields = (free0 - torch.cuda.mem_get_info()[0]) / (4.0 * n * m * l)
    b.close()
    assert fields < 16.5, fields
