"""FP64 stage kernels where their dispatch turns, bit for bit against the oracle:
the stored pair sums in the standard form (velocity pairs in the first pass
only) and in every warp, partial ones and those at walls included; unit
densities there and one cell off.  And a step whose chained kernels are captured
into a graph gives a launched step's bits."""
import numpy as np
import pytest

from advectionhpctester_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def M(native_lib):
    from advectionhpctester_gb300 import mpdata
    return mpdata


def fields(n, ibc, density, **kw):
    f = W.random_fields(*n, ibc=ibc, seed=sum(n), courant=0.3, **kw)
    if density != "random":
        f.h[...] = 1.0
        f.rhr[...] = 1.0
        if density == "one_off":
            f.h[n[0] // 2, n[1] // 2, n[2] // 2] = 1.25
    return f


@pytest.mark.parametrize("density", ["random", "unit", "one_off"])
@pytest.mark.parametrize("ibc", [(0, 0, 0), (1, 1, 0), (0, 1, 1), (1, 1, 1)])
@pytest.mark.parametrize("n", [(31, 5, 2), (33, 4, 3), (64, 9, 4), (97, 6, 5)])
@pytest.mark.parametrize("gauge", [1, 0], ids=["gauge", "std"])
def test_pair_sums_in_every_warp(M, oracle, n, ibc, gauge, density):
    iord = 2 + n[0] % 2
    f = fields(n, ibc, density, sign_change=not gauge)
    d = {k: M.fortran_device(getattr(f, k)) for k in ("x", "u1", "u2", "u3", "h", "rhr", "bcx", "bcy")}
    ws = M.Workspace(*n, f.ih, *ibc, iord=iord, nonos=1, gauge=gauge)
    for _ in range(2):
        ws.step(d["x"], d["u1"], d["u2"], d["u3"], d["h"], d["rhr"], d["bcx"], d["bcy"])
    got = M.to_numpy(d["x"])
    ws.close()
    oracle.advec_dwarf(oracle.grid(*n, f.ih, *ibc), f.x, f.bcx, f.bcy, f.u1, f.u2, f.u3, f.rhr, f.h, legacyoptmode=4,
                       t_adv=1 if gauge else 2, iord=iord, nonos=1, nsteps=2)
    np.testing.assert_array_equal(W.interior(got).view(np.uint64), W.interior(f.x).view(np.uint64))


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("gauge", [1, 0], ids=["gauge", "std"])
def test_captured_step(M, gauge, precision):
    import torch
    dt = np.float64 if precision == 64 else np.float32
    f = fields((70, 13, 6), (1, 1, 0), "random")
    d = {k: M.fortran_device(getattr(f, k), dtype=dt) for k in ("x", "u1", "u2", "u3", "h", "rhr", "bcx", "bcy")}
    x0 = d["x"].clone()
    ws = M.Workspace(70, 13, 6, f.ih, 1, 1, 0, iord=3, nonos=1, gauge=gauge, precision=precision)
    step = lambda: ws.step(d["x"], d["u1"], d["u2"], d["u3"], d["h"], d["rhr"], d["bcx"], d["bcy"])
    for _ in range(3):
        step()
    want = d["x"].clone()
    d["x"].copy_(x0)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    d["x"].copy_(x0)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(d["x"], want)
    ws.close()
