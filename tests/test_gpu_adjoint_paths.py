"""The reverse kernels' dispatch at its edges, against the oracle's FP64 AD:
FP32 gathers the pseudo-velocity's reverse where every axis is periodic and
scatters it elsewhere; a cell owns its lower faces in the limiter's and the
upwind's reverse, where the inner face of a z wall counts its wall cell twice
also for a warp away from the wall; blocks pack the cells that the bounds'
reverse works on.

Tolerances: FP64 as test_gpu_adjoint.py (1e-12).  FP32: some hundred roundings
of 2^-24 on each path from an input to a gradient, a few of them amplified by
the differences of neighbouring values (about 0.1 of the values): 1e-4, as the
FP32 tests of one step there."""
import numpy as np
import pytest

from . import test_gpu_adjoint as A
from . import test_gpu_rho_adjoint as RA
from .test_gpu_adjoint import M  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iord", [2, 3])
@pytest.mark.parametrize("n,ibc", [((3, 3, 3), (1, 1, 1)), ((33, 5, 4), (1, 1, 1)), ((70, 10, 8), (1, 1, 1)),
                                   ((70, 10, 8), (1, 1, 0))])
def test_fp32_step_adjoint(M, oracle, n, ibc, iord):
    f, target = A.problem(n, ibc, seed=13 + n[0])
    for k in ("x", "u1", "u2", "u3", "h", "rhr", "bcx", "bcy"):
        setattr(f, k, np.asfortranarray(getattr(f, k).astype(np.float32).astype(np.float64)))
    target = np.asfortranarray(target.astype(np.float32).astype(np.float64))
    _, _, gx, *gu, _ = A.gpu_adjoint_run(M, f, target, 1, iord=iord, precision=32)
    _, _, gxo, *guo = A.oracle_adjoint(oracle, f, target, 1, iord=iord)
    for a, b in zip((gx, *gu), (gxo, *guo)):
        assert A.rel(a.astype(np.float64), b) <= 1e-4


@pytest.mark.parametrize("nonos", [1, 0])
@pytest.mark.parametrize("n", [(80, 10, 3), (96, 6, 5)])
def test_interior_warps_next_to_z_walls(M, oracle, n, nonos):
    f, target = A.problem(n, (1, 0, 0), seed=7)
    _, _, gx, *gu, _ = A.gpu_adjoint_run(M, f, target, 1, nonos=nonos, iord=3)
    _, _, gxo, *guo = A.oracle_adjoint(oracle, f, target, 1, nonos=nonos, iord=3)
    for a, b in zip((gx, *gu), (gxo, *guo)):
        assert A.rel(a, b) <= 1e-12


@pytest.mark.parametrize("ibc", [(1, 1, 1), (0, 0, 0), (1, 1, 0)])
def test_density_step_interior_warps(M, oracle, ibc):
    n = (80, 8, 5)
    sh, f = RA.problem(n, 17 + sum(ibc))
    lam = RA.cotangents(n, sh, 19)
    for a, b in zip(RA.gpu_rho_adjoint(M, n, ibc, f, lam), RA.oracle_rho_adjoint(oracle, n, ibc, f, lam)):
        assert RA.rel(a, b) <= 1e-12


@pytest.mark.parametrize("n,ibc,nsteps,interval", [((12, 10, 8), (0, 0, 0), 5, 2), ((70, 13, 5), (1, 1, 1), 4, 0),
                                                   ((65, 14, 4), (1, 1, 0), 3, 3), ((9, 25, 3), (0, 1, 1), 3, 2)])
def test_fp32_run_records_by_the_fused_kernels(M, n, ibc, nsteps, interval):
    """A run whose interval is above one records its steps by the fused kernels,
    the last segment's as the forward sweep passes it: psi_N has a plain run's
    bits, and the gradients are those of an interval of one, which records by
    the stage kernels (the same records; sums in another order, 1e-5)."""
    f, target = A.problem(n, ibc, seed=23)
    J, xN, gx, *gu, peak = A.gpu_adjoint_run(M, f, target, nsteps, interval=interval, precision=32)
    J1, xN1, gx1, *gu1, _ = A.gpu_adjoint_run(M, f, target, nsteps, interval=1, precision=32)
    np.testing.assert_array_equal(xN, xN1)
    assert J == J1 and peak > 0
    for a, b in zip((gx, *gu[:3]), (gx1, *gu1[:3])):
        assert A.rel(a.astype(np.float64), b.astype(np.float64)) <= 1e-5


@pytest.mark.parametrize("precision", [32, 64])
def test_two_streams_add_to_the_same_gradients(M, precision):
    """Step adjoints on two streams add their dJ/du into one set of arrays: the
    sum of both, whatever the interleaving (rounding of two sums, 1e-5 and 1e-13)."""
    import torch
    dt = np.float32 if precision == 32 else np.float64
    f, _ = A.problem((96, 40, 16), (1, 1, 1), seed=3)
    rng = np.random.default_rng(4)
    d = {k: M.fortran_device(getattr(f, k), dtype=dt) for k in ("x", "u1", "u2", "u3", "h", "rhr", "bcx", "bcy")}
    lams = [np.asfortranarray(rng.uniform(-1, 1, f.x.shape)) for _ in range(2)]
    ws = [M.Workspace(f.np, f.mp, f.lp, f.ih, 1, 1, 1, iord=2, nonos=1, gauge=1, precision=precision) for _ in range(2)]
    zeros = lambda: [torch.zeros_like(d[k]) for k in ("u1", "u2", "u3")]

    def add(w, lam, gu, stream=None):
        l = M.fortran_device(lam, dtype=dt)
        torch.cuda.synchronize()
        for _ in range(8):
            l2 = l.clone()
            torch.cuda.current_stream().synchronize()
            w.step_adjoint(d["x"], d["u1"], d["u2"], d["u3"], d["h"], d["rhr"], l2, *gu, d["bcx"], d["bcy"], stream=stream)
            yield l2

    want = zeros()
    for w, lam in zip(ws, lams):
        keep = list(add(w, lam, want))
    torch.cuda.synchronize()
    got, streams = zeros(), [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    keep = list(zip(add(ws[0], lams[0], got, streams[0].cuda_stream), add(ws[1], lams[1], got, streams[1].cuda_stream)))
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert A.rel(M.to_numpy(a).astype(np.float64), M.to_numpy(b).astype(np.float64)) <= (1e-5 if precision == 32 else 1e-13)
    for w in ws:
        w.close()
