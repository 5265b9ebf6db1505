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
