"""Chained and plain launches on one stream: steps of both kinds in turn, without
a wait between them, and a plain upwind step, against the oracle bit for bit."""
import numpy as np
import pytest

from advectionhpctester_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def M(native_lib):
    from advectionhpctester_gb300 import mpdata
    return mpdata


def compare(M, O, f, gauge, iords):
    d = {k: M.fortran_device(getattr(f, k), dtype=f.dtype) for k in ("x", "u1", "u2", "u3", "h", "rhr", "bcx", "bcy")}
    ws = {i: M.Workspace(f.np, f.mp, f.lp, f.ih, f.ibcx, f.ibcy, f.ibcz, iord=i, nonos=int(i > 1), gauge=gauge,
                         precision=64 if f.dtype == np.float64 else 32) for i in set(iords)}
    for i in iords:
        ws[i].step(d["x"], d["u1"], d["u2"], d["u3"], d["h"], d["rhr"], d["bcx"], d["bcy"])
    g = f.copy()
    for i in iords:
        O.advec_dwarf(O.grid(g.np, g.mp, g.lp, g.ih, g.ibcx, g.ibcy, g.ibcz), g.x, g.bcx, g.bcy, g.u1, g.u2, g.u3,
                      g.rhr, g.h, legacyoptmode=4 if i > 1 else 6, t_adv=1 if gauge else 2, iord=i, nonos=1, nsteps=1)
    got, want = W.interior(M.to_numpy(d["x"])), W.interior(g.x)
    for w in ws.values():
        w.close()
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("gauge", [1, 0], ids=["gauge", "std"])
@pytest.mark.parametrize("ibc", [(1, 1, 1), (0, 0, 0)], ids=["periodic", "walls"])
def test_plain_and_chained_steps_in_turn(M, oracle, ibc, gauge):
    f = W.random_fields(32, 32, 32, ibc=ibc, seed=8, courant=0.2)
    compare(M, oracle, f, gauge, [2, 1, 2, 3, 1])  # iord 1 is chained, the others plain


def test_plain_fp32_upwind_step(M, oracle):
    f = W.random_fields(255, 193, 65, ibc=(0, 1, 0), seed=9, courant=0.3, dtype=np.float32)
    compare(M, oracle, f, 1, [1, 1])
