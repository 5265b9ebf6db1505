"""Performance cases of the MPDATA advection framework.

Each case is one pass of work that a user's program has the library do over
and over: a time step (with or without the velocity predictor), the dwarf
driver, the multi-field step, a batched step, a step adjoint, a whole
checkpointed adjoint run, a density step.  Sizes are this repository's own
configurations (512x512x128, 256x256x64, 64x64x32, 59^3, the uneven domains)
or generic ragged ones.  Velocities are non-divergent under the boundary rule of
the case (the headline flow apart), so a state can be stepped any number of
times.
"""
import math
import random

import torch

from advectionhpctester_gb300 import mpdata

DEV = "cuda"
DTYPE = {64: torch.float64, 32: torch.float32}
EP = 1e-10  # the limiter's and the standard form's guard in the denominators
DOMAINS = ((32, 32, 32), (64, 64, 64), (128, 128, 64), (256, 256, 64), (192, 96, 48))
# the fields of the multi-field step and which of them take the standard form (choice 0)
CE = (("th", 0), ("u", 1), ("v", 1), ("w", 1), ("tht", 1), ("pstr", 1), ("qv", 0), ("qc", 0), ("qr", 0),
      ("qi", 0), ("qs", 0), ("qg", 0))


def listed():
    return [
        # the headline workload: predictor + infinite-gauge iord=3 step of the time loop
        dict(name="headline_f64", kind="step", entry="predictor", nx=512, ny=512, nz=128, bx=1, by=1, bz=1, form="gauge",
             iord=3, prec=64, density="unit", field="noise"),
        # the same loop run in single precision
        dict(name="headline_f32", kind="step", entry="predictor", nx=512, ny=512, nz=128, bx=1, by=1, bz=1, form="gauge",
             iord=3, prec=32, density="unit", field="noise"),
        # the reference's standard form on the CPU-runnable size, through the dwarf driver
        dict(name="dwarf_std_f64_64", kind="step", entry="dwarf", nx=64, ny=64, nz=32, bx=1, by=1, bz=1, form="std",
             iord=2, prec=64, density="unit", field="cone"),
        # the reference's own test set-up: a ball on zeros in an open/wall 59^3 box, gauge form
        dict(name="ball_walls_f64_59", kind="step", entry="dwarf", nx=59, ny=59, nz=59, bx=0, by=0, bz=0, form="gauge",
             iord=2, prec=64, density="unit", field="ball"),
        # a limited-area scalar (standard form) with a varying density, ragged sizes
        dict(name="std_walls_density_f64", kind="step", entry="dwarf", nx=191, ny=157, nz=61, bx=0, by=0, bz=0,
             form="std", iord=2, prec=64, density="variable", field="noise"),
        # a limited-area momentum-like field (gauge form) in single precision, ragged sizes
        dict(name="gauge_walls_f32", kind="step", entry="step", nx=255, ny=193, nz=65, bx=0, by=0, bz=0, form="gauge",
             iord=2, prec=32, density="variable", field="noise"),
        # the dycore's multi-field step: six dry and six moist fields on one velocity
        dict(name="ce_moist_f32", kind="ce", nx=127, ny=95, nz=48, bx=0, by=0, bz=0, prec=32, density="variable",
             nfields=12),
        # an ensemble of 64 small domains of uneven sizes, one graph launch a step
        dict(name="batch_uneven_f32", kind="batch", nprob=64, sizes_seed=7, iord=2, prec=32, form="gauge"),
        # the smallest domain on its own: launch latency
        dict(name="small_f32_32", kind="step", entry="step", nx=32, ny=32, nz=32, bx=1, by=1, bz=1, form="gauge", iord=2,
             prec=32, density="unit", field="cone"),
        # backward: one reverse step of data assimilation
        dict(name="adjoint_f64_256", kind="adjoint", nx=256, ny=256, nz=64, bx=1, by=1, bz=1, form="gauge", iord=2,
             prec=64, density="unit"),
        # a whole forward + backward sweep of an assimilation window, with checkpoints
        dict(name="adjoint_run_f32", kind="adjoint_run", nx=128, ny=128, nz=64, bx=1, by=1, bz=1, form="gauge", iord=2,
             prec=32, density="unit", nsteps=16),
        # the dycore's density step under a rigid lid
        dict(name="density_lid_f64", kind="density", nx=160, ny=129, nz=48, bx=1, by=1, bz=0, iord=2, prec=64),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["ce", "batch", "adjoint", "adjoint_run", "density"])
    prec = rng.choice([64, 32])
    per = dict(bx=1, by=1, bz=1)
    bc = rng.choice([per, per, dict(bx=0, by=0, bz=0), dict(bx=1, by=1, bz=0)])
    if kind == "step":
        form = rng.choice(["gauge", "gauge", "std"])
        iord = rng.choice([2, 2, 3])
        entry = rng.choice(["step", "dwarf", "predictor"])
        field = "noise" if entry == "predictor" else rng.choice(["noise", "cone", "ball"])
        # a drawn step stays below the headline step's cost
        most = 33.5e6 / (1 if form == "gauge" else 2.5)
        while True:
            s = dict(nx=_size(rng, 24, 640), ny=_size(rng, 24, 640), nz=_size(rng, 12, 160))
            if s["nx"] * s["ny"] * s["nz"] < most * 0.5:
                break
        return dict(kind=kind, entry=entry, form=form, iord=iord, prec=prec, field=field,
                    density=rng.choice(["unit", "variable"]), **s, **bc)
    if kind == "ce":
        return dict(kind=kind, nx=_size(rng, 32, 160), ny=_size(rng, 32, 160), nz=_size(rng, 16, 64), prec=prec,
                    density=rng.choice(["unit", "variable"]), nfields=rng.choice([6, 9, 12]), **bc)
    if kind == "batch":
        return dict(kind=kind, nprob=rng.choice([8, 16, 32]), sizes_seed=rng.randrange(1000), iord=rng.choice([2, 3]),
                    prec=prec, form=rng.choice(["gauge", "gauge", "std"]))
    s = dict(nx=_size(rng, 32, 256), ny=_size(rng, 32, 256), nz=_size(rng, 16, 64))
    if kind == "density":
        return dict(kind=kind, prec=prec, iord=2, bx=1, by=1, bz=0, **s)
    form = rng.choice(["gauge", "gauge", "std"])
    if kind == "adjoint":
        return dict(kind=kind, prec=prec, iord=rng.choice([2, 2, 3]), form=form, density=rng.choice(["unit", "variable"]),
                    **s, **bc)
    s = {k: max(24, v // 2) for k, v in s.items()}
    return dict(kind=kind, prec=prec, iord=2, form=form, density="unit", nsteps=rng.choice([4, 7, 9]), **s, **bc)


# ---- inputs: plain tensors in the Fortran layout the library takes ----------------------------


def _fort(shape, dtype):
    """Zeros of a Fortran-ordered shape."""
    return torch.zeros(tuple(reversed(shape)), dtype=dtype, device=DEV).permute(*reversed(range(len(shape))))


def _put(a_kji, shape, dtype, ih=1):
    """The (k, j, i) interior a placed in a Fortran-ordered array with a halo."""
    t = _fort(shape, dtype)
    k, j, i = a_kji.shape
    t.permute(2, 1, 0)[ih:ih + k, ih:ih + j, ih:ih + i] = a_kji
    return t


def _axis(n, dtype=torch.float64):
    return torch.arange(n, dtype=dtype, device=DEV)


def _flow(c, courant):
    """C-grid Courant numbers (k, j, i), faces 1..n+1 of their own axis: an xy
    and an xz stream function, non-divergent under the case's boundary rule (a
    z wall's cells count their inner face twice)."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    sx = torch.sin(math.pi * _axis(nx + 1) / nx) ** 2
    sy = torch.sin(math.pi * _axis(ny + 1) / ny) ** 2
    u1 = (nx * (sy[1:] - sy[:-1])[None, :, None] * sx[None, None, :]).expand(nz, ny, nx + 1).clone()
    u2 = (-nx * sy[None, :, None] * (sx[1:] - sx[:-1])[None, None, :]).expand(nz, ny + 1, nx).clone()
    u3 = torch.zeros(nz + 1, ny, nx, dtype=torch.float64, device=DEV)
    f = _axis(nz + 1)
    if c["bz"]:
        t = torch.sin(2 * math.pi * f / nz)
        du = t[1:] - t[:-1]
    else:
        t = torch.sin(math.pi * (f - 0.5) / max(1, nz - 1))
        t[0] = t[nz] = 0.0
        du = t[1:] - t[:-1]
        du[0], du[-1] = 2 * t[1], -2 * t[nz - 1]
    a = 0.3 * nz
    u1 += a * du[:, None, None] * sx[None, None, :]
    u3 += -a * t[:, None, None] * (sx[1:] - sx[:-1])[None, None, :]
    if not c["bz"]:
        u3[0], u3[nz] = -u3[1], -u3[nz - 1]
    top = (u1.abs().amax() + u2.abs().amax() + u3.abs().amax()).item()
    return [u * (courant / top) for u in (u1, u2, u3)]


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, dtype=torch.float64, device=DEV)


def _field(c, g, what):
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    x, y, z = ((_axis(n) + 0.5) / n for n in (nx, ny, nz))
    ctr = (0.3 + 0.4 * _rand(g, 3)).tolist()
    r2 = (x - ctr[0])[None, None, :] ** 2 + (y - ctr[1])[None, :, None] ** 2 + (z - ctr[2])[:, None, None] ** 2
    if what == "ball":  # a ball of value 4 on an exactly zero background
        return torch.where(r2 <= 0.15 ** 2, 4.0, 0.0).to(torch.float64)
    if what == "cone":  # a Gaussian cone on 1
        return 1.0 + 4.0 * torch.exp(-r2 / (2 * 0.07 ** 2))
    if what == "signed":  # a momentum-like field
        return _rand(g, nz, ny, nx) - 0.5 + torch.exp(-r2 / (2 * 0.1 ** 2))
    if what == "cloud":  # a condensate: zero outside a blob
        return torch.clamp(torch.exp(-r2 / (2 * 0.15 ** 2)) - 0.2, min=0.0)
    return 1.0 + _rand(g, nz, ny, nx) + torch.exp(-r2 / (2 * 0.05 ** 2))


def _density(c, kind):
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    if kind == "unit":
        return torch.ones(nz, ny, nx, dtype=torch.float64, device=DEV)
    x, y, z = ((_axis(n) + 0.5) / n for n in (nx, ny, nz))
    return 1.0 + 0.1 * torch.sin(2 * math.pi * x)[None, None, :] * torch.cos(2 * math.pi * y)[None, :, None] * torch.cos(
        2 * math.pi * z)[:, None, None]


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _shapes(c, ih=1):
    return mpdata.shapes(c["nx"], c["ny"], c["nz"], ih)


def _inputs(c, seed, what="noise", courant=0.4):
    """psi, velocities, densities and halo values of one problem."""
    d, s, g = DTYPE[c["prec"]], _shapes(c), _gen(seed)
    q = {}
    q["psi"] = _put(_field(c, g, what), s["psi"], d)
    for n, u in zip(("u1", "u2", "u3"), _flow(c, courant * (0.9 + 0.1 * _rand(g, 1).item()))):
        q[n] = _put(u, s[n], d)
    var = c.get("density", "unit")
    h = _density(c, var)
    q["h"] = _put(h, s["psi"], d)
    # the ratio of two successive densities: 1 up to the flow's compressibility
    q["rhr"] = _put(1.0 + (1e-6 * (_rand(g, *h.shape) - 0.5) if var == "variable" else 0.0 * h), s["psi"], d)
    for n in ("bcx", "bcy"):
        q[n] = _fort(s[n], d)
        if what not in ("ball", "cloud", "signed"):
            q[n] += 1.0
    return q


def _headline(c, seed):
    """Momentum stacks (level 0 at n, level 2 at n-1) of the flow on the A grid."""
    d, s, g = DTYPE[c["prec"]], _shapes(c), _gen(seed + 1)
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    x, y, z = ((_axis(n) + 0.5) / n for n in (nx, ny, nz))
    if not c["bz"]:
        z = _axis(nz) / max(1, nz - 1)
    amp = 0.4 * (0.9 + 0.1 * _rand(g, 1).item())
    zero = torch.zeros(nz, ny, nx, dtype=torch.float64, device=DEV)
    u = zero + amp * (torch.sin(math.pi * x) ** 2)[None, None, :] * torch.sin(2 * math.pi * y)[None, :, None]
    v = zero - amp * (torch.sin(math.pi * y) ** 2)[None, :, None] * torch.sin(2 * math.pi * x)[None, None, :]
    w = zero + 0.04 * amp * torch.sin(2 * math.pi * z)[:, None, None]
    h = _density(c, c.get("density", "unit"))
    out = {}
    for n, a in zip(("ox", "oy", "oz"), (u, v, w)):
        t = _fort(s["psi"] + (3,), d)
        v4 = t.permute(3, 2, 1, 0)
        v4[0, 1:-1, 1:-1, 1:-1] = a / h
        v4[2, 1:-1, 1:-1, 1:-1] = 0.98 * a
        out[n] = t
    return out


def _density_inputs(c, seed):
    """Momenta and fields of the density step: periodic in x and y, lid and ground in z."""
    d, s, g = DTYPE[c["prec"]], _shapes(c), _gen(seed)
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    a = 0.2 * (0.9 + 0.1 * _rand(g, 1).item())
    px, pz = 2 * math.pi * _axis(nx) / nx, math.pi * _axis(nz) / (nz - 1)
    h = _density(c, "variable")
    zero = torch.zeros(nz, ny, nx, dtype=torch.float64, device=DEV)
    # a roll in xz: u = a sin(x) cos(z), w chosen so that the C-grid divergence vanishes
    u = zero + a * torch.sin(px)[None, None, :] * torch.cos(pz)[:, None, None]
    w = zero - a * math.sin(2 * math.pi / nx) / math.sin(math.pi / (nz - 1)) * torch.cos(px)[None, None, :] * torch.sin(
        pz)[:, None, None]
    v = zero + 0.1 * a * torch.sin(px)[None, None, :]
    top = (u.abs() + v.abs() + w.abs()).amax().item()
    q = {}
    for n, b in zip(("ox", "oy", "oz"), (u, v, w)):
        t = _fort(s["psi"] + (3,), d)
        b = b * (0.35 / top)
        t.permute(3, 2, 1, 0)[0, 1:-1, 1:-1, 1:-1] = b / h
        t.permute(3, 2, 1, 0)[2, 1:-1, 1:-1, 1:-1] = b
        q[n] = t
    x = 1.0 + 0.05 * _rand(g, nz, ny, nx) + 0.1 * torch.cos(px)[None, None, :]
    q["x_in"] = _put(x, s["psi"], d)
    q["x_incomp"] = _put(x * h, s["psi"], d)
    q["h"] = _put(h, s["psi"], d)
    q["pexe"] = _put(1.0 + 0.01 * _rand(g, nz, ny, nx), s["psi"], d)
    for n in ("rhoadv", "rhr", "pexr1", "pexr2"):
        q[n] = _fort(s["psi"], d)
    for n in ("u1", "u2", "u3"):
        q[n] = _fort(s[n], d)
    return q


def _batch_cases(c):
    r = random.Random(c["sizes_seed"])
    return [dict(nx=n[0], ny=n[1], nz=n[2], bx=1, by=1, bz=1, prec=c["prec"], density="unit", form=c["form"],
                 courant=r.uniform(0.2, 0.5)) for n in (r.choice(DOMAINS) for _ in range(c["nprob"]))]


def _ce_inputs(c, seed):
    q = _inputs(c, seed)
    d, s, g = DTYPE[c["prec"]], _shapes(c), _gen(seed + 3)
    fields = {}
    for n, gauge in CE[:c["nfields"]]:
        what = "signed" if n in ("u", "v", "w") else "cloud" if n in ("qc", "qr", "qi", "qs", "qg") else "noise"
        bc = [_fort(s[b], d) + (1.0 if what == "noise" else 0.0) for b in ("bcx", "bcy")]
        fields[n] = (_put(_field(c, g, what), s["psi"], d), bc[0], bc[1])
    return q, fields


def _cotangent(c, seed):
    d, s, g = DTYPE[c["prec"]], _shapes(c), _gen(seed + 5)
    return _put(_rand(g, c["nz"], c["ny"], c["nx"]) - 0.5, s["psi"], d)


# ---- the framework's work ---------------------------------------------------------------------


def _workspace(c, gauge=None):
    return mpdata.Workspace(c["nx"], c["ny"], c["nz"], 1, c["bx"], c["by"], c["bz"], c["iord"], 1,
                            int(c.get("form", "gauge") == "gauge") if gauge is None else gauge, c["prec"])


def prepare(case, seed):
    c, k = case, case["kind"]
    st = dict(c=c)
    if k == "step":
        st.update(_inputs(c, seed, c["field"]))
        if c["entry"] == "predictor":
            st.update(_headline(c, seed))
        if c["entry"] != "dwarf":
            st["ws"] = _workspace(c)
    elif k == "ce":
        st["q"], st["fields"] = _ce_inputs(c, seed)
    elif k == "batch":
        subs = _batch_cases(c)
        st["batch"] = mpdata.Batch([dict(np=p["nx"], mp=p["ny"], lp=p["nz"], gauge=int(c["form"] == "gauge")) for p in subs],
                                   ih=1, iord=c["iord"], nonos=1, precision=c["prec"])
        st["psi"] = []
        for n, p in enumerate(subs):
            q = _inputs(p, seed * 100 + n, "noise", p["courant"])
            st["batch"].set(n, q["psi"], q["u1"], q["u2"], q["u3"], q["h"], q["rhr"], q["bcx"], q["bcy"])
            st["psi"].append(q["psi"])
        st["batch"].graph(True)
    elif k in ("adjoint", "adjoint_run"):
        st.update(_inputs(c, seed))
        st["ws"] = _workspace(c)
        s, d = _shapes(c), DTYPE[c["prec"]]
        for n in ("u1", "u2", "u3"):
            st["g_" + n] = _fort(s[n], d)
        if k == "adjoint":
            st["cot"] = _cotangent(c, seed)
            st["lam"] = _fort(s["psi"], d)
        else:
            st["target"] = _inputs(c, seed + 50)["psi"]
            st["psi0"], st["g_psi0"] = st["psi"], _fort(s["psi"], d)
            st["psi"] = _fort(s["psi"], d)
    else:
        st.update(_density_inputs(c, seed))
        st["ws"] = _workspace(c, 1)
    return st


def run(state):
    s, c = state, state["c"]
    k = c["kind"]
    if k == "step":
        if c["entry"] == "dwarf":
            mpdata.advec_dwarf(4, 1 if c["form"] == "gauge" else 2, False, False, c["nx"], c["ny"], c["nz"], 1, 0, c["bx"],
                               c["by"], c["bz"], s["psi"], s["bcx"], s["bcy"], s["u1"], s["u2"], s["u3"], s["rhr"], s["h"],
                               iord=c["iord"])
            return [s["psi"]]
        if c["entry"] == "predictor":
            s["ws"].velprd(s["ox"], s["oy"], s["oz"], s["h"], 1.0, 1.0, 1.0, 1.0, 1.0, s["u1"], s["u2"], s["u3"])
        s["ws"].step(s["psi"], s["u1"], s["u2"], s["u3"], s["h"], s["rhr"], s["bcx"], s["bcy"])
        if c["entry"] == "predictor":
            return [s["psi"], s["u1"], s["u2"], s["u3"], s["ox"], s["oy"], s["oz"]]
        return [s["psi"]]
    if k == "ce":
        q = s["q"]
        mpdata.ce_advection(0, 0, 0, c["bx"], c["by"], c["bz"], c["nx"], c["ny"], c["nz"], 1, q["rhr"], q["h"], q["u1"],
                            q["u2"], q["u3"], **s["fields"])
        return [f[0] for f in s["fields"].values()]
    if k == "batch":
        s["batch"].step()
        return s["psi"]
    g = [s["g_u1"], s["g_u2"], s["g_u3"]] if "g_u1" in s else None
    if k == "adjoint":
        s["lam"].copy_(s["cot"])
        for t in g:
            t.zero_()
        s["ws"].step_adjoint(s["psi"], s["u1"], s["u2"], s["u3"], s["h"], s["rhr"], s["lam"], *g, s["bcx"], s["bcy"])
        return [s["lam"]] + g
    if k == "adjoint_run":
        s["psi"].copy_(s["psi0"])
        for t in g:
            t.zero_()
        cost, _ = s["ws"].adjoint_run(c["nsteps"], s["psi"], s["u1"], s["u2"], s["u3"], s["h"], s["rhr"], s["target"],
                                      s["g_psi0"], *g, s["bcx"], s["bcy"])
        return [cost, s["psi"], s["g_psi0"]] + g
    s["ws"].rho_gauge(s["ox"], s["oy"], s["oz"], s["u1"], s["u2"], s["u3"], s["x_in"], s["x_incomp"], s["h"], s["rhoadv"],
                      s["rhr"], s["pexe"], s["pexr1"], s["pexr2"], 1.0, 1.0, 1.0, 1.0, 1.0)
    return [s[n] for n in ("x_in", "x_incomp", "rhoadv", "rhr", "pexr1", "pexr2", "u1", "u2", "u3", "ox", "oy", "oz")]


# operations of the formulas per cell: the upwind pass, and one corrective pass of each form
_UP, _PASS = 20, {"gauge": 90, "std": 150}


def work(case):
    c, k = case, case["kind"]
    if k == "batch":
        cells = sum(p["nx"] * p["ny"] * p["nz"] for p in _batch_cases(c))
    else:
        cells = c["nx"] * c["ny"] * c["nz"]
    el = c["prec"] // 8
    ops = _UP + (c.get("iord", 2) - 1) * _PASS[c.get("form", "gauge")]
    # arrays read and written once per cell
    if k == "step":
        arrays = 7 if c["entry"] != "predictor" else 7 + 3 + 6 + 6
    elif k == "ce":
        n = c["nfields"]
        std = sum(1 for _, gauge in CE[:n] if not gauge)
        arrays, ops = 5 + 2 * n, n * _UP + std * _PASS["std"] + (n - std) * _PASS["gauge"]
    elif k == "batch":
        arrays = 7
    elif k == "adjoint":  # psi, u1..3, h, rhr, the cotangent; its result and the gradients
        arrays, ops = 7 + 4, 3 * ops
    elif k == "adjoint_run":
        arrays, ops = 7 + 5, 4 * c["nsteps"] * ops
    else:
        arrays = 6 + 4 + 15
    return {"bytes": float(cells * el * arrays), "flops": float(cells * ops)}


# ---- the same in 64 bits with plain torch (arrays in (k, j, i) order) --------------------------


def _inner(t, ih=1):
    return t.permute(2, 1, 0)[ih:-ih, ih:-ih, ih:-ih].double()


def _pad(x, axis, how):
    """One cell more on both sides of an axis: 1 wraps, "refl" mirrors about the
    first and last cell, "edge" repeats them, "zero" adds zeros."""
    n = x.shape[axis]
    take = lambda a: x.narrow(axis, a, 1)  # noqa: E731
    if how == 1:
        lo, hi = take(n - 1), take(0)
    elif how == "refl":
        lo, hi = take(1), take(n - 2)
    elif how == "edge":
        lo, hi = take(0), take(n - 1)
    else:
        lo = hi = torch.zeros_like(take(0))
    return torch.cat([lo, x, hi], axis)


def _halo(x, c, wall):
    x = _pad(x, 1, 1 if c["by"] else wall)
    x = _pad(x, 2, 1 if c["bx"] else wall)
    return _pad(x, 0, 1 if c["bz"] else "edge")


def _at(x, di, dj, dk):
    """x(i+di, j+dj, k+dk) of a one-cell-padded x."""
    k, j, i = x.shape
    return x[1 + dk:k - 1 + dk, 1 + dj:j - 1 + dj, 1 + di:i - 1 + di]


def _pp(y):
    return torch.where(y > 0, y, torch.zeros_like(y))


def _pn(y):
    return torch.where(y < 0, -y, torch.zeros_like(y))


def _mx(a, b):
    return torch.where(a > b, a, b)


def _mn(a, b):
    return torch.where(a < b, a, b)


def _abs(x):
    return torch.where(torch.signbit(x), -x, x)


def _donor(a, b, u):
    return _pp(u) * a - _pn(u) * b


def _faces(c, caller):
    """Faces 1..n+1 of each axis from the caller's arrays (periodic: n+1 is 1)."""
    out = []
    for ax, per, t in ((2, c["bx"], caller[0]), (1, c["by"], caller[1]), (0, c["bz"], caller[2])):
        f = _inner(t)
        if per:
            f = torch.cat([f.narrow(ax, 0, f.shape[ax] - 1), f.narrow(ax, 0, 1)], ax)
        out.append(f)
    return out


def _face_bc(c, v):
    """Faces 1..n+1 of an antidiffusive field from faces 1..n."""
    out = []
    for ax, per, f in ((2, c["bx"], v[0]), (1, c["by"], v[1]), (0, c["bz"], v[2])):
        n = f.shape[ax]
        if per:
            f = torch.cat([f, f.narrow(ax, 0, 1)], ax)
        elif ax == 0:
            f = torch.cat([-f.narrow(0, 1, 1), f.narrow(0, 1, n - 1), -f.narrow(0, n - 1, 1)], 0)
        else:
            z = torch.zeros_like(f.narrow(ax, 0, 1))
            f = torch.cat([z, f.narrow(ax, 1, n - 1), z], ax)
        out.append(f)
    return out


def _lohi(f, ax):
    n = f.shape[ax] - 1
    return f.narrow(ax, 0, n), f.narrow(ax, 1, n)


def _div(f):
    r = 0
    for ax, g in ((2, f[0]), (1, f[1]), (0, f[2])):
        lo, hi = _lohi(g, ax)
        r = r + (hi - lo)
    return r


def _upwind_fluxes(c, x, u, bcx, bcy):
    """Donor fluxes on faces 1..n+1 with psi's halo rule."""
    if c["bx"]:
        ex = _pad(x, 2, 1)
    else:
        b = bcx.permute(2, 1, 0).double()
        ex = torch.cat([b[0][:, :, None], x, b[1][:, :, None]], 2)
    if c["by"]:
        ey = _pad(x, 1, 1)
    else:
        b = bcy.permute(2, 1, 0).double()
        ey = torch.cat([b[0][:, None, :], x, b[1][:, None, :]], 1)
    ez = _pad(x, 0, 1 if c["bz"] else "edge")
    f = [_donor(e.narrow(ax, 0, n), e.narrow(ax, 1, n), g)
         for ax, e, g, n in ((2, ex, u[0], u[0].shape[2]), (1, ey, u[1], u[1].shape[1]), (0, ez, u[2], u[2].shape[0]))]
    if not c["bz"]:
        n = f[2].shape[0]
        f[2] = torch.cat([-f[2][1:2], f[2][1:n - 1], -f[2][n - 2:n - 1]], 0)
    return f


def _pseudo(c, gauge, x, a, h):
    """Antidiffusive pseudo-velocities on faces 1..n+1 (and, in the standard
    form, their donor fluxes)."""
    X, H = _halo(x, c, "refl"), _halo(h, c, "edge")
    wx, wy, wz = (1 if c[b] else "edge" for b in ("bx", "by", "bz"))
    A = [_pad(_pad(a[0], 1, wy), 0, wz), _pad(_pad(a[1], 2, wx), 0, wz), _pad(_pad(a[2], 2, wx), 1, wy)]
    K, J, I = x.shape

    def fx(f, dj, dk):
        return A[0][1 + dk:1 + dk + K, 1 + dj:1 + dj + J, f:f + I]

    def fy(di, f, dk):
        return A[1][1 + dk:1 + dk + K, f:f + J, 1 + di:1 + di + I]

    def fz(di, dj, f):
        return A[2][f:f + K, 1 + dj:1 + dj + J, 1 + di:1 + di + I]

    s2x = fy(-1, 0, 0) + fy(-1, 1, 0) + fy(0, 0, 0) + fy(0, 1, 0)
    s3x = fz(-1, 0, 0) + fz(-1, 0, 1) + fz(0, 0, 0) + fz(0, 0, 1)
    s1y = fx(0, -1, 0) + fx(1, -1, 0) + fx(0, 0, 0) + fx(1, 0, 0)
    s3y = fz(0, -1, 0) + fz(0, -1, 1) + fz(0, 0, 0) + fz(0, 0, 1)
    s1z = fx(0, 0, -1) + fx(1, 0, -1) + fx(0, 0, 0) + fx(1, 0, 0)
    s2z = fy(0, 0, -1) + fy(0, 1, -1) + fy(0, 0, 0) + fy(0, 1, 0)
    zt = torch.ones(K, 1, 1, dtype=x.dtype, device=x.device)
    if not c["bz"]:
        zt[0] = zt[-1] = 0.0
    own = [fx(0, 0, 0), fy(0, 0, 0), fz(0, 0, 0)]
    ex, ey, ez = (1, 0, 0), (0, 1, 0), (0, 0, 1)
    v = []
    for e, u, crosses in ((ex, own[0], ((ey, s2x, None), (ez, s3x, zt))), (ey, own[1], ((ex, s1y, None), (ez, s3y, zt))),
                          (ez, own[2], ((ex, s1z, None), (ey, s2z, None)))):
        m = tuple(-t for t in e)
        hm = 1.0 / (0.5 * (_at(H, *m) + _at(H, 0, 0, 0)))
        x1, x2 = _at(X, *m), _at(X, 0, 0, 0)
        ka = _abs(u) - u * u * hm
        if gauge:
            w = ka * (x2 - x1) * 0.5
        else:
            w = ka * (_abs(x2) - _abs(x1)) / (_abs(x2) + _abs(x1) + EP)
        for t, s, mask in crosses:
            up = tuple(p + q for p, q in zip(m, t))
            dn = tuple(p - q for p, q in zip(m, t))
            mt = tuple(-q for q in t)
            z3, z2, z1, z0 = _at(X, *t), _at(X, *up), _at(X, *mt), _at(X, *dn)
            if gauge:
                term = 0.125 * u * hm * s * (((z3 + z2) - (z1 + z0)) * 0.25)
            else:
                z3, z2, z1, z0 = _abs(z3), _abs(z2), _abs(z1), _abs(z0)
                term = 0.125 * u * s * ((z3 + z2) - (z1 + z0)) * hm / (z3 + z2 + z1 + z0 + EP)
            w = w - (term if mask is None else term * mask)
        v.append(w)
    v_bc = _face_bc(c, v)
    if gauge:
        return v_bc, v_bc
    m = ((-1, 0, 0), (0, -1, 0), (0, 0, -1))
    return v_bc, _face_bc(c, [_donor(_at(X, *e), _at(X, 0, 0, 0), w) for e, w in zip(m, v)])


def _star(c, X, f, r):
    for di, dj in ((-1, 0), (1, 0), (0, -1), (0, 1), (0, 0)):
        r = _at(X, di, dj, 0) if r is None else f(r, _at(X, di, dj, 0))
    for dk in (-1, 1):  # a z wall's plane repeats its own value: no change
        r = f(r, _at(X, 0, 0, dk))
    return r


def _limit(c, gauge, x, q, v, F, mx, mn, h):
    dp = dn = EP
    for ax, f in ((2, F[0]), (1, F[1]), (0, F[2])):
        lo, hi = _lohi(f, ax)
        dp = dp + _pn(hi) + _pp(lo)
        dn = dn + _pp(hi) + _pn(lo)
    cp, cn = (_halo(t, c, "zero") for t in ((mx - x) * h / dp, (x - mn) * h / dn))
    X, Q = _halo(x, c, "edge"), _halo(q, c, "edge")
    one = torch.ones_like(x)
    w, g = [], []
    for e, ax, f in (((-1, 0, 0), 2, v[0]), ((0, -1, 0), 1, v[1]), ((0, 0, -1), 0, v[2])):
        u = _lohi(f, ax)[0]
        a1 = _mn(_mn(one, _at(cp, 0, 0, 0)), _at(cn, *e))
        a2 = _mn(_mn(one, _at(cp, *e)), _at(cn, 0, 0, 0))
        if gauge:
            w.append(_pp(u) * a1 - _pn(u) * a2)
        else:
            xl, xr = _at(X, *e), _at(X, 0, 0, 0)
            w.append(_pp(u) * torch.where(torch.signbit(xl), a2, a1) - _pn(u) * torch.where(torch.signbit(xr), a1, a2))
            g.append(_donor(_at(Q, *e), _at(Q, 0, 0, 0), w[-1]))
    return _face_bc(c, w), (_face_bc(c, w) if gauge else _face_bc(c, g))


def _step64(c, gauge, iord, x, u, h, rhr, bcx, bcy, rho=False):
    """One step: the new interior, and the upwind and last limited fluxes."""
    f = _upwind_fluxes(c, x, u, bcx, bcy)
    xc = x - _div(f) / h if rho else rhr * (x - _div(f) / h)
    a, mx, mn = u, None, None
    E = _halo(x, c, "edge")
    for p in range(2, iord + 1):
        v, F = _pseudo(c, gauge, xc, a, h)
        if p == 2:
            mx, mn = _star(c, E, _mx, None), _star(c, E, _mn, None)
        X = _halo(xc, c, "refl")
        mx, mn = _star(c, X, _mx, mx), _star(c, X, _mn, mn)
        q = xc if rho else xc / rhr
        w, g = _limit(c, gauge, xc, q, v, F, mx, mn, h)
        xc = q - _div(g) / h
        xc = xc if rho else xc * rhr
        a = w
    return xc, f, a


def _psi_out(c, psi, new):
    """psi's array after a step: the new interior, and on open x and y walls the
    old boundary values in its halo."""
    out = psi.double().clone(memory_format=torch.preserve_format)
    t = out.permute(2, 1, 0)
    if not c["bx"]:
        t[1:-1, 1:-1, 0], t[1:-1, 1:-1, -1] = t[1:-1, 1:-1, 1].clone(), t[1:-1, 1:-1, -2].clone()
    if not c["by"]:
        t[1:-1, 0, 1:-1], t[1:-1, -1, 1:-1] = (psi.permute(2, 1, 0)[1:-1, 1, 1:-1].double(),
                                               psi.permute(2, 1, 0)[1:-1, -2, 1:-1].double())
    t[1:-1, 1:-1, 1:-1] = new
    return out


def _predict64(c, q):
    """The predictor with unit steps: C-grid faces 1..n+1 and the new stacks."""
    h, faces, stacks = _inner(q["h"]), [], []
    for ax, per, n in ((2, c["bx"], "ox"), (1, c["by"], "oy"), (0, c["bz"], "oz")):
        t = q[n].double().clone(memory_format=torch.preserve_format)
        lv = t.permute(3, 2, 1, 0)
        a0, a2 = lv[0, 1:-1, 1:-1, 1:-1] * h, lv[2, 1:-1, 1:-1, 1:-1]
        a = 0.5 * ((a0 + (a0 - a2)) + a0)
        m = a.shape[ax]
        if per:
            e = _pad(a, ax, 1)
        else:
            e = torch.cat([2 * a.narrow(ax, 0, 1) - a.narrow(ax, 1, 1), a,
                           2 * a.narrow(ax, m - 1, 1) - a.narrow(ax, m - 2, 1)], ax)
        f = 0.5 * (e.narrow(ax, 0, m + 1) + e.narrow(ax, 1, m + 1))
        faces.append(f)
        lv[1, 1:-1, 1:-1, 1:-1] = a
        lv[2, 1:-1, 1:-1, 1:-1] = a0
        if not per:  # the extrapolated momenta stand in the stack's halo
            for at, src in ((0, 0), (m + 1, m + 1)):
                lv[1, 1:-1, 1:-1, 1:-1] = a
                idx = [slice(1, -1)] * 3
                idx[ax] = at
                lv[1][tuple(idx)] = e.select(ax, src)
        stacks.append(t)
    return faces, stacks


def _whole(faces, shapes, like):
    return [_put(f, s, torch.float64) for f, s in zip(faces, shapes)]


def exact(case, seed):
    c, k = case, case["kind"]
    s = _shapes(c) if k != "batch" else None
    gauge = c.get("form", "gauge") == "gauge"
    if k == "step":
        q = _inputs(c, seed, c["field"])
        if c["entry"] == "predictor":
            q.update(_headline(c, seed))
            u, stacks = _predict64(c, q)
        else:
            u = _faces(c, (q["u1"], q["u2"], q["u3"]))
        new = _step64(c, gauge, c["iord"], _inner(q["psi"]), u, _inner(q["h"]), _inner(q["rhr"]), q["bcx"], q["bcy"])[0]
        out = [_psi_out(c, q["psi"], new)]
        if c["entry"] == "predictor":
            # the C-grid arrays keep their halo; the stacks' halo on open axes is scratch
            full = _whole(u, (s["u1"], s["u2"], s["u3"]), None)
            out += full + [None if not (c["bx"] and c["by"] and c["bz"]) else t for t in stacks]
        return out
    if k == "ce":
        q, fields = _ce_inputs(c, seed)
        u, h, rhr = _faces(c, (q["u1"], q["u2"], q["u3"])), _inner(q["h"]), _inner(q["rhr"])
        out = []
        for n, g in CE[:c["nfields"]]:
            x, b1, b2 = fields[n]
            out.append(_psi_out(c, x, _step64(c, bool(g), 2, _inner(x), u, h, rhr, b1, b2)[0]))
        return out
    if k == "batch":
        out = []
        for n, p in enumerate(_batch_cases(c)):
            q = _inputs(p, seed * 100 + n, "noise", p["courant"])
            new = _step64(p, gauge, c["iord"], _inner(q["psi"]), _faces(p, (q["u1"], q["u2"], q["u3"])), _inner(q["h"]),
                          _inner(q["rhr"]), q["bcx"], q["bcy"])[0]
            out.append(_psi_out(p, q["psi"], new))
        return out
    if k == "density":
        q = _density_inputs(c, seed)
        u, stacks = _predict64(c, q)
        h, x = _inner(q["h"]), _inner(q["x_in"])
        rhoadv = _inner(q["x_incomp"])
        new, f, w = _step64(c, True, c["iord"], x, u, h, None, None, None, rho=True)
        xc = new * h
        cells = [new, xc, rhoadv, rhoadv / xc, xc * _inner(q["pexe"]), xc]
        out = [_put(t, s["psi"], torch.float64) for t in cells]
        mass = [f[0] + w[0], f[1] + w[1], f[2] + w[2]]
        out += _whole(mass, (s["u1"], s["u2"], s["u3"]), None)
        return out + [stacks[0], stacks[1], None]
    # adjoints: reverse-mode differentiation of the 64-bit step
    q = _inputs(c, seed)
    h, rhr = _inner(q["h"]), _inner(q["rhr"])
    leaf = [t.double().clone(memory_format=torch.preserve_format).requires_grad_() for t in (q["u1"], q["u2"], q["u3"])]

    def back(x, lam):
        x = x.detach().requires_grad_()
        y = _step64(c, gauge, c["iord"], x, _faces(c, leaf), h, rhr, q["bcx"], q["bcy"])[0]
        return torch.autograd.grad(y, [x] + leaf, lam)

    if k == "adjoint":
        cot = _cotangent(c, seed)
        r = back(_inner(q["psi"]), _inner(cot))
        lam = cot.double().clone(memory_format=torch.preserve_format)
        lam.permute(2, 1, 0)[1:-1, 1:-1, 1:-1] = r[0]
        return [lam] + list(r[1:])
    psi, states = q["psi"].double(), []
    with torch.no_grad():
        for _ in range(c["nsteps"]):
            states.append(_inner(psi))
            psi = _psi_out(c, psi, _step64(c, gauge, c["iord"], states[-1], _faces(c, leaf), h, rhr, q["bcx"], q["bcy"])[0])
    lam = _inner(psi) - _inner(_inputs(c, seed + 50)["psi"])
    cost, g = 0.5 * lam.square().sum().item(), [torch.zeros_like(t) for t in leaf]
    for x in reversed(states):
        r = back(x, lam)
        lam = r[0]
        g = [a + b for a, b in zip(g, r[1:])]
    return [cost, psi, _put(lam, s["psi"], torch.float64)] + g
