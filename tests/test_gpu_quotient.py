"""The FP64 quotient on the integer pipe (quot in mpdata_common.cuh) against
IEEE division, bit for bit.

The density step's rhr = rhoadv/x_incomp (mpdata3d-rho-gauge-gpubc.f90:570-609)
with zero momenta and h = 1 is the quotient of two caller arrays, cell by cell:
x_incomp's input over x_in.  The operands cover the places where the long
division can go wrong: significands of all ones, of few leading bits, equal and
almost equal significands, quotients next to the middle of two numbers, the
exponents at both ends of its range, and what leaves it (zeros, subnormals,
infinities, NaN).
"""
import numpy as np
import pytest

from advectionhpctester_gb300 import mpdata as M

pytestmark = pytest.mark.gpu


def operands(kind, n, seed):
    rng = np.random.default_rng(seed)

    def mant(which):
        m = rng.integers(0, 1 << 52, n, dtype=np.int64)
        return {"any": m, "ones": (1 << 52) - 1 - (m & 3), "few": (m & 0x7FFFFF) << 29, "low": m & 7,
                "float_ones": ((m & 0x7FFFFF) << 29) | 0x1FFFFFFF}[which]

    def number(m, lo, hi):
        e = rng.integers(lo, hi + 1, n, dtype=np.int64)
        s = rng.integers(0, 2, n, dtype=np.int64)
        return ((s << 63) | (e << 52) | m).view(np.float64)

    if kind == "significands":
        names = ["any", "ones", "few", "low", "float_ones"]
        a = np.choose(rng.integers(0, 5, n), [mant(k) for k in names])
        b = np.choose(rng.integers(0, 5, n), [mant(k) for k in names])
        near = rng.integers(0, 4, n) == 0
        a = np.where(near, np.clip(b + rng.integers(-2, 3, n), 0, (1 << 52) - 1), a)
        return number(a, 1013, 1033), number(b, 1013, 1033)
    if kind == "middles":  # n = d*(q + half an ulp), rounded and one off
        d = mant("any") | (1 << 52)
        q = 2 * (mant("any") | (1 << 52)) + 1
        p = [int(x) * int(y) for x, y in zip(d, q)]
        off = rng.integers(-1, 2, n)
        a = np.array([(v >> (v.bit_length() - 53)) for v in p], dtype=np.int64) + off
        a = np.clip(a, 1 << 52, (1 << 53) - 1)
        return number(a & ((1 << 52) - 1), 1023, 1023), number(d & ((1 << 52) - 1), 1023, 1023)
    if kind == "range":  # both ends of the exponents it takes itself, and beyond
        e = np.array([1, 2, 522, 523, 524, 1023, 1521, 1522, 1523, 1524, 2045, 2046])
        return (number(mant("any"), 0, 0).view(np.int64) + (rng.choice(e, n) << 52)).view(np.float64), (
            number(mant("any"), 0, 0).view(np.int64) + (rng.choice(e, n) << 52)).view(np.float64)
    a = rng.choice(np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -1e-310, 2.0 ** -1022, 1.0]), n)
    b = rng.choice(np.array([1.0, -3.0, 1e-310, 5e-324, 1e300, -1e-300, 2.0 ** -500, 2.0 ** 501]), n)
    return a, b


@pytest.mark.parametrize("kind", ["significands", "middles", "range", "special"])
def test_quotient_matches_ieee(native_lib, kind):
    import torch
    n = (33, 35, 17)
    a, b = (v.reshape(n, order="F") for v in operands(kind, int(np.prod(n)), 11))
    s = M.shapes(*n, 1)
    z = lambda k: M.fortran_empty(s[k], torch.float64)  # noqa: E731

    def cells(v, fill):
        t = np.full(s["psi"], fill, order="F")
        t[1:-1, 1:-1, 1:-1] = v
        return M.fortran_device(t)

    ws = M.Workspace(*n, 1, 1, 1, 1, iord=2, nonos=1, gauge=1, precision=64)
    stacks = [M.fortran_empty(s["psi"] + (3,), torch.float64) for _ in range(3)]
    x, xi, h, rhr = cells(b, 1.0), cells(a, 1.0), cells(np.ones(n), 1.0), z("psi")
    ws.rho_gauge(*stacks, z("u1"), z("u2"), z("u3"), x, xi, h, z("psi"), rhr, z("psi"), z("psi"), z("psi"),
                 1.0, 1.0, 1.0, 1.0, 1.0, liner=1)
    got = M.to_numpy(rhr)[1:-1, 1:-1, 1:-1]
    ws.close()
    with np.errstate(all="ignore"):
        want = a / b
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got.view(np.int64)[~nan], want.view(np.int64)[~nan])
