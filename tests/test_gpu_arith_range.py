"""The kernels' point arithmetic (csrc/p2de_arith.cuh) over its argument ranges, at their
cut-offs and beyond, where CUDA's functions take over.

Reciprocal, root and quotient are held to the bits of the correctly rounded result (NumPy's);
of reciprocals with a mantissa of 53 ones, a tie to 2^-106, to one unit in the last place.
The logarithm is held to 1.5 units (its parts' roundings 0.5 + 0.25 next to 1 and the final
0.5), the exponential to 0.55 (a final rounding and 2^-8 for the reduced argument's), x^y to
0.55 + |y| 2^-7 for |y| < 128 (the logarithm's two parts carry it to 2^-60.5). Where CUDA's functions take
over, their documented bounds of 1 unit, and 2 for pow, hold and the final rounding is added.
The references are long double, 64 or 113 bits.
"""
import ctypes
import importlib.util

import numpy as np
import pytest

import p2de
from p2de import abi, problems
from p2de import solver as S
from p2de.types import ZhangShuLimiter

from conftest import ROOT, relerr
from helpers import setup

pytestmark = pytest.mark.gpu

RCP, SQRT, DIV, LOG, LOG_HALF, EXP, POW = range(7)
RNG_N = 200_000


@pytest.fixture(scope="module")
def arith():
    spec = importlib.util.spec_from_file_location("p2de_build", ROOT / "p2de.jl_gb300" / "build.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    lib = ctypes.CDLL(str(mod.build_probe()))
    P = ctypes.POINTER(ctypes.c_double)
    lib.p2de_probe_arith.argtypes = [ctypes.c_int, ctypes.c_int32, ctypes.c_int64, P, P, P]

    def call(op, a, b=None):
        a = np.ascontiguousarray(a, dtype=np.float64)
        b = a if b is None else np.ascontiguousarray(b, dtype=np.float64)
        out = np.empty_like(a)
        ptr = lambda v: v.ctypes.data_as(P)
        assert lib.p2de_probe_arith(0, op, a.size, ptr(a), ptr(b), ptr(out)) == 0
        return out

    return call


def any_bits(seed, n=RNG_N):
    """Doubles of uniformly random bits (every exponent, both signs)."""
    return np.random.default_rng(seed).integers(0, 2**64, n, dtype=np.uint64).view(np.float64)


def around(*values):
    """The values, their three neighbours on either side, and their negatives."""
    out = []
    for v in values:
        lo = hi = v
        out.append(v)
        for _ in range(3):
            lo, hi = np.nextafter(lo, -np.inf), np.nextafter(hi, np.inf)
            out += [lo, hi]
    out = np.array(out)
    return np.concatenate([out, -out])


SPECIAL = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, np.finfo(float).max, np.finfo(float).tiny])


def ones_mantissa(x):
    return (x.view(np.uint64) & np.uint64(0xFFFFFFFFFFFFF)) == np.uint64(0xFFFFFFFFFFFFF)


def ulps(got, want):
    """Distance in units in the last place of the (long double) wanted values."""
    w = np.abs(want).astype(np.float64)
    return np.abs(got.astype(np.longdouble) - want) / np.spacing(w).astype(np.longdouble)


def test_reciprocal(arith):
    cut = around(*(2.0**e for e in (-1022, -1021, -1020, 0, 1, 1020, 1021, 1022)))
    a = np.concatenate([any_bits(1), 1.0 + np.random.default_rng(2).random(RNG_N), cut, SPECIAL])
    with np.errstate(all="ignore"):
        want = 1.0 / a
    got = arith(RCP, a)
    exact = ~ones_mantissa(a)
    np.testing.assert_array_equal(got[exact], want[exact])
    rest = ~exact & np.isfinite(a)
    assert (np.abs(got[rest] - want[rest]) <= np.spacing(np.abs(want[rest]))).all()


def test_square_root(arith):
    cut = around(*(2.0**e for e in (-901, -900, -899, -1, 0, 1, 2, 899, 900, 901)))
    a = np.concatenate([any_bits(3), 1.0 + 3.0 * np.random.default_rng(4).random(RNG_N), cut, SPECIAL])
    with np.errstate(all="ignore"):
        want = np.sqrt(a)
    np.testing.assert_array_equal(arith(SQRT, a), want)


def test_quotient(arith):
    rng = np.random.default_rng(5)
    cut = np.concatenate([around(*(2.0**e for e in (-256, -255, -254, 0, 254, 255, 256))), SPECIAL,
                          np.array([2.0 - 2.0**-52, 4.0 - 2.0**-51, 0.75])])
    x, y = (v.ravel() for v in np.meshgrid(cut, cut))
    mid = lambda: np.ldexp(1.0 + rng.random(RNG_N), rng.integers(-256, 257, RNG_N)) * rng.choice([-1.0, 1.0], RNG_N)
    a = np.concatenate([any_bits(6), mid(), 1.0 + rng.random(RNG_N), x])
    b = np.concatenate([any_bits(7), mid(), 1.0 + rng.random(RNG_N), y])
    with np.errstate(all="ignore"):
        want = a / b
    got = arith(DIV, a, b)
    np.testing.assert_array_equal(got, want)
    np.testing.assert_array_equal(np.signbit(got[want == 0]), np.signbit(want[want == 0]))


def test_logarithm(arith):
    rng = np.random.default_rng(8)
    table = 1.0 + np.arange(257) / 256.0  # the table's points and the ends of their intervals
    cut = np.abs(around(*np.concatenate([table, table + 1.0 / 512, 0.5 * table, 1.0 + 2.0 ** -np.arange(1.0, 53),
                                         1.0 - 2.0 ** -np.arange(1.0, 53), [2.0**-1022, 2.0**-1021, 2.0**1023]])))
    a = np.concatenate([np.abs(any_bits(9)), np.exp(rng.uniform(-20, 20, RNG_N)), 1.0 + rng.uniform(-0.01, 0.01, RNG_N), cut])
    a = a[np.isfinite(a) & (a > 0)]
    want = np.log(a.astype(np.longdouble))
    some = a != 1.0
    got = arith(LOG, a)
    assert ulps(got[some], want[some]).max() <= 1.5
    assert (got[~some] == 0.0).all()
    normal = a >= 2.0**-1021
    np.testing.assert_array_equal(arith(LOG_HALF, a[normal]), arith(LOG, 0.5 * a[normal]))
    with np.errstate(all="ignore"):
        odd = np.array([0.0, -0.0, -1.0, np.inf, np.nan, -np.inf])
        np.testing.assert_array_equal(arith(LOG, odd), np.log(odd))


def test_exponential(arith):
    rng = np.random.default_rng(10)
    a = np.concatenate([rng.uniform(-699.9, 699.9, RNG_N), rng.uniform(-1, 1, RNG_N), around(1e-300, 2.0**-60, 1e-3),
                        np.arange(-500, 500) * (np.log(2.0) / 128), [0.0, -0.0]])
    assert ulps(arith(EXP, a), np.exp(a.astype(np.longdouble))).max() <= 0.55
    out = np.concatenate([around(700.0), [705.0, -705.0, 709.0]])  # both sides of the cut-off
    assert ulps(arith(EXP, out), np.exp(out.astype(np.longdouble))).max() <= 1.5
    odd = np.array([np.inf, -np.inf, np.nan, 800.0, -800.0])
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(arith(EXP, odd), np.exp(odd))


@pytest.mark.parametrize("y", [1.4, -1.4, 5.0 / 3.0, -5.0 / 3.0, 2.5, 0.4, -3.5, 1.0, 10.0, -100.0, 127.9, -128.0, 1e5])
def test_power(arith, y):
    rng = np.random.default_rng(11)
    span = min(690.0 / abs(y), 700.0)
    cut = np.abs(around(*(1.0 + np.arange(257) / 256.0), 1.0 - 2.0**-53))
    a = np.concatenate([np.exp(rng.uniform(-span, span, RNG_N)), np.exp(rng.uniform(-1.0, 1.0, RNG_N) * min(0.7, span)), cut])
    a = a[np.abs(y * np.log(a)) < 700.0]
    yl = np.longdouble(y)
    got = arith(POW, a, np.full(a.shape, y))
    bound = 0.55 + abs(y) * 2.0**-7 if abs(y) < 128 else 2.5  # pow's beyond
    assert ulps(got, a.astype(np.longdouble) ** yl).max() <= bound
    with np.errstate(over="ignore"):
        edge = np.exp(around(700.0 / abs(y)))  # both sides of the cut-off, where x is in range
    edge = edge[(edge > np.finfo(float).tiny) & np.isfinite(edge)]
    want = edge.astype(np.longdouble) ** yl
    normal = np.abs(want) > np.longdouble(2.0) ** -1022
    if edge.size:
        assert ulps(arith(POW, edge, np.full(edge.shape, y)), want)[normal].max() <= 2.5 + (abs(y) * 2.0**-7 if abs(y) < 128 else 0.0)
    odd = np.array([0.0, -0.0, -1.0, np.inf, np.nan, -np.inf, 5e-324])
    with np.errstate(all="ignore"):
        w = np.power(odd, y)
    got = arith(POW, odd, np.full(odd.shape, y))
    np.testing.assert_allclose(got, w, rtol=1e-15)


# Densities are 2^a and velocities 2^c times those of the first run, pressures 2^(a + 2c): all
# terms but the logarithms scale exactly, so the high-order right-hand side scales by
# 2^(a + c, a + 2c, a + 2c, a + 3c). Neighbouring densities and rho/p differ by 1e-5 (the log
# means' series) or by an eighth and more (their quotients, where the logarithms of up to 360
# are off by 4e-14 at differences of 0.1: 1e-12 with the sums of a line). The outer two leave
# the range in which one reciprocal serves the three quotients.
@pytest.mark.parametrize("form", ["flux", "nodal"])
@pytest.mark.parametrize("N", [1, 3, 5])
@pytest.mark.parametrize("a,c", [(0, 160), (-200, 100), (-260, 260), (260, -260)])
def test_two_point_flux_scales_over_the_range(N, a, c, form):
    # Zhang-Shu's limiter keeps the nodal form, on axis-aligned elements too
    limiter = {} if form == "flux" else dict(rhs_limiter=ZhangShuLimiter())
    param, md, bc, desc, U0 = setup(problems.kelvin_helmholtz, N=N, Kx=4, Ky=3, **limiter)
    rng = np.random.default_rng(N)
    shape = U0.shape[:-1]
    rho = rng.choice([1.0, 2.0, 4.0], shape) * (1.0 + 1e-5 * rng.random(shape))
    p = rng.choice([1.0, 3.0, 9.0], shape) * (1.0 + 1e-5 * rng.random(shape))
    u, v = rng.standard_normal((2, *shape))

    def rhs(a, c):
        U = np.empty_like(U0)
        U[..., 0], U[..., 1], U[..., 2] = rho, rho * u, rho * v
        U[..., 3] = p / 0.4 + 0.5 * rho * (u * u + v * v)
        g = S.Solver(param, md, desc)
        g.set_Uq(U * np.exp2([a, a + c, a + c, a + 2 * c]))
        S.rhs_bang(None, g, None, p2de.TimeParam(0.0, 1e-4 * 2.0**-c, 2))
        out = g.get_field(abi.FIELD_RHSH).reshape(U.shape)
        g.close()
        return out * np.exp2(-np.array([a + c, a + 2.0 * c, a + 2 * c, a + 3 * c]))

    want, got = rhs(0, 0), rhs(a, c)
    for q in range(4):
        assert relerr(got[..., q], want[..., q]) <= 1e-11, q
