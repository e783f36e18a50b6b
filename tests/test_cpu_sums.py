"""The dot products' sums (skt_sum.hpp, compiled for the host) against exact rational arithmetic: no worse
than FP64 products and FP64 sums over the exponents that FP64 holds and FP32 does not. A warp of 32 lanes
takes 16 terms each, as the kernels do.

Bounds. A warp's total: two roundings to FP64 of the total and one of the FP64 part (2^-51 of the total), and 2^-60 of the
terms' magnitudes for what is rounded below that (the third part's 16 roundings of 2^-24 of some 2^-44 of the
lane's terms, and the cuts' 2^-70). The terms outside FP32's range are summed in FP64, and that sum's own
bound comes on top where there are any: 512 * 2^-53 = 2^-44 of their magnitudes. 32 doubles: one rounding
of the total, and below 2^-51 of the largest value for what is cut off (32 times 2^-57 of it, twice that
for the value's own place below its power of two, and 2^-52 for the last five bits)."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from skewtcloudsim_gb300 import build

SOURCE = r"""
#include "skt_sum.hpp"
using namespace skt;
static double warp(Sum* v, bool third) {
    unsigned top = 0;
    for (int i = 0; i < 32; ++i) {
        if (third) normalise<true>(v[i]); else normalise<false>(v[i]);
        const unsigned m = float_bits(v[i].h) & 0x7fffffffu;
        top = m > top ? m : top;
    }
    WarpSum w{0, 0, 0, (top >> 23) > 48u ? top >> 23 : 48u};
    double far = 0.0;
    for (int i = 0; i < 32; ++i) {
        far += v[i].far;
        if (w.e == 255u) continue;
        int a, b, c;
        if (third) cut<true>(v[i], w.e, a, b, c); else cut<false>(v[i], w.e, a, b, c);
        if (__builtin_add_overflow(w.a, a, &w.a) || __builtin_add_overflow(w.b, b, &w.b) || __builtin_add_overflow(w.c, c, &w.c)) return NAN;
    }
    return value(fixed_of(w)) + far;
}
extern "C" float quot(double a, double b) { return quotient(a, b); }
static Fixed lanes_fixed(const double* d) {  // the total of 32 doubles
    Fixed f[32];
    int u = -2048, hi = 0, mid = 0, lo = 0;
    for (int i = 0; i < 32; ++i) {
        f[i] = fixed_of(d[i]);
        if ((f[i].v || f[i].u == kNotFinite) && f[i].u > u) u = f[i].u;
    }
    for (int i = 0; i < 32; ++i) {
        int a, b, c;
        if (!f[i].v && f[i].u != kNotFinite) continue;
        split(f[i], u, a, b, c);
        if (__builtin_add_overflow(hi, a, &hi) || __builtin_add_overflow(mid, b, &mid) || __builtin_add_overflow(lo, c, &lo)) return Fixed{0, 4096};
    }
    return joined<5>(hi, mid, lo, u);
}
extern "C" double lanes(const double* d) { return value(lanes_fixed(d)); }
extern "C" int unit(const double* d) { return lanes_fixed(d).u; }
extern "C" double dot(const float* a, const float* b, int n) {
    Sum v[32];
    for (int i = 0; i < n; ++i) v[i % 32].add_prod(a[i], b[i]);
    return warp(v, true);
}
extern "C" int holds(double t) { return Sum::total_holds(t); }
extern "C" double dot16(const float* a, const float* b, int how) {  // the same 512 terms, a lane's 16 at a time
    Sum v[32];
    for (int i = 0; i < 32; ++i) {
        float x[16], y[16];
        for (int j = 0; j < 16; ++j) {
            x[j] = a[i + 32 * j];
            y[j] = b[i + 32 * j];
        }
        if (how == 0) v[i].add_prods(x, y);
        else if (how == 1) v[i].add_near(x, y);
        else v[i].add_far(x, y);
    }
    return warp(v, true);
}
extern "C" double total(const float* s, const float* c) {  // of 32 running sums with their compensations
    Sum v[32];
    for (int i = 0; i < 32; ++i) v[i] = sum_of(s[i], c[i]);
    return warp(v, false);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("sums")
    (d / "sums.cpp").write_text(SOURCE)
    so = str(d / "sums.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", build.CSRC, str(d / "sums.cpp"), "-o", so], check=True)
    lb = ctypes.CDLL(so)
    p = ctypes.POINTER(ctypes.c_float)
    lb.dot.restype = lb.dot16.restype = lb.total.restype = ctypes.c_double
    lb.dot16.argtypes = [p, p, ctypes.c_int]
    lb.holds.argtypes = [ctypes.c_double]
    lb.quot.restype = ctypes.c_float
    lb.quot.argtypes = [ctypes.c_double, ctypes.c_double]
    lb.lanes.restype = ctypes.c_double
    lb.unit.argtypes = [ctypes.POINTER(ctypes.c_double)]
    lb.lanes.argtypes = [ctypes.POINTER(ctypes.c_double)]
    lb.dot.argtypes = [p, p, ctypes.c_int]
    lb.total.argtypes = [p, p]
    return lb


def _ptr(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_float))


def _terms(rng, kind, n=512):
    a, b = rng.standard_normal(n), rng.standard_normal(n)
    scale = {"one": 0, "tiny": -70, "huge": 62, "edge": -50, "denormal": -120}.get(kind, 0)
    if kind == "residual":   # z.r: all of one sign, over many decades, with zeros
        b = a * 10.0 ** rng.uniform(-6, 0, n)
        a = b * 0.2
        a[::7] = 0.0
    if kind == "spread":     # products from far below FP32's range to far above it
        a, b = a * 2.0 ** rng.integers(-140, 100, n), b * 2.0 ** rng.integers(-140, 100, n)
    if kind == "cancel":     # sums that cancel to their last bits
        a[1::2], b[1::2] = -a[::2], b[::2] * (1 + 2.0 ** -23 * rng.integers(-1, 2, n // 2))
    if kind == "gone":       # lanes whose leading parts cancel exactly
        a[256:], b[256:] = -a[:256], b[:256]
        a[64:96], b[64:96] = 2.0 ** -30, 2.0 ** -20
    return (a * 2.0 ** scale).astype(np.float32), (b * 2.0 ** (scale if kind != "denormal" else 0)).astype(np.float32)


@pytest.mark.parametrize("kind", ["one", "residual", "cancel", "gone", "tiny", "huge", "edge", "denormal", "spread"])
@pytest.mark.parametrize("seed", range(8))
def test_dot_is_no_worse_than_fp64(lib, kind, seed):
    rng = np.random.default_rng(seed)
    a, b = _terms(rng, kind)
    prods = [Fraction(float(x)) * Fraction(float(y)) for x, y in zip(a, b)]
    exact, size = sum(prods), sum(abs(p) for p in prods)
    got = lib.dot(_ptr(a), _ptr(b), a.size)
    assert np.isfinite(got)
    far = sum(abs(p) for p in prods if not 2.0 ** -98 <= abs(p) < 2.0 ** 100)  # (one bit of slack for the rounded product)
    assert abs(Fraction(got) - exact) <= abs(exact) / 2 ** 51 + size / 2 ** 60 + far / 2 ** 44, (kind, seed, got, float(exact))


def test_far_products_against_fp64(lib):
    """Terms that the FP64 sum takes: as far off as FP64 is, and what is not finite stays so."""
    a = np.full(512, 1e25, np.float32)
    assert abs(lib.dot(_ptr(a), _ptr(a), 512) / (512 * float(a[0]) ** 2) - 1) < 512 * 2.0 ** -53
    z = np.zeros(512, np.float32)
    assert lib.dot(_ptr(z), _ptr(a), 512) == 0.0
    for bad in (np.inf, -np.inf, np.nan):
        b = a.copy()
        b[37] = bad
        assert not np.isfinite(lib.dot(_ptr(b), _ptr(a), 512)) and not np.isfinite(lib.dot(_ptr(b), _ptr(z), 512))
        assert not np.isfinite(lib.dot(_ptr(b), _ptr(np.ones(512, np.float32)), 512))


@pytest.mark.parametrize("scale", [0, -126, -149, 90])
def test_total_of_compensated_sums(lib, scale):
    rng = np.random.default_rng(scale + 200)
    s = (rng.standard_normal(32) * 10.0 ** rng.uniform(-12, 0, 32) * 2.0 ** scale).astype(np.float32)
    c = (s * 2.0 ** -24 * rng.uniform(-1, 1, 32).astype(np.float32)).astype(np.float32)
    s[3], c[3] = 0.0, np.float32(2.0 ** (scale - 20))  # nothing but the compensation
    exact = sum(Fraction(float(x)) - Fraction(float(y)) for x, y in zip(s, c))
    size = sum(abs(Fraction(float(x))) + abs(Fraction(float(y))) for x, y in zip(s, c))
    got = lib.total(_ptr(s), _ptr(c))
    assert abs(Fraction(got) - exact) <= abs(exact) / 2 ** 51 + size / 2 ** 60
    s[5] = np.inf
    assert not np.isfinite(lib.total(_ptr(s), _ptr(c)))


def test_units_fit_a_message(lib):
    """A sum's unit travels in twelve bits: that of a sum of 0 too, which has no bits to place."""
    for d in (0.0, -0.0, 5e-324, 2.0 ** -298, 1.0, -1e300, np.inf, np.nan):
        a = np.zeros(32)
        a[7] = d
        p = ctypes.POINTER(ctypes.c_double)
        assert -2048 <= lib.unit(a.ctypes.data_as(p)) <= 2047, d
        got = lib.lanes(a.ctypes.data_as(p))
        assert got == d or not (np.isfinite(d) or np.isfinite(got)) or abs(d) < 2.0 ** -1000, (d, got)


@pytest.mark.parametrize("spread", [0, 8, 60, 200])
@pytest.mark.parametrize("seed", range(8))
def test_total_of_doubles(lib, spread, seed):
    rng = np.random.default_rng(1000 * seed + spread)
    d = rng.standard_normal(32) * 2.0 ** rng.integers(-spread, 1, 32)
    if seed % 2:
        d = np.abs(d)
    d[rng.integers(0, 32, 5)] = 0.0
    exact = sum(Fraction(float(x)) for x in d)
    got = lib.lanes(d.ctypes.data_as(ctypes.POINTER(ctypes.c_double)))
    assert abs(Fraction(got) - exact) <= abs(exact) / 2 ** 53 + Fraction(float(np.abs(d).max())) / 2 ** 51
    for scale in (2.0 ** -290, 2.0 ** 250):
        e = d * scale
        assert lib.lanes(e.ctypes.data_as(ctypes.POINTER(ctypes.c_double))) == got * scale


def test_quotient_is_rounded_once(lib):
    """The step lengths: the float nearest to the quotient of two doubles, with quotients next to the middle of
    two floats among them, and FP64's division where FP32 has no room."""
    rng = np.random.default_rng(5)
    for i in range(20000):
        b = float(rng.standard_normal() * 2.0 ** rng.integers(-50, 50))
        if i % 4 == 0:  # near a middle: (f + half an ulp) * b, and a last place or two of the product off
            f = np.float32(rng.uniform(0.5, 1.0))
            a = (float(f) + float(np.spacing(f)) / 2) * b
            for _ in range(int(rng.integers(0, 3))):
                a = float(np.nextafter(a, np.inf if rng.random() < 0.5 else -np.inf))
        else:
            a = float(rng.standard_normal() * 2.0 ** rng.integers(-50, 50))
        got, q = lib.quot(a, b), Fraction(a) / Fraction(b)
        near = np.float32(float(q))
        best = min((near, np.nextafter(near, np.float32(np.inf)), np.nextafter(near, np.float32(-np.inf))), key=lambda f: abs(Fraction(float(f)) - q))
        assert abs(Fraction(got) - q) <= abs(Fraction(float(best)) - q) * (1 + Fraction(1, 2 ** 20)), (a, b, got)
    for a, b in ((1e-60, 3e-60), (1e50, 7e49), (0.0, 2.0), (1.0, 0.0), (-1.0, 0.0), (0.0, 0.0), (np.nan, 1.0), (1.0, np.inf)):
        with np.errstate(all="ignore"):
            want = np.float32(np.float64(a) / np.float64(b))
        assert np.float32(lib.quot(a, b)).tobytes() == want.tobytes() or (np.isnan(want) and np.isnan(lib.quot(a, b))), (a, b)


@pytest.mark.parametrize("kind", ["one", "residual", "cancel", "gone", "tiny", "huge", "edge", "denormal", "spread"])
@pytest.mark.parametrize("seed", range(8))
def test_products_of_a_lane_together(lib, kind, seed):
    """The bound of test_dot_is_no_worse_than_fp64, where a lane goes to FP64 when its largest product lies outside
    2^-90 to 2^101; inside, a product too small for FP32 loses 2^-149, 16 of them 2^-55 of the largest."""
    a, b = _terms(np.random.default_rng(seed), kind)
    prods = [Fraction(float(x)) * Fraction(float(y)) for x, y in zip(a, b)]
    exact, size, far, small = sum(prods), sum(abs(p) for p in prods), Fraction(0), Fraction(0)
    for lane in range(32):
        mine = [abs(p) for p in prods[lane::32]]
        if not 2.0 ** -89 <= max(mine) < 2.0 ** 100:
            far += sum(mine)
        else:
            small += sum(Fraction(1, 2 ** 149) for p in mine if p < 2.0 ** -98)
    got = lib.dot16(_ptr(a), _ptr(b), 0)
    assert abs(Fraction(got) - exact) <= abs(exact) / 2 ** 51 + size / 2 ** 60 + far / 2 ** 44 + small, (kind, seed, got, float(exact))


def test_far_products_of_a_lane_together(lib):
    one, z = np.ones(512, np.float32), np.zeros(512, np.float32)
    for big in (1e25, 1e-25):
        a = np.full(512, big, np.float32)
        assert abs(lib.dot16(_ptr(a), _ptr(a), 0) / (512 * float(a[0]) ** 2) - 1) < 512 * 2.0 ** -53
        for bad in (np.inf, np.nan):
            b = a.copy()
            b[37] = bad
            for other in (a, one, z):
                assert not np.isfinite(lib.dot16(_ptr(b), _ptr(other), 0))
    assert lib.dot16(_ptr(z), _ptr(one), 0) == 0.0


@pytest.mark.parametrize("kind", ["one", "residual", "cancel", "gone", "tiny", "huge", "edge", "denormal", "spread"])
@pytest.mark.parametrize("seed", range(8))
def test_untested_products_stand_where_the_total_holds(lib, kind, seed):
    """Products without a test for their range, 2^-149 lost by each at most: where their total holds it meets the
    bound of the tested ones, and where it does not (too small, too large, not finite) FP64's sum takes its
    place, within FP64's own bound."""
    a, b = _terms(np.random.default_rng(seed), kind)
    prods = [Fraction(float(x)) * Fraction(float(y)) for x, y in zip(a, b)]
    exact, size = sum(prods), sum(abs(p) for p in prods)
    got = lib.dot16(_ptr(a), _ptr(b), 1)
    if lib.holds(got):
        assert abs(Fraction(got) - exact) <= abs(exact) / 2 ** 51 + size / 2 ** 60 + Fraction(512, 2 ** 149)
    else:
        assert kind not in ("one", "residual")
        got = lib.dot16(_ptr(a), _ptr(b), 2)
        assert abs(Fraction(got) - exact) <= size / 2 ** 44


def test_totals_that_do_not_hold(lib):
    for t in (0.0, 8e-19, 1.4e36, np.inf, np.nan):
        assert not lib.holds(t) and not lib.holds(-t)
    for t in (9e-19, 1.0, 1.3e36):
        assert lib.holds(t) and lib.holds(-t)
