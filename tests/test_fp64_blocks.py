"""cs_fp64.cuh on the host: the header's arithmetic is plain IEEE FP64, so g++
compiles it with the CUDA intrinsics replaced by their definitions.  rsqrtf, whose
result the CUDA documentation bounds to 2 ulp, is given every error in that range.

Bounds (in units of the last place of the result, from the series):
  cs_rcp       final rounding 1/2, cut-off e^3 < 2^-67 of the value < 2^-14 ulp: 0.51
  cs_rsqrt     final rounding 1/2, rounding of x r in h up to 1/2, cut-off
               5/16 h^3 < 2^-63 of the value < 2^-10 ulp: 1.01
  g            final rounding of the Newton step, whose cut-off (2.5 2^-53)^2 / 2 and
               rounding of a residual of 5 2^-53 are far below: 0.51
  t            half of a's 2.5 of 2^-53 (|x0| a is at most half of |v|^2 / 2), two
               roundings of 1: 3.25 of 2^-53 relative, and the cut-offs: 3.3
"""
import ctypes
import os
import subprocess
from decimal import Decimal, getcontext

import numpy as np
import pytest

from conftest import ROOT

getcontext().prec = 60
HARNESS = r"""
#include <math.h>
#include <stdint.h>
#include <string.h>
#define __device__
#define __forceinline__ inline
static inline int64_t bits(double x) { int64_t b; memcpy(&b, &x, 8); return b; }
static inline double value(int64_t b) { double x; memcpy(&x, &b, 8); return x; }
static inline int __double2hiint(double x) { return (int)(bits(x) >> 32); }
static inline int __double2loint(double x) { return (int)(uint32_t)bits(x); }
static inline double __hiloint2double(int h, int l) { return value((int64_t)(((uint64_t)(uint32_t)h << 32) | (uint32_t)l)); }
static inline long long __double_as_longlong(double x) { return bits(x); }
static inline unsigned __float_as_uint(float x) { unsigned b; memcpy(&b, &x, 4); return b; }
static inline float __uint_as_float(unsigned b) { float x; memcpy(&x, &b, 4); return x; }
static inline float __frcp_rn(float x) { return 1.0f / x; }
static int seed_error;
static inline float test_rsqrtf(float x) {
  float r = (float)(1.0 / sqrt((double)x));
  for (int i = 0; i < (seed_error < 0 ? -seed_error : seed_error); ++i) r = nextafterf(r, seed_error < 0 ? 0.0f : 4.0f);
  return r;
}
#define rsqrtf test_rsqrtf
#include "cs_fp64.cuh"
extern "C" void set_seed_error(int e) { seed_error = e; }
extern "C" void rcp(int n, const double* x, double* y) { for (int i = 0; i < n; ++i) y[i] = cs_rcp(x[i]); }
extern "C" void rsq(int n, const double* x, double* y) { for (int i = 0; i < n; ++i) y[i] = cs_rsqrt(x[i]); }
extern "C" int reflector(double ss, double x0, double* out, long long least) {
  return least ? cs_reflector(ss, x0, out, out + 1, out + 2, least) : cs_reflector(ss, x0, out, out + 1, out + 2);
}
"""
NAN, INF = float("nan"), float("inf")
LEAST_BABD = 0x03A8F2B061AEA072  # 1e-290 / 2


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fp64")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "collocation-solver-cuda_gb300", "csrc"), "-o", str(d / "h.so"), str(d / "h.cpp")],
                   check=True)
    lib = ctypes.CDLL(str(d / "h.so"))
    dbl = ctypes.POINTER(ctypes.c_double)
    for f in (lib.rcp, lib.rsq):
        f.argtypes = [ctypes.c_int, dbl, dbl]
    lib.reflector.argtypes = [ctypes.c_double, ctypes.c_double, dbl, ctypes.c_longlong]
    return lib


def call(f, x):
    x = np.ascontiguousarray(x, dtype=np.float64)
    y = np.empty_like(x)
    dbl = ctypes.POINTER(ctypes.c_double)
    f(len(x), x.ctypes.data_as(dbl), y.ctypes.data_as(dbl))
    return y


def ulps(got, exact):
    return abs(Decimal(float(got)) - exact) / Decimal(float(np.spacing(abs(got))))


def samples(rng):
    """Random numbers of every magnitude the series take, powers of two and their
    neighbours, and both ends of the exponent range."""
    ex = np.concatenate([rng.integers(16, 2031, 400), [16, 17, 1022, 1023, 1024, 2029, 2030]])
    man = np.concatenate([rng.integers(0, 2**52, 400), np.zeros(7, int)])
    base = ((ex.astype(np.int64) << 52) | man).view(np.float64)
    return np.concatenate([base, np.nextafter(base[400:], INF), np.nextafter(base[401:], 0.0)])


def test_reciprocal(lib):
    x = samples(np.random.default_rng(1))
    for v in (x, -x):
        for a, y in zip(v, call(lib.rcp, v)):
            assert ulps(y, 1 / Decimal(float(a))) <= Decimal("0.51"), a


def test_reciprocal_square_root(lib):
    x = samples(np.random.default_rng(2))
    for e in range(-2, 3):
        lib.set_seed_error(e)
        for a, y in zip(x, call(lib.rsq, x)):
            assert ulps(y, 1 / Decimal(float(a)).sqrt()) <= Decimal("1.01"), (a, e)
    lib.set_seed_error(0)


def test_ends_of_the_range_divide(lib):
    tiny = 2.0**-1074
    x = np.array([0.0, -0.0, INF, -INF, NAN, tiny, 2.0**-1022, 2.0**-1008, 2.0**1008, 1.7e308, -tiny, -1.7e308])
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(call(lib.rcp, x), 1.0 / x)
        np.testing.assert_array_equal(call(lib.rsq, x), 1.0 / np.sqrt(x))


@pytest.mark.parametrize("seed_error", [-2, 0, 2])
def test_reflector_of_ordinary_columns(lib, seed_error):
    rng = np.random.default_rng(3)
    lib.set_seed_error(seed_error)
    out = (ctypes.c_double * 3)()
    for scale in (1e-100, 1.0, 1e100):
        for _ in range(100):
            c = scale * rng.standard_normal(int(rng.integers(1, 12)))
            ss, x0 = float(np.dot(c, c)), float(c[0])
            assert lib.reflector(ss, x0, out, LEAST_BABD)
            g = Decimal(ss).sqrt() * (-1 if x0 >= 0 else 1)
            assert ulps(out[0], g) <= Decimal("0.51")
            assert out[1] == x0 - out[0]
            t = 1 / (Decimal(ss) + abs(Decimal(x0) * g))
            assert abs(Decimal(out[2]) / t - 1) <= Decimal("3.3") * Decimal(2)**-53
    lib.set_seed_error(0)


@pytest.mark.parametrize("ss,x0,least,reflects", [
    (0.0, 0.0, 0, False), (0.0, 1e-170, LEAST_BABD, False), (1e-17, 0.0, 0, False), (1e-15, 0.0, 0, True),
    (1e-291, 0.0, LEAST_BABD, False), (1e-289, 0.0, LEAST_BABD, True), (1e-320, 1e-160, 0, False),
    # a column with a NaN or an infinity is never "nothing to eliminate"
    (NAN, 1.0, 0, True), (NAN, NAN, 0, True), (NAN, INF, 0, True), (INF, 1.0, 0, True), (INF, INF, 0, True),
    (INF, -INF, 0, True), (NAN, 0.0, LEAST_BABD, True), (INF, -INF, LEAST_BABD, True), (-NAN, 1.0, 0, True)])
def test_reflector_skips_only_a_number_below_the_limit(lib, ss, x0, least, reflects):
    out = (ctypes.c_double * 3)()
    assert bool(lib.reflector(ss, x0, out, least)) == reflects
    if reflects and not np.isfinite(ss):
        assert np.isnan(out[0])
