"""The FP64 form's powers, logarithms, sines and cosines (64-bit fixed point, csrc/kernels/sample_body.cuh),
compiled for the host from the source that the kernels are compiled from, against 50-digit values.

Bounds: the result's rounding is half an ulp.  A logarithm is off by at most 2^-61 (Q62 table entry, its series
and one truncated product) and is multiplied by exponents of up to 32, two of them in a product, and by ln 2;
2^x adds 2^-61: below 2^-55 relative, a quarter of an ulp, before the rounding, so a power is within 0.75 ulp.
Sines and cosines are within 2^-58 absolute, and below pi/128 the sine within 0.75 ulp."""
import ctypes
import os
import random
import re
import subprocess

import numpy as np
import pytest

from feyntrop_gb300 import build as native

mp = pytest.importorskip("mpmath")

SHIMS = r"""
#include <cmath>
#include <cstdint>
#include <cstring>
#include <algorithm>
using std::max; using std::min;
#define __device__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
struct ulonglong2 { unsigned long long x, y; };
struct double2 { double x, y; };
typedef unsigned long long u64;
typedef unsigned int u32;
static long long __double_as_longlong(double x) { long long r; memcpy(&r, &x, 8); return r; }
static double __longlong_as_double(long long x) { double r; memcpy(&r, &x, 8); return r; }
static int __double2hiint(double x) { return (int)(__double_as_longlong(x) >> 32); }
static double __hiloint2double(int h, int l) { return __longlong_as_double((long long)((u64)(u32)h << 32 | (u32)l)); }
static int __clzll(long long x) { return x ? __builtin_clzll((u64)x) : 64; }
static int __clz(int x) { return x ? __builtin_clz((u32)x) : 32; }
static u64 __umul64hi(u64 a, u64 b) { return (u64)((unsigned __int128)a * b >> 64); }
static double u01(u64 x) { return (double)(x >> 11) * 0x1.0p-53; }
"""

CALLS = r"""
extern "C" void pow1mu(int n, const u64* x, const double* y, double* out)
{
    for (int i = 0; i < n; i++) out[i] = pow_1mu(x[i], y[i]);
}
extern "C" void power(int n, double a, const double* x, double b, const double* y, double* out)
{
    for (int i = 0; i < n; i++) out[i] = power_product(a, log2_64(x[i]), b, log2_64(y[i]));
}
extern "C" void difference(int n, const double* x, const double* y, int L, double* out)
{
    for (int i = 0; i < n; i++) out[i] = log2_difference(log2_64(x[i]), log2_64(y[i]), L);
}
extern "C" void reach(int n, double a, const double* x, int* out)
{
    for (int i = 0; i < n; i++) out[i] = in_reach(log2_64(x[i]), log2_limit(a));
}
extern "C" void sine_cosine(int n, const double* x, double* s, double* c)
{
    for (int i = 0; i < n; i++) sincos_64(x[i], s[i], c[i]);
}
"""


@pytest.fixture(scope="module")
def fn(tmp_path_factory):
    native.build()
    tmp = tmp_path_factory.mktemp("fp64")
    here = os.path.dirname(native.LIB)
    (tmp / "dump.cpp").write_text("""#include <cstdio>
#include "%s"
int main()
{
    ft::kernel_key k;
    k.E = 2; k.V = 2; k.loops = 1; k.ek = {1, 1}; k.el = {0, 0};
    std::fputs(ft::kernel_source(k).c_str(), stdout);
}
""" % os.path.join(native.CSRC, "jit.hpp"))
    subprocess.run([native.CXX, "-std=c++17", "-I" + os.path.join(native.CUDA, "include"), str(tmp / "dump.cpp"), "-o",
                    str(tmp / "dump"), "-L" + here, "-lfeyntrop_gb300", "-Wl,-rpath," + here], check=True)
    text = subprocess.run([str(tmp / "dump")], check=True, capture_output=True, text=True).stdout
    tables = re.search(r"__device__ const ulonglong2 FT_LOG64.*?#define FT_STEP_Q69 \w+\n", text, re.S).group(0)
    code = text[text.index("static __device__ __forceinline__ int hi_word"):
                text.index("static __device__ __noinline__ double rcp_slow")]
    (tmp / "fn.cpp").write_text(SHIMS + tables + code + CALLS)
    subprocess.run([native.CXX, "-std=c++17", "-O2", "-ffp-contract=off", "-w", "-shared", "-fPIC",
                    str(tmp / "fn.cpp"), "-o", str(tmp / "fn.so")], check=True)
    return ctypes.CDLL(str(tmp / "fn.so"))


def ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def ulps(got, exact):
    """|got - exact| in units of the last place of exact"""
    return float(abs(mp.mpf(float(got)) - exact) / mp.mpf(2) ** (mp.frexp(exact)[1] - 53))


@pytest.mark.parametrize("y", [0.02, 0.5, 1.0, 7.3, 31.9, 49.7, 119.3, 1e3, 1e6])
def test_powers_of_uniform_draws(fn, y):
    rng = random.Random(repr(y))
    x = [rng.getrandbits(64) for _ in range(1500)]
    x += [rng.getrandbits(64) >> rng.randint(0, 52) for _ in range(400)]            # u near 0
    x += [~(rng.getrandbits(64) >> rng.randint(0, 53)) % 2**64 for _ in range(400)]  # u near 1
    x += [0, 2047, 2048, 2**64 - 1]
    xs, ys, out = np.array(x, dtype=np.uint64), np.full(len(x), y), np.empty(len(x))
    fn.pow1mu(len(x), ptr(xs), ptr(ys), ptr(out))
    with mp.workdps(50):
        for v, got in zip(x, out):
            exact = (1 - mp.mpf(v >> 11) / 2**53) ** mp.mpf(y)
            if exact < 1e-300:
                assert got < 2e-300
            else:
                assert ulps(got, exact) <= (0.75 if y < 32 else 1.0), (v, y)


@pytest.mark.parametrize("a,b", [(-2.0, -1.0), (-2.0, -3.0), (-1.0, -10.0), (-3.0, -30.0), (0.5, -30.0), (30.0, 30.0),
                                 (-0.4375, 0.15625), (-1.0, 0.0), (0.0, -2.5), (-3.25, 1.5), (-1e-6, 2e-9)])
def test_products_of_powers(fn, a, b):
    rng = random.Random(repr((a, b)))
    draw = [lambda: 1.0 + rng.uniform(-1, 1) * 2.0**-rng.randint(1, 52), lambda: rng.uniform(0.01, 100),
            lambda: 2.0**rng.uniform(-15, 15)]
    x = np.array([rng.choice(draw)() for _ in range(2000)])
    y = np.array([rng.choice(draw)() for _ in range(2000)])
    out = np.empty(2000)
    fn.power(2000, ctypes.c_double(a), ptr(x), ctypes.c_double(b), ptr(y), ptr(out))
    with mp.workdps(50):
        for u, v, got in zip(x, y, out):
            assert ulps(got, mp.mpf(u) ** mp.mpf(a) * mp.mpf(v) ** mp.mpf(b)) <= 0.75, (u, v)


@pytest.mark.parametrize("loops", [0, 1, 3, 20])
def test_differences_of_logarithms(fn, loops):
    rng = random.Random(loops)
    x = np.array([2.0 ** rng.choice((rng.uniform(-300, 300), rng.uniform(-2, 2), rng.uniform(-1e-9, 1e-9))) for _ in range(2000)])
    y = np.array([2.0 ** rng.choice((rng.uniform(-300, 300), rng.uniform(-2, 2), rng.uniform(-1e-9, 1e-9))) for _ in range(2000)])
    x[:2], y[:2], out = 1.0, 1.0, np.empty(2000)
    fn.difference(2000, ptr(x), ptr(y), loops, ptr(out))
    with mp.workdps(50):
        for u, v, got in zip(x, y, out):
            exact = mp.log(mp.mpf(u), 2) - loops * mp.log(mp.mpf(v), 2)
            assert abs(got - exact) <= (loops + 1) * mp.mpf(2)**-61 + abs(exact) * mp.mpf(2)**-53, (u, v)


def test_reach_of_the_fixed_point_powers(fn):
    """In reach: |a| below 32 and |a log2 x| at most 500; 1 and its neighbours always are."""
    rng = random.Random(3)
    for a in [0.0, -0.0, 2.0**-60, 1e-30, 0.01, 0.5, 1.0, 2.0, 3.5, 31.99, 32.0, 1e3, 1e300, np.inf, np.nan]:
        for s in (a, -a):
            x = np.array([2.0 ** rng.uniform(-1022, 1023) for _ in range(500)] + [0.75, 1.0, 1.5])
            got = np.zeros(len(x), dtype=np.int32)
            fn.reach(len(x), ctypes.c_double(s), ptr(x), ptr(got))
            if not a < 32 or 0 < a < 2.0**-60:
                assert not got.any()
            else:
                assert (np.abs(s * np.log2(x))[got != 0] <= 500).all() and got[-3:].all()


def test_sines_and_cosines(fn):
    rng = random.Random(7)
    x = [s * 10.0 ** rng.uniform(-300, 5) for s in (1, -1) for _ in range(300)]
    x += [s * 10.0 ** rng.uniform(-12, 0) for s in (1, -1) for _ in range(1500)]
    x += [rng.uniform(-50, 50) for _ in range(1500)]
    x += [k * np.pi / 128 + d for k in (-3, -1, 1, 2, 64, 129) for d in (-1e-9, 0.0, 1e-9)] + [0.0, -0.0, 5e-324, 1e-310]
    x = np.array(x)
    s, c = np.empty(len(x)), np.empty(len(x))
    fn.sine_cosine(len(x), ptr(x), ptr(s), ptr(c))
    with mp.workdps(400):
        for v, gs, gc in zip(x, s, c):
            es, ec = mp.sin(mp.mpf(float(v))), mp.cos(mp.mpf(float(v)))
            # an absolute 2^-58 and the rounding of the value
            assert abs(gs - es) <= mp.mpf(2)**-58 + abs(es) * mp.mpf(2)**-53, v
            assert abs(gc - ec) <= mp.mpf(2)**-58 + abs(ec) * mp.mpf(2)**-53, v
            if 1e-300 < abs(v) < np.pi / 128:
                assert ulps(gs, es) <= 0.75, v
            elif abs(v) <= 1e-300:
                assert gs == v and gc == 1.0
