"""The solver's FP32 dot accumulator (csrc/dot.cuh, compiled for the host) against the FP64 sum it stands
for.  Joining 32 sums: within one FP64 rounding of the exact sum, as long as no more than 2^10
cancels.  Long chains: rms error over the trials no larger than with FP64 fused multiply-adds."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fem_taichi_gb300", "csrc")
SRC = r"""
#include <cmath>
#define __device__
#define __forceinline__ inline
static inline float __fadd_rn(float a, float b) { volatile float r = a + b; return r; }
static inline float __fsub_rn(float a, float b) { volatile float r = a - b; return r; }
static inline float __fmul_rn(float a, float b) { volatile float r = a * b; return r; }
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
using std::fma;
#include "dot.cuh"
using D = fem::Dot<float>;
extern "C" {
// warp tree over 32 lanes, each the sum of n nodes' products a b
double warp_sum(const float* a, const float* b, int n) {
    D d[32], t[32];
    for (int l = 0; l < 32; ++l)
        for (int i = 0; i < n; ++i) {
            const float *x = a + 3 * (l * n + i), *y = b + 3 * (l * n + i);
            d[l].add3(x[0], y[0], x[1], y[1], x[2], y[2]);
        }
    for (int off = 16; off >= 1; off >>= 1) {
        for (int l = 0; l < 32; ++l) {
            t[l] = d[l];
            t[l].join(d[l ^ off].s, d[l ^ off].c, d[l ^ off].d);
        }
        for (int l = 0; l < 32; ++l) d[l] = t[l];
    }
    return d[0].value();
}
double chain(const float* a, const float* b, int n) {
    D d;
    for (int i = 0; i < n; ++i) d.add3(a[3 * i], b[3 * i], a[3 * i + 1], b[3 * i + 1], a[3 * i + 2], b[3 * i + 2]);
    return d.value();
}
double single(const float* a, const float* b, int n) {
    D d;
    for (int i = 0; i < n; ++i) d.add(a[i], b[i]);
    return d.value();
}
double chain64(const float* a, const float* b, int n) {
    fem::Dot<double> d;
    for (int i = 0; i < 3 * n; i += 3) d.add3(a[i], b[i], a[i + 1], b[i + 1], a[i + 2], b[i + 2]);
    return d.value();
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("dot")
    (d / "dot.cpp").write_text(SRC)
    so = str(d / "dot.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC, str(d / "dot.cpp"),
                    "-o", so], check=True)
    L = ctypes.CDLL(so)
    for f in (L.warp_sum, L.chain, L.single, L.chain64):
        f.restype = ctypes.c_double
        f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int]
    return L


def _exact(a, b):
    """Correctly rounded sum of the products (each exact in FP64: 24-bit factors)."""
    import math
    return math.fsum((a.astype(np.float64) * b.astype(np.float64)).tolist())


def _call(f, a, b, n):
    return f(a.ctypes.data, b.ctypes.data, n)


@pytest.mark.parametrize("spread", [0, 6])
def test_warp_sum_of_single_products(lib, spread):
    """One product a lane: nothing but the joins rounds."""
    rng = np.random.default_rng(spread)
    worst = 0.0
    for _ in range(300):
        a, b = (rng.standard_normal((32, 3)) * 10.0 ** rng.uniform(-spread / 2, spread / 2, (32, 3)) for _ in range(2))
        a[:, 1:] = 0
        a, b = a.astype(np.float32), b.astype(np.float32)
        want = _exact(a.ravel(), b.ravel())
        if abs(want) < 2.0 ** -10 * np.abs(a.astype(float) * b).sum():
            continue
        worst = max(worst, abs(_call(lib.warp_sum, a, b, 1) - want) / abs(want))
    assert worst <= 2.0 ** -52


@pytest.mark.parametrize("signs", [False, True])
def test_long_chains(lib, signs):
    rng = np.random.default_rng(1)
    n, e, e64 = 2000, [], []
    for _ in range(60):
        a = rng.standard_normal(3 * n).astype(np.float32)
        b = (rng.standard_normal(3 * n) if signs else a * (1 + 0.3 * rng.random(3 * n))).astype(np.float32)
        want = _exact(a, b)
        e.append(_call(lib.chain, a, b, n) - want)
        e64.append(_call(lib.chain64, a, b, n) - want)
    assert np.sqrt(np.mean(np.square(e))) <= np.sqrt(np.mean(np.square(e64)))


def test_one_node_and_single_products_are_pairs(lib):
    """Up to three products are within 2^-46 of the largest: two-sums and one rounding of the low part each."""
    rng = np.random.default_rng(2)
    for _ in range(200):
        a, b = (rng.standard_normal(3).astype(np.float32) for _ in range(2))
        want, big = _exact(a, b), np.abs(a.astype(float) * b).sum()
        assert abs(_call(lib.chain, a, b, 1) - want) <= 2.0 ** -46 * big
        assert abs(_call(lib.single, a, b, 3) - want) <= 2.0 ** -46 * big


def test_not_finite(lib):
    a = np.ones(96, np.float32)
    b = a.copy()
    b[40] = np.inf
    assert not np.isfinite(_call(lib.warp_sum, a, b, 1))
    b[40] = np.nan
    assert np.isnan(_call(lib.warp_sum, a, b, 1))
