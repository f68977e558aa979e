"""The 64-bit fixed-point cell of the FP64 kernels (csrc/lmm_fix64.h), compiled
for the host and checked against long double: 2^x, the logistic t, a whole
step, its exact reversal, and the conversions, at the edges of their ranges.

Bounds, in units of the formats' last place: a truncated product is low by at
most 2 units, a shift by 1; a table entry is within 2 units of 2^-62, and
2^x adds one product (2 units) and the polynomial (2^-66). The reciprocal of a
D in (1, 3] leaves out e^3 < 2^-60 and truncates 4 units of 2^-62 against
r > 1/3.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG_NAME, ROOT

SRC = r"""
#include "lmm_fix64.h"
#include <cmath>
using namespace lmm;
typedef long double ld;
static uint64_t tab[kFxTable];
static ld up(ld a, ld b) { return a > b ? a : b; }
static ld val(uint64_t v) { return (ld)v * 0x1p-56L; }
extern "C" {
void init() { for (int j = 0; j < kFxTable; ++j) tab[j] = fx_table_entry(j); }
// largest relative errors of 2^frac, t, 1 - t (as doubles) and r
void logistic(const uint64_t *X, int n, double *err)
{
    ld a = 0, b = 0, c = 0, d = 0;
    for (int i = 0; i < n; ++i) {
        const ld x = val(X[i]), f = x - floorl(x), E = exp2l(x - kFxOff), t = 1 / (1 + E), u = 1 / (1 + 1 / E);
        const FxT q = fx_logistic(X[i], tab);
        a = up(a, fabsl((ld)q.Em * 0x1p-62L / exp2l(f) - 1));
        b = up(b, fabsl((ld)q.r * 0x1p-62L * exp2l(-(int)q.up) / t - 1));
        c = up(c, fabsl(fx_t(q) / t - 1));
        d = up(d, fabsl(fx_1mt(q) / u - 1));
    }
    err[0] = a; err[1] = b; err[2] = c; err[3] = d;
}
// largest errors of a drift term (units of 2^-58), of X after a step (2^-56) and of sigma t (1-t) (relative);
// returns the steps that do not reverse to the same bits
int steps(const uint64_t *X, const double *z, const double *sigma, const int *kk, int n, double *err)
{
    int bad = 0;
    ld a = 0, b = 0, c = 0;
    for (int i = 0; i < n; ++i) {
        const FxConst k = fx_const(sigma[i], kk[i]);
        const FxT q = fx_logistic(X[i], tab);
        uint64_t Y = fx_normal(z[i]);
        const ld E = exp2l(val(X[i]) - kFxOff), t = 1 / (1 + E), s = sigma[i], lag = 0.52L * (kk[i] + 1);
        a = up(a, fabsl((ld)fx_drift(q, k) - s * t * 0x1p58L));
        const uint64_t x = fx_step(X[i], Y, k);
        // the step at the drift sum that Y stands for, lag units above it
        const ld y = (ld)(int64_t)(Y - (16ull << 58)) + lag;
        const ld xe = (ld)X[i] - s * 1.44269504088896340735992468100189214L * (y / 4 - s * 0x1p55L);
        b = up(b, fabsl((ld)(int64_t)x - xe));
        bad += fx_unstep(x, Y, k) != X[i];
        if (s > 0) c = up(c, fabsl(fx_slope(q, k) / (s * t / (1 + 1 / E)) - 1));
    }
    err[0] = a; err[1] = b; err[2] = c;
    return bad;
}
// largest error of X for v = delta L0 (units of 2^-56); -1 where the top bit tells v outside
double rate(double v)
{
    const uint64_t X = fx_rate(v, std::log2(v), tab);
    return X >> 63 ? -1.0 : (double)fabsl(((ld)X - (kFxOff - log2l((ld)v)) * 0x1p56L));
}
double from_signed(int64_t v) { return fx_signed(v); }
}
"""


@pytest.fixture(scope="module")
def fx(tmp_path_factory):
    d = tmp_path_factory.mktemp("fix64")
    (d / "fx.cpp").write_text(SRC)
    so = str(d / "fx.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(ROOT, PKG_NAME, "csrc"),
                    str(d / "fx.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.rate.restype = lib.from_signed.restype = ctypes.c_double
    lib.rate.argtypes = [ctypes.c_double]
    lib.from_signed.argtypes = [ctypes.c_int64]
    lib.init()
    return lib


def _rates(n):
    rng = np.random.default_rng(7)
    X = rng.integers(0, 1 << 63, n, dtype=np.uint64)
    edges = [(e << 56) + d for e in range(128) for d in (0, 1, (1 << 56) - 1, 1 << 46, (1 << 46) - 1)]
    return np.concatenate([X, np.array(edges, dtype=np.uint64)])


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def test_logistic(fx):
    X, err = _rates(300_000), np.zeros(4)
    fx.logistic(_p(X), len(X), _p(err))
    assert err[0] <= 4.5 * 2.0 ** -62 + 2.0 ** -64
    assert err[1] <= 2.0 ** -58
    assert err[2] <= 2.0 ** -53 * 1.01 + 2.0 ** -58
    assert err[3] <= 2.0 ** -53 * 1.01 + 2.0 ** -57


@pytest.mark.parametrize("lo,hi", [(0.0, 0.0), (1e-12, 1e-6), (1e-3, 0.2), (0.2, 0.34)])
def test_step_and_exact_reversal(fx, lo, hi):
    rng = np.random.default_rng(8)
    X = _rates(20_000)
    X = np.ascontiguousarray(X[(X >> np.uint64(56) >= 9) & (X >> np.uint64(56) < 119)])     # stays in range for any z
    n = len(X)
    z, sigma = rng.uniform(-15.5, 15.5, n), rng.uniform(lo, hi, n)
    k = rng.integers(0, 256, n).astype(np.int32)
    err = np.zeros(3)
    assert fx.steps(_p(X), _p(z), _p(sigma), _p(k), n, _p(err)) == 0
    # product 2 units and shift 1; product 2 units, constant 1 unit (its 0.75 taken out), X's own place
    assert err[0] <= 3.5 and err[1] <= 3.5
    # three products of at most 2 units each on values above 2^55, and the double's own rounding
    assert err[2] <= 2.0 ** -53 * 1.01 + 3 * 2.0 ** -54


def test_rate_conversion_and_range(fx):
    for v in np.exp2(np.concatenate([np.linspace(-55.9, 71.9, 5001), np.arange(-55.0, 72), [-1e-15, 1e-15]])):
        assert 0.0 <= fx.rate(float(v)) <= 4.0
    for v in (2.0 ** 72, 2.0 ** -56, 1e300, 5e-324, float("inf"), float("nan"), 0.0, -1.0):
        assert fx.rate(v) == -1.0


def test_signed_conversion(fx):
    for v in (1, -1, 3, -3, 1 << 57, -(1 << 57), (1 << 58) - 1, (1 << 62) - 1, -(1 << 62) + 1, 0x123456789abcdef):
        got, want = fx.from_signed(v), (v | 1 if v > 0 else -(-v | 1)) * 2.0 ** -58
        assert abs(got - want) <= 2.0 ** -53 * 1.01 * abs(want)
