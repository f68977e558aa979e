"""The integer binary64 arithmetic of the FP64 normals (csrc/lmm_soft64.h),
compiled for the host and compared bit by bit with the machine's doubles: the
four operations on random and edge mantissas over the exponents they are used
with, and AS241's central branch over MRG32k3a's integers."""
import ctypes
import os
import subprocess

import pytest

from conftest import PKG_NAME, ROOT

SRC = r"""
#include "lmm_soft64.h"
#include <cmath>
#include <random>
using namespace lmm;
static uint64_t B(double d) { uint64_t b; memcpy(&b, &d, 8); return b; }
static double D(uint64_t b) { double d; memcpy(&d, &b, 8); return d; }
static S64 S(double d) { return d == 0 ? S64{0, 0} : s64_bits(B(d)); }
static std::mt19937_64 g(1);
static double rnd(double lo, double hi)
{
    uint64_t b = B(std::exp(std::log(lo) + (std::log(hi) - std::log(lo)) * (g() >> 11) * 0x1p-53));
    switch (g() % 8) {                                  // mantissas that make ties and carries
        case 0: b &= ~0xffffffffull; break;
        case 1: b |= 0xffffffffull; break;
        case 2: b &= ~((1ull << 40) - 1); break;
        case 3: b &= ~((1ull << 27) - 1); break;
        case 4: b |= (1ull << 52) - 1; break;
    }
    return D(b);
}
extern "C" long ops(int op, int n)
{
    long bad = 0;
    for (int i = 0; i < n; ++i) {
        volatile double want;
        S64 got;
        if (op == 0) {
            const double a = rnd(1e-18, 1e5), b = rnd(1e-18, 0.2);
            want = a * b;
            got = s64_mul(S(a), S(b));
        } else if (op == 1) {
            const double c = rnd(1, 1e5), a = i % 100 ? rnd(1e-20, c * 200) : 0.0;
            want = c + a;
            got = s64_add(S(c), S(a));
        } else if (op == 2) {
            const double c = rnd(0.1, 1);
            double a = i & 1 ? rnd(1e-20, c) : c * (1 - rnd(1e-16, 0.5));
            if (a > c || i % 1000 == 0) a = c;
            want = c - a;
            got = s64_sub(S(c), S(a));
        } else {
            const double a = rnd(1e-17, 1e5), b = rnd(1, 1e5);
            want = a / b;
            got = s64_div(S(a), S(b));
        }
        bad += s64_to_bits(got) != B(want);
    }
    return bad;
}
static double horner(const double *c, double x)
{
    double r = c[7];
    for (int i = 6; i >= 0; --i) {
        volatile double p = r * x;
        r = p + c[i];
    }
    return r;
}
extern "C" long central(uint32_t z0, uint32_t step, int n)
{
    const double a[8] = {3.3871328727963666080e0, 1.3314166789178437745e+2, 1.9715909503065514427e+3, 1.3731693765509461125e+4,
                         4.5921953931549871457e+4, 6.7265770927008700853e+4, 3.3430575583588128105e+4, 2.5090809287301226727e+3};
    const double b[8] = {1.0, 4.2313330701600911252e+1, 6.8718700749205790830e+2, 5.3941960214247511077e+3,
                         2.1213794301586595867e+4, 3.9307895800092710610e+4, 2.8729085735721942674e+4, 5.2264952788528545610e+3};
    long bad = 0;
    for (int i = 0; i < n; ++i) {
        const uint32_t z = z0 + (uint32_t)i * step;
        if (z < 1 || z > 4294967087u) continue;
        uint64_t ub;
        bool c;
        const uint64_t got = as241_central(z, &ub, &c);
        volatile double u = (double)z * (1.0 / 4294967088.0), q = u - 0.5;
        bad += ub != B(u) || c != (std::fabs(q) <= 0.425);
        if (std::fabs(q) > 0.425) continue;
        volatile double qq = q * q, r = 0.180625 - qq, qn = q * horner(a, r), v = qn / horner(b, r);
        bad += got != B(v);
    }
    return bad;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("soft64")
    (d / "s.cpp").write_text(SRC)
    so = str(d / "s.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, PKG_NAME, "csrc"), str(d / "s.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.ops.restype = lib.central.restype = ctypes.c_long
    lib.central.argtypes = [ctypes.c_uint32, ctypes.c_uint32, ctypes.c_int]
    return lib


@pytest.mark.parametrize("op", [0, 1, 2, 3], ids=["mul", "add", "sub", "div"])
def test_operations_round_as_doubles(lib, op):
    assert lib.ops(op, 2_000_000) == 0


@pytest.mark.parametrize("z0,step,n", [(1, 1, 100_000), (4294967087 - 99_999, 1, 100_000), (2147483544 - 200_000, 1, 400_000),
                                       (322122531 - 1000, 1, 2000), (3972844556 - 1000, 1, 2000), (7, 2147, 2_000_000)])
def test_central_branch_bits(lib, z0, step, n):
    """The ends of the stream's integers, the middle (q through 0), the branch's edges, and a sweep of all."""
    assert lib.central(z0, step, n) == 0
