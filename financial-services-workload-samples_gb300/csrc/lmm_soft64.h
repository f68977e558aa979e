// Binary64 multiply, add, subtract and divide with round-to-nearest-even in
// integer arithmetic, for the positive, normal, moderate numbers of the AS241
// central branch (lmm_mrg.cu), host and device.
//
// GB300 issues 1.7 DMUL or DADD lanes per clock and SM; a rounded product here
// is about 20 integer instructions and a rounded sum about 25 (128 issue slots
// a clock), so the sequence of rounded operations that defines the generator's
// numbers keeps every bit and leaves the FP64 pipe.
//
// A number is m 2^e with 2^52 <= m <= 2^53 (m = 2^53 after a rounding carry is
// left as it is), or m = 0.
#pragma once

#include <cstdint>
#include <cstring>

#include "lmm_fix64.h"

namespace lmm {

struct S64 {
    uint64_t m;
    int e;
};

// The positive normal double of bits b.
LMM_HD constexpr S64 s64_bits(uint64_t b)
{
    return S64{(b & 0xfffffffffffffull) | (1ull << 52), (int)(b >> 52) - 1075};
}

LMM_HD uint64_t s64_to_bits(S64 a) { return a.m == 0 ? 0 : a.m + ((uint64_t)(uint32_t)(a.e + 1074) << 52); }

// The full product a b.
LMM_HD void s64_mul128(uint64_t a, uint64_t b, uint64_t &hi, uint64_t &lo)
{
    const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
    const uint64_t p0 = (uint64_t)al * bl;
    const uint64_t p1 = (uint64_t)al * bh + (p0 >> 32);
    const uint64_t p2 = (uint64_t)ah * bl + (uint32_t)p1;
    hi = (uint64_t)ah * bh + (p1 >> 32) + (p2 >> 32);
    lo = (p2 << 32) | (uint32_t)p0;
}

// m + (1 if the fraction rem 2^-64 rounds it up).
LMM_HD uint64_t s64_round(uint64_t m, uint64_t rem)
{
    const uint64_t up = (rem >> 63) & ((uint64_t)((rem << 1) != 0) | (m & 1));
    return m + up;
}

LMM_HD S64 s64_mul(S64 a, S64 b)
{
    uint64_t hi, lo;
    s64_mul128(a.m, b.m << 11, hi, lo);             // a.m b.m 2^11; hi in [2^51, 2^53]
    const int n = (int)(hi >> 52) != 0;             // 53 bits already
    const uint64_t m = n ? hi : (hi << 1) | (lo >> 63), rem = n ? lo : lo << 1;
    return S64{s64_round(m, rem), a.e + b.e + 52 + n};
}

// v 2^e rounded to 53 bits, v >= 2^53; from 2^54 its lowest bit may be a sticky bit.
LMM_HD S64 s64_norm(uint64_t v, int e)
{
    const int d = 11 - fx_clz(v);                   // bits to drop, at least 1
    const uint64_t rem = v << (64 - d);
    return S64{s64_round(v >> d, rem), e + d};
}

// v 2^s in integer units, bits below the unit collected in the lowest bit.
LMM_HD uint64_t s64_align(uint64_t v, int s)
{
    if (s >= 0) return v << s;
    const int r = -s;
    if (r > 63) return v != 0;
    return (v >> r) | (uint64_t)((v << (64 - r)) != 0);
}

// c + a for c with 2^52 <= c.m < 2^53 and a < 2^9 c.
LMM_HD S64 s64_add(S64 c, S64 a)
{
    return s64_norm((c.m << 2) + s64_align(a.m, a.e - c.e + 2), c.e - 2);
}

// c - a for a <= c and c with 2^52 <= c.m < 2^53.
LMM_HD S64 s64_sub(S64 c, S64 a)
{
    const int s = a.e - c.e + 7;                    // a in units of 2^(c.e - 7): floor and sticky bit
    const uint64_t lost = s >= 0 ? 0 : s < -63 ? a.m : a.m << (64 + s);
    const uint64_t fl = s >= 0 ? a.m << s : s < -63 ? 0 : a.m >> -s;
    const uint64_t sticky = lost != 0;
    const uint64_t v = (c.m << 7) - fl - sticky;    // c - a = v + (a fraction if sticky)
    if (v >= (1ull << 53)) return s64_norm(v | sticky, c.e - 7);
    const int n = v ? fx_clz(v) - 11 : 0;           // a > c/2 here: nothing below the unit, exact
    return S64{v << n, c.e - 7 - n};
}

// a / b.
LMM_HD S64 s64_div(S64 a, S64 b)
{
    const bool less = a.m < b.m;
    const uint64_t am = less ? a.m << 1 : a.m;      // am / bm in [1, 2)
    const uint64_t r = fx_recip(b.m << 10);         // 2^114 / b.m to a few units
    uint64_t q = fx_mulhi_full(am << 3, r);         // am 2^53 / b.m to within 2
    int64_t rem = (int64_t)((am << 53) - q * b.m);
    if (rem < 0) { rem += (int64_t)b.m; --q; }
    if (rem < 0) { rem += (int64_t)b.m; --q; }
    if (rem >= (int64_t)b.m) { rem -= (int64_t)b.m; ++q; }
    if (rem >= (int64_t)b.m) { rem -= (int64_t)b.m; ++q; }
    const uint64_t f = (q << 63) | (uint64_t)(rem != 0);
    return S64{s64_round(q >> 1, f), a.e - b.e - 52 - (less ? 1 : 0)};
}

LMM_HD S64 s64_of(double x)
{
#if defined(__CUDA_ARCH__)
    return s64_bits((uint64_t)__double_as_longlong(x));
#else
    uint64_t b;
    memcpy(&b, &x, 8);
    return s64_bits(b);
#endif
}

// c + a on the FP64 pipe.
LMM_HD S64 s64_dadd(S64 c, S64 a)
{
    const double x = fx_bits(s64_to_bits(c)), y = fx_bits(s64_to_bits(a));
#if defined(__CUDA_ARCH__)
    return s64_of(__dadd_rn(x, y));
#else
    return s64_of(x + y);
#endif
}

// The rounded operations of PPND16's central branch (M. J. Wichura, Applied
// Statistics 37(3), 1988, AS241) for the uniform u = z / (m1 + 1) of MRG32k3a:
// u = z (1/4294967088), q = u - 1/2 (to *tail: the bits of u) and, for |q| <=
// 0.425, r = 0.180625 - q^2 and q num(r) / den(r), each operation rounded to
// binary64 as plain double code evaluates it. Returns the bits of the result;
// *central says whether the branch applies. The numerator's sums run on the FP64
// pipe beside the integer ones (GB300, 167,772,160 normals: every sum in
// integers 9.88 ms, the numerator's on the FP64 pipe 8.63, both polynomials' 8.89).
LMM_HD uint64_t as241_central(uint32_t z, uint64_t *ubits, bool *central)
{
    const S64 a[8] = {s64_of(3.3871328727963666080e0), s64_of(1.3314166789178437745e+2), s64_of(1.9715909503065514427e+3),
                      s64_of(1.3731693765509461125e+4), s64_of(4.5921953931549871457e+4), s64_of(6.7265770927008700853e+4),
                      s64_of(3.3430575583588128105e+4), s64_of(2.5090809287301226727e+3)};
    const S64 b[8] = {s64_of(1.0), s64_of(4.2313330701600911252e+1), s64_of(6.8718700749205790830e+2),
                      s64_of(5.3941960214247511077e+3), s64_of(2.1213794301586595867e+4), s64_of(3.9307895800092710610e+4),
                      s64_of(2.8729085735721942674e+4), s64_of(5.2264952788528545610e+3)};
    const int n = fx_clz(z | 1);                                  // z >= 1
    const uint64_t ub = s64_to_bits(s64_mul(S64{(uint64_t)z << (n - 11), 11 - n}, s64_of(1.0 / 4294967088.0)));
    *ubits = ub;
    const S64 u = s64_bits(ub), half = s64_of(0.5);
    const bool low = ub < 0x3fe0000000000000ull;                  // u < 1/2
    const S64 q = s64_sub(low ? half : u, low ? u : half);
    *central = s64_to_bits(q) <= 0x3fdb333333333333ull;           // 0.425
    const S64 r = s64_sub(s64_of(0.180625), s64_mul(q, q));
    S64 num = a[7], den = b[7];
#pragma unroll
    for (int i = 6; i >= 0; --i) {
        num = s64_dadd(a[i], s64_mul(num, r));
        den = s64_add(b[i], s64_mul(den, r));
    }
    if (q.m == 0) return 0;
    return s64_to_bits(s64_div(s64_mul(q, num), den)) | ((uint64_t)low << 63);
}

}  // namespace lmm
