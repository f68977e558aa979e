// 64-bit fixed-point LMM cells for the FP64 kernels (lmm_f64.cu), host and device.
//
// What bounds an FP64 cell on GB300 is the FP64 pipe: 2 DFMA lanes per clock
// and SM, against 32 IMAD.WIDE (32 x 32 -> 64 bit) and 64 integer adds, shifts
// or logic operations. A truncated 64 x 64 -> 64-bit product (three
// IMAD.WIDE, 0.1 clocks) costs a fifth of a DFMA and keeps 58 to 64
// fraction bits where a double keeps 53. So the Euler step, which is
// transcendental in FP64 (an exp and a divide per cell), runs here in
// integers, and the FP64 pipe keeps what needs a floating range: the payoff
// and the adjoint sums.
//
// Representation. With sigma_k = lambda_k sqrt(delta), the step n of rate i
// (k = i-n-1) of path_calc_b1 (LiborMarketModel/liborSwaptionGreeks.cpp:66-72)
// is, in x = -log2(delta L) and y = z + sum_j sigma_j t_j (the drift sum with
// the normal term, in units of sqrt(delta)),
//   t = delta L / (1 + delta L) = 1 / (1 + 2^x),  y += sigma_k t,
//   x -= sigma_k log2(e) (y - sigma_k / 2).
// The rate is carried as its logarithm, so the multiplicative update is an
// addition without rounding. Formats (Qm.f: value = integer 2^-f):
//   X = 72 + x in [0, 128)    Q8.56, top bit clear: delta L in (2^-56, 2^72)
//   Y = 16 + y in [0, 32)     Q6.58, top bit clear: |z| < 15.5
//   2^x = Em 2^e with Em in [1, 2) Q2.62; t = r 2^-s, s = max(e, 0), r = 1/D
//   in (1/3, 1] Q0.62, D = 2^-s + Em 2^(e-s) Q2.62 in (1, 3];
//   1 - t = Em r 2^(e-s).
// The upper end matters: drifts feed on high rates. With limits at 2 one path
// in half a million left the range at 80/40 and lambda = 0.2 (its plain FP64
// run alone takes 5 ms), with limits at 256 one in nine of the 160/120
// workload.
// A value outside shows in its top bit; such a path is flagged and run in
// plain FP64 (lmm_f64.cu). Subtracting the step's exact integer increments
// runs it backwards without any error, so the reverse sweep needs no
// trajectory and no checkpoints.
#pragma once

#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define LMM_HD __host__ __device__ __forceinline__
#else
#define LMM_HD inline
#endif

namespace lmm {

constexpr int kFxX = 56, kFxY = 58;     // fraction bits
constexpr int kFxOff = 72;              // X = kFxOff + x
constexpr int kFxTable = 1024;          // 2^(j/1024) entries
constexpr double kFxZMax = 15.5;        // normals beyond take the FP64 path
// sigma log2(e) < 1/2 keeps the cross products of fx_mulhi below 2^64.
constexpr double kFxSigmaMax = 0.34;

// 2^(j/32) and 2^(j/1024), j < 32, Q2.62, rounded to nearest; the 1024-entry
// table is their products.
#if defined(__CUDACC__)
#define LMM_FX_TABLE static __device__ const
#else
#define LMM_FX_TABLE static const
#endif
LMM_FX_TABLE uint64_t kFxHi[32] = {
    0x4000000000000000ull, 0x4166c34c5615d0ecull, 0x42d561b3e6243d8aull, 0x444c0740496d4294ull,
    0x45cae0f1f545eb73ull, 0x47521cc5a2e6a9e0ull, 0x48e1e9b9d588e19bull, 0x4a7a77d47f7b84b1ull,
    0x4c1bf828c6dc54b8ull, 0x4dc69cdceaa72a9cull, 0x4f7a993048d088d7ull, 0x513821818624b40cull,
    0x52ff6b54d8a89c75ull, 0x54d0ad5a753e077cull, 0x56ac1f752150a563ull, 0x5891fac0e95612c8ull,
    0x5a827999fcef3242ull, 0x5c7dd7a3b17dcf75ull, 0x5e8451cfac061b5full, 0x6096266533384a2bull,
    0x62b39508aa836d6full, 0x64dcdec3371793d1ull, 0x6712460a8fc24072ull, 0x69540ec8f895722dull,
    0x6ba27e656b4eb57aull, 0x6dfddbcbed791babull, 0x70666f76154a7089ull, 0x72dc8373be41a454ull,
    0x75606373ee921c97ull, 0x77f25ccdee6d7ae6ull, 0x7a92be8a92436616ull, 0x7d41d96db915019dull,
};
LMM_FX_TABLE uint64_t kFxLo[32] = {
    0x4000000000000000ull, 0x400b18178ba33b14ull, 0x4016321b687027a8ull, 0x40214e0bebbe0c77ull,
    0x402c6be96af2fb58ull, 0x40378bb43b83d3d8ull, 0x4042ad6cb2f445c2ull, 0x404dd11326d6d3b5ull,
    0x4058f6a7ecccd5b6ull, 0x40641e2b5a867bc0ull, 0x406f479dc5c2d058ull, 0x407a72ff844fbb1full,
    0x4085a050ec0a036aull, 0x4090cf9252dd52cfull, 0x409c00c40ec437beull, 0x40a733e675c82816ull,
    0x40b268f9de0183baull, 0x40bd9ffe9d979724ull, 0x40c8d8f50ac09dffull, 0x40d413dd7bc1c5bcull,
    0x40df50b846ef302bull, 0x40ea8f85c2abf60eull, 0x40f5d046456a29b8ull, 0x410112fa25aad99eull,
    0x410c57a1b9fe12f6ull, 0x41179e3d5902e44dull, 0x4122e6cd59676024ull, 0x412e315211e89f86ull,
    0x41397dcbd952c4a6ull, 0x4144cc3b0680fd7aull, 0x41501c9ff05d8654ull, 0x415b6efaede1ac83ull,
};
constexpr uint64_t kFxLog2e = 0xb8aa3b295c17f0bcull;     // Q1.63
// 1024 (2^(R/1024) - 1) = R (k1 + R (k2 + R (k3 + R k4))), R in [0, 1):
// Chebyshev interpolation of (2^x - 1)/x, relative error of 2^x 2^-66.5.
// k1, k2 in units of 2^-64, k3, k4 of 2^-54.
constexpr uint64_t kFxK1 = 0xb17217f7d1cf78fdull, kFxK2 = 0x000f5fdeffc178a1ull;
constexpr uint32_t kFxK3 = 0x38d61193u, kFxK4 = 0x27681u;

LMM_HD uint32_t fx_mulhi32(uint32_t a, uint32_t b)
{
#if defined(__CUDA_ARCH__)
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}

// (a b) >> 64 to within 2 units (lo x lo and the carries below bit 64 left
// out), for a_hi b_lo + a_lo b_hi < 2^64 (both below 2^63, or one small).
LMM_HD uint64_t fx_mulhi(uint64_t a, uint64_t b)
{
    const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
    const uint64_t m = (uint64_t)ah * bl + (uint64_t)al * bh;
    return (uint64_t)ah * bh + (m >> 32);
}

// (a b) >> 64, all four partial products (block set-up only).
LMM_HD uint64_t fx_mulhi_full(uint64_t a, uint64_t b)
{
    const uint64_t ah = a >> 32, al = (uint32_t)a, bh = b >> 32, bl = (uint32_t)b;
    const uint64_t m1 = ah * bl + ((al * bl) >> 32), m2 = al * bh + (uint32_t)m1;
    return ah * bh + (m1 >> 32) + (m2 >> 32);
}

LMM_HD int fx_clz(uint64_t v)
{
#if defined(__CUDA_ARCH__)
    return __clzll((long long)v);
#else
    return __builtin_clzll(v);
#endif
}

LMM_HD double fx_bits(uint64_t b)
{
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)b);
#else
    double d;
    memcpy(&d, &b, 8);
    return d;
#endif
}

// v 2^ex for v != 0, rounded half up.
LMM_HD double fx_double(uint64_t v, int ex)
{
    const int n = fx_clz(v);
    const uint64_t m = (((v << n) >> 10) + 1) >> 1;       // 2^52 <= m <= 2^53
    return fx_bits(m + ((uint64_t)(uint32_t)(ex - n + 1085) << 52));
}

// v 2^-kFxY for a signed v (its lowest bit is set).
LMM_HD double fx_signed(int64_t v)
{
    const uint64_t neg = (uint64_t)(v >> 63);
    const uint64_t m = (((uint64_t)v ^ neg) - neg) | 1u;
    const int n = fx_clz(m);
    const uint64_t f = (((m << n) >> 10) + 1) >> 1;
    return fx_bits((f + ((uint64_t)(uint32_t)(1085 - kFxY - n) << 52)) | (neg & (1ull << 63)));
}

// Entry j of the 2^(j/1024) table, from its two factors.
#if defined(__CUDACC__)
__device__ __forceinline__
#else
inline
#endif
uint64_t fx_table_entry(int j) { return fx_mulhi_full(kFxHi[j >> 5] << 1, kFxLo[j & 31] << 1); }

// 2^frac(X) as Q2.62.
LMM_HD uint64_t fx_exp2(uint64_t X, const uint64_t *tab)
{
    const uint32_t hi = (uint32_t)(X >> 32);
    const uint64_t T = tab[(hi >> (kFxX - 42)) & (kFxTable - 1)], R = X << (74 - kFxX);   // R, Q0.64
    const uint32_t rh = (uint32_t)(R >> 32), rl = (uint32_t)R;
    const uint32_t q3 = fx_mulhi32(kFxK4, rh) + kFxK3;
    const uint64_t q2 = (uint64_t)fx_mulhi32(q3, rh) * 1024u + kFxK2;
    const uint32_t q2h = (uint32_t)(q2 >> 32), q2l = (uint32_t)q2;
    const uint64_t q1 = (uint64_t)q2h * rh + (kFxK1 + fx_mulhi32(q2l, rh) + fx_mulhi32(q2h, rl));
    const uint64_t rho = (X & ((1ull << (kFxX - 10)) - 1)) << (64 - kFxX);   // R/1024, Q0.64
    return T + fx_mulhi(T, fx_mulhi(q1, rho));
}

// r = 1/D, Q0.62, for D Q2.62 in (1, 4): an FP32 reciprocal biased downwards
// (so that e = 1 - D r0 is in [0, 2^-20)) and r = r0 (1 + e + e^2); the cubic
// term left out is below 2^-60 of r.
LMM_HD uint64_t fx_recip(uint64_t D)
{
    const uint32_t dh = (uint32_t)(D >> 32), dl = (uint32_t)D;
#if defined(__CUDA_ARCH__)
    float f;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"(__uint2float_rn(dh)));
    const uint32_t bits = __float_as_uint(__fmaf_rn(f, 1073741312.0f, 1.0f));   // 2^30 (1 - 2^-21)
#else
    const float f = 1.0f / (float)dh;
    const float g = __builtin_fmaf(f, 1073741312.0f, 1.0f);
    uint32_t bits;
    memcpy(&bits, &g, 4);
#endif
    const uint32_t r0 = bits << 9;                                   // Q0.32
    const uint64_t phi = (uint64_t)dh * r0 + (((uint64_t)dl * r0) >> 32);
    // e = 2^62 - 1 - phi, Q2.62, below 2^42, as the complement: nvcc 13.0.88
    // drops a carry in 2^63 - phi + x where the low word of phi is 0.
    const uint64_t e = phi ^ ((1ull << 62) - 1);
    const uint32_t es = (uint32_t)(e >> 15);
    const uint64_t g2 = (e | (1ull << 62)) + fx_mulhi32(es, es);     // 1 + e + e^2
    return (uint64_t)r0 * (uint32_t)(g2 >> 32) + (((uint64_t)r0 * (uint32_t)g2) >> 32);
}

// The logistic of a rate X (formats above).
struct FxT {
    uint64_t Em, r;
    uint32_t up, down;      // max(e, 0), max(-e, 0)
};

LMM_HD FxT fx_logistic(uint64_t X, const uint64_t *tab)
{
    const uint32_t e = (uint32_t)(X >> kFxX);
    FxT q;
    q.up = e > kFxOff ? e - kFxOff : 0;
    q.down = e < kFxOff ? kFxOff - e : 0;
    q.Em = fx_exp2(X, tab);
#if defined(__CUDA_ARCH__)
    uint64_t low;                                    // shr clamps: 0 from 64 on
    asm("shr.u64 %0, %1, %2;" : "=l"(low) : "l"(q.Em), "r"(q.down));
#else
    const uint64_t low = q.down < 64 ? q.Em >> q.down : 0;
#endif
    q.r = fx_recip(low + ((1ull << 62) >> q.up));
    return q;
}

// t and 1 - t as doubles.
LMM_HD double fx_t(const FxT &q) { return fx_double(q.r, -62 - (int)q.up); }
LMM_HD double fx_1mt(const FxT &q) { return fx_double(fx_mulhi(q.Em, q.r) + 1, -60 - (int)q.down); }

// Constants of one time to maturity k. sigma = sn 2^(wx+2) with sn in
// [1/4, 1/2) (0 for sigma = 0).
struct FxConst {
    uint64_t a, c;      // sigma log2(e) / 4 Q0.64; sigma log2(e) (16 + sigma/2), Q8.56
    uint64_t s16, h;    // sigma / 16 Q0.64; 16 + sigma Q6.58
    uint64_t sn;        // normalised sigma Q0.64
    double sg;          // sigma
    int64_t wx, pad;
};

// sigma in [0, kFxSigmaMax]. c and h also take out the mean of what the steps
// truncate: a product loses 0.75 units on average and the shift of a drift
// term about half a unit of Y, k + 1 times before Y is read at the cell. (Left
// in, the means over paths were off by up to 8e-16 at 160/120, a systematic
// part that more paths do not average out.)
LMM_HD FxConst fx_const(double sigma, int k)
{
    FxConst f;
    const uint64_t s = (uint64_t)(sigma * 18446744073709551616.0);   // Q0.64 (exact from 2^-11 up)
    const uint64_t a = fx_mulhi_full(s, kFxLog2e) << 1, as = fx_mulhi_full(a, s);
    const double lag = 0.52 * (k + 1);
    const double part = (double)(a & 15) / 16 + (double)(as & 511) / 512 - 0.75 - lag * sigma * 0.36067376022224085;
    f.a = a >> 2;
    f.c = (a >> 4) + (as >> 9) + (uint64_t)(int64_t)(part < 0 ? part - 0.5 : part + 0.5);
    f.s16 = s >> 4;
    f.h = (16ull << kFxY) + (s >> 6) - (uint64_t)(lag + 0.5);
    f.sg = sigma;
    uint64_t b;
    memcpy(&b, &sigma, 8);
    f.sn = s ? ((b & 0xfffffffffffffull) | (1ull << 52)) << 10 : 0;
    f.wx = s ? (int64_t)((b >> 52) & 2047) - 1023 : 0;               // sigma = 1.m 2^wx
    f.pad = 0;
    return f;
}

// Y of a normal z, |z| < kFxZMax.
LMM_HD uint64_t fx_normal(double z) { return (uint64_t)((int64_t)(z * 288230376151711744.0) + (16ll << kFxY)); }

// X of v = delta L0 (log2 in FP64, one correction step against 2^x); the top
// bit is set when v lies outside the range.
LMM_HD uint64_t fx_rate(double v, double log2v, const uint64_t *tab)
{
    if (!(log2v > kFxOff - 127.999 && log2v < kFxOff - 0.001)) return 1ull << 63;
    const double unit = 72057594037927936.0;                         // 2^kFxX
    int64_t X = (int64_t)((kFxOff - log2v) * unit);
    uint64_t b;
    memcpy(&b, &v, 8);
    const int ev = (int)((b >> 52) & 2047) - 1023;                   // v = 1.m 2^ev
    const uint64_t mv = ((b & 0xfffffffffffffull) | (1ull << 52)) << 11;   // Q1.63
    const int e = (int)(X >> kFxX) - kFxOff;                           // 2^x = Em 2^e
    const uint64_t P = fx_mulhi_full(mv, fx_exp2((uint64_t)X, tab)); // Q3.61: v 2^x 2^-(ev+e)
    const int64_t one = (int64_t)1 << (61 - (ev + e));               // ev + e is 0 or -1
    const double eps = (double)((int64_t)P - one) / (double)one;     // v 2^x - 1
    return (uint64_t)(X - (int64_t)(eps * 1.4426950408889634 * unit));
}

// The drift term sigma t of a cell, units of Y.
LMM_HD uint64_t fx_drift(const FxT &q, const FxConst &k) { return fx_mulhi(k.s16, q.r) >> q.up; }

// The step of rate X at drift sum Y, and the same undone.
LMM_HD uint64_t fx_step(uint64_t X, uint64_t Y, const FxConst &k) { return X - fx_mulhi(k.a, Y) + k.c; }
LMM_HD uint64_t fx_unstep(uint64_t X, uint64_t Y, const FxConst &k) { return X + fx_mulhi(k.a, Y) - k.c; }

// sigma t (1 - t) of a cell.
LMM_HD double fx_slope(const FxT &q, const FxConst &k)
{
    const uint64_t w = fx_mulhi(fx_mulhi(k.sn, q.r) << 2, fx_mulhi(q.Em, q.r)) + 1;
    return fx_double(w, (int)k.wx - 58 - (int)(q.up + q.down));
}

}  // namespace lmm
