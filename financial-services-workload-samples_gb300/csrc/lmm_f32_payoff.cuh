// Pieces the thread-per-path FP32 kernels share: a launch's batches and the
// portfolio's payoff and adjoint.
#pragma once

#include "lmm_device.cuh"

namespace lmm {
namespace {

// Paths of batch jb of an item (0 or less: there is none).
__device__ __forceinline__ int batch_left(const Work &w, int item, int jb)
{
    const int64_t p0 = (int64_t)item * w.ipaths + (int64_t)jb * w.bpaths;
    const int64_t iend = min((int64_t)(item + 1) * w.ipaths, w.paths);
    return (int)max(min(iend - p0, (int64_t)w.bpaths), (int64_t)0);
}

// 1/(1 + delta L) with the rounding that bond_ratio leaves, while delta L < 1.
__device__ __forceinline__ F2 bond_ratio2(float il, float delta)
{
    const float t = rcp_approx(il + delta);
    const float hi = bond_ratio_t(il, delta, t);
    return {hi, il > delta ? __fmaf_rn(-delta, t, __fsub_rn(1.0f, hi)) : 0.0f};
}

// Portfolio value, portfolio_b :133-171 and :186-197, from the inverse rates.
// The factors 1/(1+delta L) come from t = 1/(IL + delta) (MUFU reciprocal,
// within 1 ulp) as 1 - delta t while delta L < 1 (within 0.5 + delta L ulp:
// about 0.5 ulp for ordinary rates) and as IL t above (within 2.5 ulp). The
// discount and annuity products, the annuity sum, the swap values and the
// payoff sum are double-FP32 (F2, lmm_device.cuh): FP64-like products on
// the FP32 pipe (FP64 products cost 10% of the fused kernel's time on
// GB300). Returns the discounted value; *disc_out receives the discount
// factor, *mask_out which swaptions (in grouped order) paid, and Bst[m*B] (if
// given) the annuity factors B[m] of :139 rounded to FP32, for the adjoint.
// From the discount product `disc` and the M annuity rates staged in ILst[m*B].
// WIDE: the factors keep their rounding (bond_ratio2).
template <int B, bool WIDE = false>
__device__ __forceinline__ float payoff_forward_staged(int M, F2 disc, float delta, const int *ost, const F2 *oKd,
                                                       const float *oWf, float *disc_out, float *Bst,
                                                       const float *ILst, unsigned long long *mask_out)
{
    F2 b{1.0f, 0.0f}, sb{0.0f, 0.0f}, vs{0.0f, 0.0f};
    unsigned long long mask = 0ull;
#pragma unroll 1
    for (int m = 0; m < M; ++m) {
        if (WIDE)
            b = f2_mul(b, bond_ratio2(ILst[m * B], delta));
        else
            b = f2_mul(b, bond_ratio(ILst[m * B], delta));
        sb = f2_add(sb, b);                                   // annuity / delta
        if (Bst) Bst[m * B] = b.hi;
        const int o1 = ost[m + 1];
#pragma unroll 1
        for (int o = ost[m]; o < o1; ++o) {
            const float sw = f2_swap_value(oKd[o], sb, b);
            if (sw < 0.0f) {
                vs = f2_add(vs, (-100.0f * sw) * oWf[o]);
                mask |= 1ull << o;
            }
        }
    }
    *disc_out = disc.hi;
    *mask_out = mask;
    const F2 v = f2_mul(vs, disc);
    return __fadd_rn(v.hi, v.lo);
}

// Payoff adjoint, portfolio_b :173-184 (with the rate and its adjoint kept
// apart) and :199-209, seeded with vbar = dOut/dV. Replaces the
// staged rates by the log-adjoints L_i dOut/dL_i. Bst[m*B] holds B[m] from the
// forward: rebuilding B[m-1] = B[m](1 + delta L) backwards from the last,
// smallest factor would underflow FP32 on paths whose rates grow large.
template <int B>
__device__ __forceinline__ void payoff_adjoint_stage(int M, float vbar, float disc, const float *Bst, float *ILst,
                                                     unsigned long long mask, float delta, const int *ost,
                                                     const float *oKf, const float *oWf)
{
    const float scale = -vbar * disc * delta;
    float Sb = 0.0f, Bb = 0.0f;
    // rolled: one copy of the code instead of one per maturity (instruction cache)
#pragma unroll 1
    for (int m = M - 1; m >= 0; --m) {
        const float il = ILst[m * B];
        const float t = rcp_approx(il + delta);               // L/(1+delta L)
        const float r = bond_ratio_t(il, delta, t);
        const float Bm = Bst[m * B];
        const int o1 = ost[m + 1];
#pragma unroll 1
        for (int o = ost[m]; o < o1; ++o) {
            if ((mask >> o) & 1ull) {
                Sb -= (100.0f * oKf[o]) * oWf[o];
                Bb -= 100.0f * oWf[o];
            }
        }
        Bb = fmaf(delta, Sb, Bb);
        ILst[m * B] = scale * Bb * Bm * t;
        Bb *= r;
    }
}

}  // namespace
}  // namespace lmm
