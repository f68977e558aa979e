// Pieces the FP32 kernels with rate blocks share: the reverse over one block and
// the column sums.
//
// The reverse runs in units of sigma = lambda sqrt(delta): with X = 1/(delta L),
// t = 1/(X + 1), y = (drift sum + normal term)/sqrt(delta) a cell is
//   X *= 2^(a y + c), y -= sigma t, S += sigma Pb, Pb += sigma (1 - t) t S,
//   vega_sigma += Pb (y - sigma) + t S        (a = sigma log2 e, c = -sigma a/2)
// so one constant serves where lambda, delta lambda and delta^2 lambda stood;
// vega_lambda = sqrt(delta) vega_sigma, applied to the block's sums.
#pragma once

#include "lmm_device.cuh"

namespace lmm {
namespace {

struct BlockStep {
    float y, S;
};

// Reverse steps n .. n-G+1 over the rates LO .. LO+H-1 in X[], Pb[]: cell (n-g,
// i+g) at position i. kr and vg point at step n's constants and vega rows of local
// position 0. A vega row stays in registers from position j to j-2(G-1) and takes
// one read-modify-write. When every step is active at the bottom rate (LO > n) the
// body runs to its last position and flushes the rows still open; otherwise it is
// left below the lowest active position (the open rows hold no-op cells of spare
// rows). With CK, rates j > tl are replaced by rs[j*B] after their last cell.
template <int H, int B, int G, bool CK>
__device__ __forceinline__ void rev_block(float (&X)[H], float (&Pb)[H], BlockStep (&st)[G], const float4 *kr, float *vg,
                                          int n, int LO, const float *rs, int tl)
{
    constexpr int JMAX = H + G - 2, W = 2 * G - 1;
    float A[W], C[W], Sg[W], acc[W];
    auto load = [&](int j) {
        const float4 q = kr[j];
        A[j % W] = q.x;
        C[j % W] = q.y;
        Sg[j % W] = q.z;
    };
#pragma unroll
    for (int j = H; j <= JMAX; ++j) {
        load(j);
        acc[j % W] = 0.0f;
    }
    const bool full = LO > n;
    const int imin = n - 2 * G + 3 - LO;     // lowest local position with an active cell
#pragma unroll
    for (int i = H - 1; i >= -(G - 1); --i) {
        if (!full && i < imin) return;
        if (i >= 0) {
            load(i);
            acc[i % W] = 0.0f;
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
            if (i + g >= 0 && i + g <= H - 1) {
                const int j = (i + 2 * g) % W, x = i + g;
                const float xn = X[x] * ex2_approx(fmaf(A[j], st[g].y, C[j]));
                const float t = rcp_approx(xn + 1.0f);
                const float h = st[g].y - Sg[j];
                st[g].y = fmaf(-Sg[j], t, st[g].y);
                st[g].S = fmaf(Sg[j], Pb[x], st[g].S);
                const float tS = t * st[g].S;
                acc[j] += fmaf(Pb[x], h, tS);
                Pb[x] = fmaf(fmaf(-Sg[j], t, Sg[j]), tS, Pb[x]);
                X[x] = xn;
            }
        }
        const int jf = i + 2 * (G - 1);
        if (jf >= 0 && jf <= JMAX) vg[jf * B] += acc[jf % W];
        const int jr = i + G - 1;
        if (CK && jr >= 0 && jr <= H - 1 && jr > tl) X[jr] = rs[jr * B];
    }
    if (full) {
#pragma unroll
        for (int j = 0; j < G - 1; ++j) vg[j * B] += acc[j % W];
    }
}

// Column sums of a warp's 32 paths: lane handles outputs k = lane, lane+32, ...,
// rows t and t+16 in the halves of packed TwoSums (half the additions: 256 curves
// x 16,384 paths 9.46 -> 9.19 ms); the (t+lane)&31 rotation keeps the lanes on 32
// different banks. Adds sums and sums of squares into FP64 accumulators.
template <int B>
__device__ __forceinline__ void column_sums(int nn, const float *vg, int warp, int lane, double *acc, int nout, int off)
{
    for (int k = lane; k < nn; k += 32) {
        const float *col = vg + k * B + warp * 32;
        P2 a = 0, c = 0, a2 = 0;
#pragma unroll 8
        for (int t = 0; t < 16; ++t) {
            const P2 x = p2(col[(t + lane) & 31], col[(t + 16 + lane) & 31]);
            const P2 s = add2(a, x), v = sub2(s, a);
            c = add2(c, add2(sub2(a, sub2(s, v)), sub2(x, v)));
            a = s;
            a2 = fma2(x, x, a2);
        }
        float s, s1, e, e1, q, q1;
        unpack(a, s, s1);
        unpack(c, e, e1);
        unpack(a2, q, q1);
        two_sum_acc(s, e, s1);
        acc[off + k] += (double)s + (double)__fadd_rn(e, e1);
        acc[nout + off + k] += (double)__fadd_rn(q, q1);
    }
}

}  // namespace
}  // namespace lmm
