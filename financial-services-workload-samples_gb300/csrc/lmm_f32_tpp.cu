// FP32 thread-per-path LMM kernels: k_tpp for NN=80, NMAT=40 without scratch in
// memory (the no-allocation call), and k_tpq for the fused NN=160, NMAT=120 call.
//
// k_tpp.
// One CUDA thread carries one Monte Carlo path through
//   forward   path_calc_b1   (LiborMarketModel/liborSwaptionGreeks.cpp:34-82)
//   payoff    portfolio_b    (:120-211), adjoint aliasing of :178/:181 fixed
//   reverse   path_calc_b2   (:86-117) plus the vega adjoint (not in the reference)
// with the NN inverse forward rates IL[] = 1/L and the log-adjoints
// Pb[] = L*dV/dL held in registers (the rate index is a compile-time register
// index; the step index is a runtime loop). Carrying 1/L gives
// t = L/(1+delta L) = 1/(IL + delta) from one add and one reciprocal, and
// r = 1/(1+delta L) = 1 - delta t.
//
// Branch-free steps. Step n moves rates i > n only. The per-maturity
// constants are stored with NMAT zero entries in front (k = i-n-1 < 0), so a
// cell with i <= n multiplies IL by 2^0 = 1 and adds 0 to every running sum:
// it is an exact no-op. The forward and the reverse each have ONE unrolled
// body over the rates, cut into chunks (LMM_TPP_CHUNK rates in the forward,
// LMM_TPP_RCHUNK in the reverse): a step enters (forward) or leaves (reverse)
// the body at the chunk holding its first active rate, so at most a chunk
// minus one no-op cells run per step and the code stays small enough for the
// instruction cache.
//
// Reverse sweep without a stored trajectory. With V_i the inclusive drift sum
// of step n (saved per step by the forward), the Euler step runs backwards,
// descending in i as the adjoint needs:
//   IL_{n,i} = IL_{n+1,i} * 2^(a_k (V_i + sqez) + c_k),  V_{i-1} = V_i - delta^2 lambda_k t
// with t = L/(1+delta L), r = 1/(1+delta L). In terms of Pb the reference's
// update (:108-111) becomes
//   S += lambda_k Pb_i,   Pb_i += delta^2 lambda_k t r S     (S is the reference's v1)
// and the vega of cell (n,i), k = i-n-1, is
//   dV/dlambda_k += Pb_i (V_i + sqez - delta lambda_k) + delta^2 t S.
// The kernel carries S' = delta^2 S (S' += delta^2 lambda_k Pb_i, Pb_i +=
// lambda_k r t S'), which saves a multiply per cell. Vega slots of no-op cells
// (k < 0) are spare rows in front of row 0 that are never read; a reverse
// window touches rows k >= 1 - (its chunk of positions), so four suffice.
// The reconstruction is a serial chain (exp -> rcp -> drift sum) per step, so
// steps are processed as a skewed wavefront: cell (n,i) next to cell
// (n-1,i+1), next to (n-2,i+2), ..., G independent chains in one instruction
// stream (G = LMM_TPP_SKEW = 4). Cell (n-g, i+g) uses the constants and vega row
// that cell (n, i+2g) used 2g positions earlier; they are kept in register
// rings (rev_group_window), so each constant is read from shared memory once
// and each vega row gets one read-modify-write per G cells. The forward
// pairs steps the same way (fwd_pair_window).
//
// Cross-path reduction: per warp, each lane sums one output column over the
// warp's 32 paths (shared-memory transpose), then adds into per-warp FP64
// accumulators; each block writes FP64 partial sums that lmm_aux.cu adds in a
// fixed order, so results are bit-reproducible.
#include "lmm_device.cuh"

#include "lmm_f32_payoff.cuh"
#include "lmm_f32_reverse.cuh"

// Threads per block: 235 registers per thread leave room for 8 warps per SM, run as one block of 256 threads so that the block
// barrier keeps all 8 warps on the same stretch of code (GB300, 4,194,304
// paths: 11.73 ms with two 128-thread blocks per SM, 11.54 ms with one of
// 256).
#ifndef LMM_TPP_BLOCK
#define LMM_TPP_BLOCK 256
#endif
// Reverse steps processed together as a skewed wavefront (independent
// reconstruction chains per instruction stream). GB300, 4,194,304 paths: 11.29 ms
// with 2, 11.08 ms with 4 (254 registers, no spills).
#ifndef LMM_TPP_SKEW
#define LMM_TPP_SKEW 4
#endif
// Rates per chunk of the single forward body, and of the reverse body (a
// step group leaves it at the first chunk below its lowest active cell).
// GB300, 4,194,304 paths, fused: reverse chunks of 4 / 8 / 16 rates: 10.98 /
// 11.09 / 11.41 ms, and of 2 see LMM_TPP_FSYNC; forward chunks of 4 were
// slower than 8.
#ifndef LMM_TPP_CHUNK
#define LMM_TPP_CHUNK 8
#endif
#ifndef LMM_TPP_RCHUNK
#define LMM_TPP_RCHUNK 2
#endif
// Forward step pairs between block barriers. GB300, 4,194,304 paths: reverse
// chunks 2 and a barrier every second pair 10.90 -> 10.80 ms.
#ifndef LMM_TPP_FSYNC
#define LMM_TPP_FSYNC 2
#endif
// The running drift sum is Y = V + sqrt(delta) z: one add fewer per cell in each
// phase (4.6% faster on GB300), at the price of accumulating the drift on top of
// the normal term (FP32 vs FP64 Greek errors about 15% larger, still 1e-6 of the
// 1e-4 bound).
// 1: a block barrier per forward step pair and reverse step group, so that
// the warps of a block stay on the same stretch of the unrolled bodies
// (instruction cache). Without it, blocks that run long drift apart: on 256
// curve scenarios x 262,144 paths (GB300) 310 ms without, 243 ms with; equal
// on one scenario.
#ifndef LMM_TPP_SYNC
#define LMM_TPP_SYNC 1
#endif
// The per-maturity constants travel as a kernel parameter and the step windows
// read them from the parameter (constant) bank. GB300, 4,194,304 paths: from
// shared memory 11.04 -> 10.85 ms (232 instead of 252 registers). Kahan-compensated
// vega rows (BF16 compensations beside the rows) took 11.04 -> 12.20 ms and left the
// errors against FP64 unchanged to three digits.
// Positions ahead at which the step windows load the constants of a rate
// (0: at the position that first uses them). GB300, one 256-thread block per SM,
// 4,194,304 paths: 0 / 1 / 2 / 3 ahead: 11.65 / 11.30 / 11.52 / 11.57 ms.
#ifndef LMM_TPP_PREF
#define LMM_TPP_PREF 1
#endif


namespace lmm {
namespace {

__host__ __device__ constexpr int align16(int x) { return (x + 15) & ~15; }

template <int NN, int NMAT>
struct TppLayout {
    static constexpr int B = LMM_TPP_BLOCK;
    static constexpr int NW = B / 32;
    static constexpr int M = NN - NMAT;
    static constexpr int PAD = NMAT;                 // k = i-n-1 >= -NMAT
    // Spare vega rows in front of row 0: a reverse window flushes rows
    // k >= 1 - (its chunk of positions) >= -3.
    static constexpr int VPAD = 4;
    static constexpr int NOUT = 1 + 2 * NN;
    static constexpr int il0 = 0;                                    // float[NN]
    static constexpr int ost = il0 + 4 * NN;                         // int[M+1]
    static constexpr int okf = align16(ost + 4 * (M + 1));           // float[kMaxNopt]
    static constexpr int owf = align16(okf + 4 * kMaxNopt);          // float[kMaxNopt] weights
    static constexpr int okk = align16(owf + 4 * kMaxNopt);          // F2[kMaxNopt]: K delta
    static constexpr int vt = align16(okk + 8 * kMaxNopt);           // float[NMAT][B]
    // per-thread vega rows k = -VPAD..NN-1; the payoff also stages the annuity rates there
    static constexpr int vg = vt + 4 * NMAT * B;                     // float[VPAD+NN][B]
    static constexpr int acc = align16(vg + 4 * (VPAD + NN) * B);    // double[NW][2*NOUT]
    static constexpr int bytes = acc + 8 * NW * 2 * NOUT;
};

// One forward cell (path_calc_b1 :66-72): drift sum and rate update on the
// inverse rate IL = 1/L. k holds the constants of k = i-n-1 (zero for k < 0:
// an exact no-op).
__device__ __forceinline__ void fwd_cell(float &IL, float &V, const float4 &k, float delta)
{
    V = fmaf(k.z, rcp_approx(IL + delta), V);
    IL *= ex2_approx(-fmaf(k.x, V, k.y));
}

// fwd_cell with its reciprocal t = 1/(IL + delta) given.
__device__ __forceinline__ void fwd_cell_t(float &IL, float &V, const float4 &k, float t)
{
    V = fmaf(k.z, t, V);
    IL *= ex2_approx(-fmaf(k.x, V, k.y));
}

// 1: the forward cells of one step at positions 2m and 2m+1 share one MUFU
// reciprocal (rcp_pair). The forward runs two
// MUFU instructions per cell and is bound by the special-function pipe (a
// reciprocal takes it twice as long as an ex2); GB300, split-reverse fused
// kernel: 4,194,304 paths 10.45 -> 10.03 ms, 16.8M Philox paths 43.73 ->
// 42.38 ms.
#ifndef LMM_FWD_RCP2
#define LMM_FWD_RCP2 1
#endif

// Forward steps n and n+1 with one body over positions p (ascending): cell
// (n, p) and cell (n+1, p-1). The second finds IL_{n+1,p-1} written by cell
// (n, p-1) one position earlier, so the two drift chains are independent
// within a position. Cell (n+1, p-1) has k = p-n-3, the constants loaded for
// cell (n, p-2), so each constant is loaded once per two cells (ring C of
// 3+P slots, loaded P positions ahead of its first use).
// Entered at the chunk holding rate n+1; step n+1's cells below its first
// active rate n+2 see zero constants and are exact no-ops.
// With LMM_FWD_RCP2 the cells of one step at positions 2m and 2m+1 share one
// reciprocal: step n's pair is formed at position 2m (both rates still at
// time n), step n+1's at position 2m+1, right after cell (n, 2m+1) (both
// rates then at time n+1), so every step pairs the same positions, as the rate-block
// kernel does, and rounds the same way; neither reciprocal of a pair depends on the drift sums.
template <int NN, int CH, int P>
__device__ __forceinline__ void fwd_pair_window(float (&IL)[NN], const float4 *kcn, float sqez0, float sqez1,
                                                float delta, int n, float &V0, float &V1)
{
    constexpr int R = 3 + P;
    float4 C[R];
    V0 = sqez0;
    V1 = sqez1;
    const int c0 = (n + 1) / CH;
    static_assert(!LMM_FWD_RCP2 || (CH % 2 == 0 && NN % 2 == 0), "reciprocal pairs (2m, 2m+1) inside chunks");
    float t0n = 0.0f, t1n = 0.0f;   // LMM_FWD_RCP2: the second reciprocals of the steps' pairs in flight
#pragma unroll
    for (int c = 0; c * CH < NN; ++c) {
        if (c >= c0) {
            if (c == c0) {
#pragma unroll
                for (int j = c * CH - 2; j < c * CH + P; ++j)
                    if (j >= 0 && j < NN) C[j % R] = kcn[j];
                // step n+1's pair below the chunk: rates inactive in step n, unchanged
                if (LMM_FWD_RCP2 && c * CH >= 2) {
                    float ta;
                    rcp_pair(IL[c * CH - 2] + delta, IL[c * CH - 1] + delta, ta, t1n);
                }
            }
#pragma unroll
            for (int p = c * CH; p < (c + 1) * CH && p < NN; ++p) {
                if (p + P < NN) C[(p + P) % R] = kcn[p + P];
                if (LMM_FWD_RCP2) {
                    float t;
                    if (p % 2 == 0) {
                        rcp_pair(IL[p] + delta, IL[p + 1] + delta, t, t0n);
                    } else {
                        t = t0n;
                    }
                    if (p >= 1) fwd_cell_t(IL[p], V0, C[p % R], t);
                    if (p % 2 == 1) {          // step n+1's pair (p-1, p), both now at time n+1
                        float ta;
                        rcp_pair(IL[p - 1] + delta, IL[p] + delta, ta, t1n);
                        if (p - 1 >= 1) fwd_cell_t(IL[p - 1], V1, C[(p + R - 2) % R], ta);
                    } else if (p - 1 >= 1) {
                        fwd_cell_t(IL[p - 1], V1, C[(p + R - 2) % R], t1n);
                    }
                } else {
                    if (p >= 1) fwd_cell(IL[p], V0, C[p % R], delta);
                    if (p - 1 >= 1) fwd_cell(IL[p - 1], V1, C[(p + R - 2) % R], delta);
                }
            }
        }
    }
    if (LMM_FWD_RCP2)
        fwd_cell_t(IL[NN - 1], V1, C[(NN - 2) % R], t1n);
    else
        fwd_cell(IL[NN - 1], V1, C[(NN - 2) % R], delta);
}

struct RevStep {
    float V, S;         // drift sum with the normal term, delta^2 times the reference's v1
    const float4 *kc;   // kc[i]: constants of k = i-n-1
    float *vg;          // vg[i*B]: this thread's vega slot of k = i-n-1
};

// The reverse windows keep d = -delta*lambda_k beside each constant of their ring
// (one multiply per position, shared by the G cells of the position), and the cell
// forms lambda(1 - delta t) as one FMA, fma(d, t, lambda).
// One reverse cell (path_calc_b2 :105-111 in log-adjoint form) + vega, with
// its constants (k, and d = -delta*k.w) and vega partial sum passed in from the
// window.
template <int NN>
__device__ __forceinline__ void rev_cell(float (&IL)[NN], float (&Pb)[NN], RevStep &s, int i,
                                         const float4 &k, float d, float &acc, float delta)
{
    const float y = s.V;
    const float iln = IL[i] * ex2_approx(fmaf(k.x, y, k.y));
    const float t = rcp_approx(iln + delta);
    s.V = fmaf(-k.z, t, s.V);
    const float pb = Pb[i];
    s.S = fmaf(k.z, pb, s.S);
    const float tS = t * s.S;
    acc += fmaf(pb, y + d, tS);
    Pb[i] = fmaf(fmaf(d, t, k.w), tS, pb);
    IL[i] = iln;
}

// Reverse steps n, n-1, ..., n-G+1 with a single body over positions
// NN-1 .. -(G-1): cell (n-g, i+g) at position i, which finds
// IL_{n-g+1, i+g} written by cell (n-g+1, i+g) one position earlier. With
// j = i+2g, the constants of cell (n-g, i+g) are st[0].kc[j] and its vega row
// is st[0].vg[j*B] (k = j-n-1 of step n): C holds the constants from
// position j+P (load, P positions ahead of the first use) and A the vega
// partial sum from position j, both to position j-2(G-1) (last use, vega
// flush), in rings of 2G-1+P slots indexed j mod (2G-1+P), so that each
// constant is loaded once and each vega row gets one read-modify-write per
// G cells. The body is left at the first
// chunk of CH positions lying wholly below the lowest active position
// n-2G+3. A vega row is valid (k >= 0) for all or none of its G
// contributors, and all contributors of a valid row sit at or above that
// position, so leaving there is exact: the rows still open are spare rows
// (k < 0), which are never read.
template <int NN, int B, int G, int CH, int P>
__device__ __forceinline__ void rev_group_window(float (&IL)[NN], float (&Pb)[NN], RevStep (&st)[G],
                                                 float delta, int n)
{
    constexpr int JMAX = NN + G - 2;
    constexpr int W = 2 * G - 1 + P;
    const float4 *kc = st[0].kc;
    float *vg = st[0].vg;
    float4 C[W];
    float D[W];
    float A[W];
#pragma unroll
    for (int j = NN - P; j <= JMAX; ++j) {
        C[j % W] = kc[j];
        D[j % W] = -delta * C[j % W].w;
        if (j >= NN) A[j % W] = 0.0f;
    }
    const int imin = n - 2 * G + 3;
#pragma unroll
    for (int q = 0; q * CH < NN + G - 1; ++q) {
        const int top = NN - 1 - q * CH;
        if (top < imin) return;
#pragma unroll
        for (int i = top; i > top - CH && i >= -(G - 1); --i) {
            if (i - P >= 1) {
                C[(i - P) % W] = kc[i - P];
                D[(i - P) % W] = -delta * C[(i - P) % W].w;
            }
            if (i >= 1) A[i % W] = 0.0f;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                if (i + g >= 1 && i + g <= NN - 1) {
                    const int j = i + 2 * g;
                    rev_cell<NN>(IL, Pb, st[g], i + g, C[j % W], D[j % W], A[j % W], delta);
                }
            }
            const int jf = i + 2 * (G - 1);
            if (jf >= 1 && jf <= JMAX) vg[jf * B] += A[jf % W];
        }
    }
}

template <int NN, int NMAT, int B>
__device__ __forceinline__ float payoff_forward(const float (&IL)[NN], float delta, const int *ost,
                                                const F2 *oKd, const float *oWf, float *disc_out,
                                                float *Bst, float *ILst, unsigned long long *mask_out)
{
    constexpr int M = NN - NMAT;
    F2 disc{1.0f, 0.0f};
#pragma unroll
    for (int n = 0; n < NMAT; ++n) disc = f2_mul(disc, bond_ratio(IL[n], delta));
    // The annuity recursion runs as a rolled loop over the rates staged in
    // shared memory: one copy of its code instead of one per maturity
    // (instruction cache).
#pragma unroll
    for (int m = 0; m < M; ++m) ILst[m * B] = IL[NMAT + m];
    return payoff_forward_staged<B>(M, disc, delta, ost, oKd, oWf, disc_out, Bst, ILst, mask_out);
}

template <int NN, int NMAT, int B>
__device__ __forceinline__ void payoff_adjoint(const float (&IL)[NN], float (&Pb)[NN], float vbar,
                                               float V, float disc, const float *Bst, float *ILst,
                                               unsigned long long mask, float delta,
                                               const int *ost, const float *oKf, const float *oWf)
{
    constexpr int M = NN - NMAT;
    payoff_adjoint_stage<B>(M, vbar, disc, Bst, ILst, mask, delta, ost, oKf, oWf);
#pragma unroll
    for (int m = 0; m < M; ++m) Pb[NMAT + m] = ILst[m * B];
    const float vs = -vbar * V * delta;
#pragma unroll
    for (int n = 0; n < NMAT; ++n) {
        Pb[n] = vs * rcp_approx(IL[n] + delta);
    }
}

// Forward over all steps, in skewed pairs.
template <int NN, int NMAT>
__device__ __forceinline__ void forward_all(float (&IL)[NN], const float4 *kc0, const float *zp, float sqd, float delta,
                                            float *vt_s)
{
    constexpr int B = LMM_TPP_BLOCK;
    static_assert(NMAT % 2 == 0, "paired forward steps");
    float4 zq, zq_next = zquad<false, NMAT>(zp, 0, 0, 0);
    for (int n = 0; n < NMAT; n += 2) {
        if (LMM_TPP_SYNC && (n % (2 * LMM_TPP_FSYNC)) == 0) __syncthreads();
        if ((n & 3) == 0) {
            zq = zq_next;
            if ((n >> 2) + 1 < NMAT / 4) zq_next = zquad<false, NMAT>(zp, 0, 0, (n >> 2) + 1);
        }
        const float sqez0 = sqd * ((n & 2) ? zq.z : zq.x);
        const float sqez1 = sqd * ((n & 2) ? zq.w : zq.y);
        float V0, V1;
        fwd_pair_window<NN, LMM_TPP_CHUNK, LMM_TPP_PREF>(IL, kc0 - (n + 1), sqez0, sqez1, delta, n, V0, V1);
        vt_s[n * B] = V0;
        vt_s[(n + 1) * B] = V1;
    }
}

// Reverse over all steps, in groups of G steps from the last. The drift sums carry
// the normal term: the reverse needs no normals.
template <int NN, int NMAT>
__device__ __forceinline__ void reverse_all(float (&IL)[NN], float (&Pb)[NN], const float4 *kc0, float *vg0, float delta,
                                            const float *vt_s)
{
    constexpr int G = LMM_TPP_SKEW, B = LMM_TPP_BLOCK;
    static_assert(NMAT % G == 0 && (G == 2 || G == 4), "whole step groups");
    static_assert(LMM_TPP_RCHUNK - 1 <= TppLayout<NN, NMAT>::VPAD, "the windows' spare vega rows lie inside the table");
    for (int n = NMAT - 1; n > 0; n -= G) {
        if (LMM_TPP_SYNC) __syncthreads();
        RevStep st[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int m = n - g;
            st[g].V = vt_s[m * B];
            st[g].S = 0.0f;
            st[g].kc = kc0 - (m + 1);
            st[g].vg = vg0 - (m + 1) * B;
        }
        rev_group_window<NN, B, G, LMM_TPP_RCHUNK, LMM_TPP_PREF>(IL, Pb, st, delta, n);
    }
}

// The per-maturity constants with NMAT zero rows in front (k = i-n-1 < 0),
// passed by value as a kernel parameter.
template <int NN, int NMAT>
struct TppConst {
    float4 v[NMAT + NN];
};

template <int NN, int NMAT>
__global__ void __launch_bounds__(LMM_TPP_BLOCK, 1)
k_tpp(const DevModel m, const float *__restrict__ z, const Work w, const __grid_constant__ TppConst<NN, NMAT> kp)
{
    using Lay = TppLayout<NN, NMAT>;
    constexpr int B = Lay::B, M = Lay::M, NOUT = Lay::NOUT, PAD = Lay::PAD;
    static_assert(NMAT % 4 == 0, "normals are read in aligned quads");
    static_assert(2 * M <= NN, "annuity staging rows inside the vega rows");
    extern __shared__ __align__(16) unsigned char smem[];
    float *il0_s = reinterpret_cast<float *>(smem + Lay::il0);
    int *ost_s = reinterpret_cast<int *>(smem + Lay::ost);
    float *okf_s = reinterpret_cast<float *>(smem + Lay::okf);
    float *owf_s = reinterpret_cast<float *>(smem + Lay::owf);
    F2 *okk_s = reinterpret_cast<F2 *>(smem + Lay::okk);
    float *vt0 = reinterpret_cast<float *>(smem + Lay::vt) + threadIdx.x;
    float *vg_s = reinterpret_cast<float *>(smem + Lay::vg);
    double *acc_s = reinterpret_cast<double *>(smem + Lay::acc);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i <= M; i += B) ost_s[i] = m.opt_start[i];
    for (int i = tid; i < m.nopt; i += B) {
        okf_s[i] = m.optKf[i];
        owf_s[i] = m.optWf[i];
        okk_s[i] = f2_from(m.optKd[i] * m.deltad);
    }
    double *acc = acc_s + warp * 2 * NOUT;
    const float delta = m.delta, sqd = m.sqd;
    const float4 *kc0 = kp.v + PAD;
    float *vgw = vg_s + Lay::VPAD * B, *vg0 = vgw + tid;

    // Units (scenario, item) in a block-stride loop: with a grid of one wave,
    // every block starts together and runs equal units, so the blocks of an
    // SM stay on the same stretch of code (instruction cache).
    const int units = m.nscen * w.items;
    for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
        const int scen = unit / w.items, item = unit % w.items;
        __syncthreads();          // the previous unit's reads of il0/acc are done
        for (int i = tid; i < NN; i += B) il0_s[i] = m.invL0f[scen * NN + i];
        for (int i = tid; i < Lay::NW * 2 * NOUT; i += B) acc_s[i] = 0.0;
        __syncthreads();

        for (int jb = 0; jb < w.ppt; ++jb) {
            const int64_t p0 = ((int64_t)item * w.ppt + jb) * B;
            if (p0 >= w.paths) break;                               // block-uniform
            const bool active = p0 + tid < w.paths;
            const int64_t pc = active ? p0 + tid : w.paths - 1;

            float IL[NN];
            float Pb[NN];
#pragma unroll
            for (int i = 0; i < NN; ++i) IL[i] = il0_s[i];
            forward_all<NN, NMAT>(IL, kc0, z + pc * NMAT, sqd, delta, vt0);

            float disc = 1.0f;
            unsigned long long mask = 0ull;
            // B[m] goes to this thread's vega column, unused until the reverse sweep;
            // the annuity rates to vega rows k = M..2M-1.
            float *Bst = vg0, *ILst = vg0 + M * B;
            const float V = payoff_forward<NN, NMAT, B>(IL, delta, ost_s, okk_s, owf_s, &disc, Bst, ILst, &mask);
            payoff_adjoint<NN, NMAT, B>(IL, Pb, 1.0f, V, disc, Bst, ILst, mask, delta, ost_s, okf_s, owf_s);
#pragma unroll
            for (int k = 0; k < NN; ++k) vg0[k * B] = 0.0f;
            reverse_all<NN, NMAT>(IL, Pb, kc0, vg0, delta, vt0);

            // ---- cross-path reduction of this batch of B paths ----
            const float v = active ? V : 0.0f;
            const float s1 = warp_sum(v), s2 = warp_sum(v * v);
            if (lane == 0) {
                acc[0] += (double)s1;
                acc[NOUT] += (double)s2;
            }
            if (!active) {
#pragma unroll
                for (int k = 0; k < NN; ++k) vg0[k * B] = 0.0f;
            }
            __syncwarp();
            column_sums<B>(NN, vgw, warp, lane, acc, NOUT, 1 + NN);
            __syncwarp();
#pragma unroll
            for (int i = 0; i < NN; ++i) vg0[i * B] = active ? Pb[i] * il0_s[i] : 0.0f;
            __syncwarp();
            column_sums<B>(NN, vgw, warp, lane, acc, NOUT, 1);
            __syncwarp();
        }

        __syncthreads();
        for (int o = tid; o < 2 * NOUT; o += B) {
            double s = 0.0;
#pragma unroll
            for (int q = 0; q < Lay::NW; ++q) s += acc_s[q * 2 * NOUT + o];
            w.partial[(size_t)unit * 2 * NOUT + o] = s;
        }
    }  // units
}

// ---------------------------------------------------------------------------
// k_tpq: the fused long-tenor call (NN = 160, NMAT = 120) with one thread per
// path, the reverse sweep in passes over blocks of 40 rates.
//
// The forward runs in two passes of 80 rates through one copy of the pass
// body (rates 0..79 for the steps that move them, then rates 80..159 for
// every step from the first pass's drift sums at rate 79), so at most 80
// inverse rates are live (255 registers in all: 8 warps, 256 paths per SM,
// the vega rows of 256 paths fill shared memory), and saves, per step, the
// drift sum at the top rate of every block and the rates every ck steps
// (ck = DevModel::ckpt, a multiple of 4); the per-maturity constants are read
// from shared memory. The reverse then runs the blocks one after another from the
// top, in one thread: block b (rates 40b .. 40b+39) for every group of four
// steps with an active cell in it, each step starting from the forward's
// drift sum at the block's top rate and from the suffix sum the block above
// left at its bottom; the rates above a checkpoint time are taken back from
// the checkpoint at group boundaries. At most 40 rates and 40 log-adjoints
// are live in the reverse, the other blocks wait in a per-block scratch, and
// one copy of the 40-position reverse body serves every block (the block's
// offset is a runtime value). The loads of the rates a group hands on (a
// checkpoint, or the block below's parked rates) are issued inside the
// group's body, each right after the group's last cell on its rate, so their
// latency overlaps the rest of the body and the next group's top positions.
// Against two threads per path (k_tp2) there is no pair to balance and no
// barrier per round; the warps of a block run without barriers.
// Scratch per block of the wave, rows of B floats (one per thread):
// [Q][NMAT] block-top drift sums, [Q-1][NMAT] block-bottom suffix sums,
// [NN-H] parked X = 1/(delta L) of the lower blocks, [NN-H] deltas of the upper
// blocks, [NCK][NN] rate checkpoints.
// ---------------------------------------------------------------------------
#ifndef LMM_TPQ_BLOCK
#define LMM_TPQ_BLOCK 256
#endif
// No block barriers: GB300, 160/120, 1,048,576 paths, rates saved every 8 steps, none
// 15.76 ms; every second forward pair 16.17; every second or fourth group 16.01,
// 15.99; every second pair and every group 17.20 (in an earlier build). The
// per-maturity constants in shared memory (one 16-byte load per ring entry) instead
// of the kernel-parameter bank 14.88 -> 14.15 ms; the reverse in units of sigma
// (lmm_f32_reverse.cuh) 14.18 -> 13.81. 384 threads, 168 registers and a window of
// vega rows 13.4 us a thousand paths in one batch, but 22 ms in this call (the warps
// drift apart on the code).
// Steps per reverse group, forward chunk length and the constant prefetch distance
// of the forward (as LMM_TPP_*). GB300, 1,048,576 paths: groups of 8 steps 18.5 ms
// (against 15.77 with 4, in an earlier build); forward chunks of 8, 16, 20 rates
// 13.83, 13.88, 13.88 ms; constants at the position of use or one position ahead
// 13.88, 13.81 ms.
#ifndef LMM_TPQ_SKEW
#define LMM_TPQ_SKEW 4
#endif
#ifndef LMM_TPQ_CHUNK
#define LMM_TPQ_CHUNK 16
#endif
#ifndef LMM_TPQ_PREF
#define LMM_TPQ_PREF 1
#endif

template <int NN, int NMAT>
struct TpqLayout {
    static constexpr int B = LMM_TPQ_BLOCK;
    static constexpr int NW = B / 32;
    static constexpr int H = 40;
    static constexpr int Q = NN / H;
    static constexpr int M = NN - NMAT;
    static constexpr int VPAD = 4;
    static constexpr int NOUT = 1 + 2 * NN;
    static constexpr int il0 = 0;                                    // float[NN]
    static constexpr int ost = align16(il0 + 4 * NN);                // int[M+1]
    static constexpr int okf = align16(ost + 4 * (M + 1));           // float[kMaxNopt]
    static constexpr int owf = align16(okf + 4 * kMaxNopt);          // float[kMaxNopt]
    static constexpr int okk = align16(owf + 4 * kMaxNopt);          // F2[kMaxNopt]
    static constexpr int vg = align16(okk + 8 * kMaxNopt);           // float[VPAD+NN][B] vega rows
    static constexpr int acc = align16(vg + 4 * (VPAD + NN) * B);    // double[NW][2*NOUT]
    static constexpr int kcs = align16(acc + 8 * NW * 2 * NOUT);     // float4[NMAT+NN]: constants of the forward
    static constexpr int krs = kcs + 16 * (NMAT + NN);               // float4[NMAT+NN]: and of the reverse
    static constexpr int bytes = krs + 16 * (NMAT + NN);
    static_assert(bytes <= 227 * 1024, "one block's shared memory");
    static constexpr int s_vt = 0, s_sb = Q * NMAT, s_il = s_sb + (Q - 1) * NMAT, s_d = s_il + NN - H,
                         s_ck = s_d + NN - H;
    static_assert(NN % H == 0 && M == H && H % 4 == 0, "the top block is the annuity rates");
};

// Forward steps n and n+1 over the NP rates LO .. LO+NP-1 held in IL[] at
// local positions 0 .. NP-1, paired as fwd_pair_window: cell (n, p) with
// cell (n+1, p-1). V0, V1 enter as the steps' drift sums below the pass (at
// rate LO-1; the normal term alone for LO = 0) and leave as the sums at its
// top rate; V0c[q], V1c[q] return the sums at local position qH + H-1, the
// top rate of each H-rate block of the pass. kcn points at step n's
// constants for local position 0 (k = LO - n - 1; the NMAT zero rows below
// k = 0 make the inactive cells exact no-ops); nrel = n - LO < NP - 1.
template <int NP, int H, int CH, int P>
__device__ __forceinline__ void fwd_pair_pass(float (&IL)[NP], const float4 *kcn, float delta, int nrel,
                                              float &V0, float &V1, float (&V0c)[NP / H], float (&V1c)[NP / H])
{
    constexpr int R = 3 + P;
    float4 C[R];
#pragma unroll
    for (int q = 0; q < NP / H; ++q) {
        V0c[q] = V0;
        V1c[q] = V1;
    }
    const int c0 = nrel + 1 > 0 ? (nrel + 1) / CH : 0;
    static_assert(!LMM_FWD_RCP2_LONG || (CH % 2 == 0 && NP % 2 == 0), "reciprocal pairs (2m, 2m+1) inside chunks");
    float t0n = 0.0f, t1n = 0.0f;   // LMM_FWD_RCP2_LONG: the second reciprocals of the steps' pairs in flight
#pragma unroll
    for (int c = 0; c * CH < NP; ++c) {
        if (c >= c0) {
            if (c == c0) {
#pragma unroll
                for (int j = c * CH - 2; j < c * CH + P; ++j)
                    if (j < NP) C[(j % R + R) % R] = kcn[j];
                // step n+1's pair below the chunk: rates inactive in step n, unchanged
                if (LMM_FWD_RCP2_LONG && c * CH >= 2) {
                    float ta;
                    rcp_pair(IL[c * CH - 2] + delta, IL[c * CH - 1] + delta, ta, t1n);
                }
            }
#pragma unroll
            for (int p = c * CH; p < (c + 1) * CH && p < NP; ++p) {
                if (p + P < NP) C[(p + P) % R] = kcn[p + P];
                if (LMM_FWD_RCP2_LONG) {     // pairs as fwd_pair_window (LO even)
                    float t;
                    if (p % 2 == 0)
                        rcp_pair(IL[p] + delta, IL[p + 1] + delta, t, t0n);
                    else
                        t = t0n;
                    fwd_cell_t(IL[p], V0, C[p % R], t);
                    if (p % 2 == 1) {
                        float ta;
                        rcp_pair(IL[p - 1] + delta, IL[p] + delta, ta, t1n);
                        fwd_cell_t(IL[p - 1], V1, C[((p - 2) % R + R) % R], ta);
                    } else if (p >= 1) {
                        fwd_cell_t(IL[p - 1], V1, C[((p - 2) % R + R) % R], t1n);
                    }
                } else {
                    fwd_cell(IL[p], V0, C[p % R], delta);
                    if (p >= 1) fwd_cell(IL[p - 1], V1, C[((p - 2) % R + R) % R], delta);
                }
                if (p % H == H - 1) V0c[p / H] = V0;
                if (p >= 1 && (p - 1) % H == H - 1) V1c[(p - 1) / H] = V1;
            }
        }
    }
    if (LMM_FWD_RCP2_LONG)
        fwd_cell_t(IL[NP - 1], V1, C[(NP - 2) % R], t1n);
    else
        fwd_cell(IL[NP - 1], V1, C[(NP - 2) % R], delta);
    V1c[NP / H - 1] = V1;
}

template <int NN, int NMAT, bool PHILOX>
__global__ void __launch_bounds__(LMM_TPQ_BLOCK, 1)
k_tpq(const DevModel m, const float *__restrict__ z, uint64_t seed, int64_t path0, const Work w,
      float *__restrict__ scr, const __grid_constant__ TppConst<NN, NMAT> kp)
{
    using Lay = TpqLayout<NN, NMAT>;
    constexpr int B = Lay::B, H = Lay::H, Q = Lay::Q, M = Lay::M, NOUT = Lay::NOUT, PAD = NMAT;
    constexpr int G = LMM_TPQ_SKEW;
    constexpr int PF = LMM_TPQ_PREF;
    static_assert(NMAT % 4 == 0 && NMAT % G == 0 && H % G == 0, "normals in quads, reverse steps in groups");
    constexpr int HF = 2 * H;      // rates per forward pass
    static_assert(NN == 2 * HF && NMAT > HF && NMAT - HF + M == HF, "two forward passes");
    extern __shared__ __align__(16) unsigned char smem[];
    float *il0_s = reinterpret_cast<float *>(smem + Lay::il0);
    int *ost_s = reinterpret_cast<int *>(smem + Lay::ost);
    float *okf_s = reinterpret_cast<float *>(smem + Lay::okf);
    float *owf_s = reinterpret_cast<float *>(smem + Lay::owf);
    F2 *okk_s = reinterpret_cast<F2 *>(smem + Lay::okk);
    float *vg_s = reinterpret_cast<float *>(smem + Lay::vg);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i <= M; i += B) ost_s[i] = m.opt_start[i];
    for (int i = tid; i < m.nopt; i += B) {
        okf_s[i] = m.optKf[i];
        owf_s[i] = m.optWf[i];
        okk_s[i] = f2_from(m.optKd[i] * m.deltad);
    }
    const float delta = m.delta, sqd = m.sqd;
    float4 *kcs = reinterpret_cast<float4 *>(smem + Lay::kcs), *krs = reinterpret_cast<float4 *>(smem + Lay::krs);
    for (int i = tid; i < NMAT + NN; i += B) {           // read by the cells after the unit loop's first barrier
        const int k = i - PAD;
        float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k >= 0) {
            const double sg = m.lamd[k] * m.sqdd, a = sg * 1.4426950408889634;
            r = make_float4((float)a, (float)(-0.5 * a * sg), (float)sg, 0.f);
        }
        kcs[i] = kp.v[i];
        krs[i] = r;
    }
    const float4 *kc0 = kcs + PAD, *kr0 = krs + PAD;
    const float inv_d = (float)(1.0 / m.deltad), inv_sqd = (float)(1.0 / m.sqdd);
    float *vg0 = vg_s + Lay::VPAD * B + tid;
    const int ck = m.ckpt;
    const int nck = ck > 0 ? (NMAT - 1) / ck : 0;
    const int ckd = ck > 0 ? ck : 1;
    const int64_t rows = Lay::s_ck + (int64_t)nck * NN;
    float *sc = scr + (size_t)blockIdx.x * rows * B + tid;          // sc[row * B]
    double *acc_s = reinterpret_cast<double *>(smem + Lay::acc);     // [NW][2*NOUT]
    double *acc = acc_s + warp * 2 * NOUT;
    float *ckp = sc + (size_t)Lay::s_ck * B;                         // checkpoint c, rate i: ckp[(c*NN + i)*B]

    const int units = m.nscen * w.items;
    for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
        const int scen = unit / w.items, item = unit % w.items;
        __syncthreads();          // the previous unit's reads of il0/acc are done
        for (int i = tid; i < NN; i += B) il0_s[i] = m.invL0f[scen * NN + i];
        for (int i = tid; i < Lay::NW * 2 * NOUT; i += B) acc_s[i] = 0.0;
        __syncthreads();

        const int64_t ibase = (int64_t)item * w.ppt * B;
        for (int jb = 0; jb < w.ppt; ++jb) {
            if (ibase + (int64_t)jb * B >= w.paths) break;          // block-uniform
            const int64_t pl = ibase + (int64_t)jb * B + tid;
            const bool active = pl < w.paths;
            const int64_t pc = active ? pl : w.paths - 1;
            const float *zp = PHILOX ? nullptr : z + pc * NMAT;
            const uint64_t gpath = (uint64_t)(path0 + pc);

            float disc = 1.0f, V, vs;
            float X[H], Pb[H];        // the block in the reverse: inverse rates, log-adjoints
            unsigned long long mask = 0ull;
            {
                // ---- forward (path_calc_b1 :34-82) in two passes of HF rates through one copy of
                // the body: pass 0 rates 0 .. HF-1 from the normals, pass 1 rates HF .. NN-1 from
                // pass 0's drift sums at rate HF-1 ----
                F2 dprod{1.0f, 0.0f};          // the discount product, rates 0 .. NMAT-1 in order
                float IL[HF];
                const float *vin = sc + (size_t)(Lay::s_vt + (HF / H - 1) * NMAT) * B;
#pragma unroll 1
                for (int ps = 0; ps < 2; ++ps) {
                    const int LOp = ps * HF;
#pragma unroll
                    for (int i = 0; i < HF; ++i) IL[i] = il0_s[LOp + i];
                    float4 zq = make_float4(0.f, 0.f, 0.f, 0.f), zq_next = zq;
                    float nv0 = 0.0f, nv1 = 0.0f;
                    if (ps == 0) {
                        zq_next = zquad<PHILOX, NMAT>(zp, seed, gpath, 0);
                    } else {
                        nv0 = vin[0];
                        nv1 = vin[B];
                    }
                    for (int n = 0; n < NMAT; n += 2) {
                        float V0, V1;
                        if (ps == 0) {
                            if ((n & 3) == 0) {
                                zq = zq_next;
                                if ((n >> 2) + 1 < NMAT / 4) zq_next = zquad<PHILOX, NMAT>(zp, seed, gpath, (n >> 2) + 1);
                            }
                            V0 = sqd * ((n & 2) ? zq.z : zq.x);     // drift sums from the normal term
                            V1 = sqd * ((n & 2) ? zq.w : zq.y);
                        } else {
                            V0 = nv0;
                            V1 = nv1;
                            if (n + 2 < NMAT) {
                                nv0 = vin[(n + 2) * B];
                                nv1 = vin[(n + 3) * B];
                            }
                        }
                        float V0c[HF / H], V1c[HF / H];
                        if (n - LOp < HF - 1) {
                            fwd_pair_pass<HF, H, LMM_TPQ_CHUNK, PF>(IL, kc0 - (n + 1) + LOp, delta, n - LOp, V0, V1,
                                                                     V0c, V1c);
                        } else {                 // no rate of the pass moves
#pragma unroll
                            for (int q = 0; q < HF / H; ++q) {
                                V0c[q] = V0;
                                V1c[q] = V1;
                            }
                        }
#pragma unroll
                        for (int q = 0; q < HF / H; ++q) {
                            sc[(Lay::s_vt + (ps * (HF / H) + q) * NMAT + n) * B] = V0c[q];
                            sc[(Lay::s_vt + (ps * (HF / H) + q) * NMAT + n + 1) * B] = V1c[q];
                        }
                        if (nck > 0 && (n + 2) % ckd == 0 && n + 2 < NMAT) {
                            // rates i <= n+2 are final from here on: only the others are saved
                            const int c = (n + 2) / ckd - 1;
#pragma unroll
                            for (int i = 0; i < HF; ++i)
                                if (LOp + i > n + 2) ckp[(c * NN + LOp + i) * B] = IL[i] * inv_d;
                        }
                    }
#pragma unroll
                    for (int i = 0; i < HF; ++i) {
                        if (LOp + i < NMAT) {
                            dprod = f2_mul(dprod, bond_ratio(IL[i], delta));
                            sc[(Lay::s_il + LOp + i) * B] = IL[i] * inv_d;
                        }
                    }
                }
                // ---- payoff (portfolio_b :133-171, :186-197) and the annuity adjoint ----
                float *Bst = vg0;
                float *ILst = vg0 + M * B;
#pragma unroll
                for (int m2 = 0; m2 < M; ++m2) ILst[m2 * B] = IL[NMAT - HF + m2];
                V = payoff_forward_staged<B>(M, dprod, delta, ost_s, okk_s, owf_s, &disc, Bst, ILst, &mask);
                payoff_adjoint_stage<B>(M, 1.0f, disc, Bst, ILst, mask, delta, ost_s, okf_s, owf_s);
#pragma unroll
                for (int i = 0; i < H; ++i) {
                    X[i] = IL[NN - HF - H + i] * inv_d;
                    Pb[i] = ILst[i * B];
                }
                vs = -V;
            }
#pragma unroll
            for (int k = 0; k < NN; ++k) vg0[k * B] = 0.0f;

            // ---- reverse: the blocks from the top, each over its groups of steps ----
            for (int b = Q - 1; b >= 0; --b) {
                const int LO = b * H;
                if (b < Q - 1) {          // X holds the block's parked rates (the last group above loaded them)
#pragma unroll
                    for (int i = 0; i < H; ++i) Pb[i] = vs * rcp_approx(X[i] + 1.0f);
                }
                // the block's first group with an active cell (its top rate above the group's lowest step)
                int n0 = NMAT - 1;
                while (LO + H - 1 <= n0 - G + 1) n0 -= G;
                float nv[G], ns[G];   // the next group's restart sums, loaded a group ahead
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    nv[g] = sc[(Lay::s_vt + b * NMAT + n0 - g) * B];
                    ns[g] = b < Q - 1 ? sc[(Lay::s_sb + b * NMAT + n0 - g) * B] : 0.0f;
                }
                for (int n = n0; n > 0; n -= G) {
                    BlockStep st[G];
#pragma unroll
                    for (int g = 0; g < G; ++g) st[g] = {nv[g] * inv_sqd, ns[g]};
                    if (n - G > 0) {
#pragma unroll
                        for (int g = 0; g < G; ++g) {
                            nv[g] = sc[(Lay::s_vt + b * NMAT + n - G - g) * B];
                            ns[g] = b < Q - 1 ? sc[(Lay::s_sb + b * NMAT + n - G - g) * B] : 0.0f;
                        }
                    }
                    // the rates the group hands on that come from memory: a checkpoint at
                    // its end time t (the reverse of steps >= t leaves rates i <= t
                    // untouched), or in a block's last group the block below's parked rates
                    const int t = n - G + 1;
                    const float *rs = sc;
                    int tl = H;
                    if (nck > 0 && t % ckd == 0 && t >= ck) {
                        rs = ckp + (size_t)((t / ckd - 1) * NN + LO) * B;
                        tl = t - LO;
                    } else if (b > 0 && n - G <= 0) {
                        rs = sc + (size_t)(Lay::s_il + LO - H) * B;
                        tl = -1;
                    }
                    rev_block<H, B, G, true>(X, Pb, st, kr0 - (n + 1) + LO, vg0 + (LO - n - 1) * B, n, LO, rs, tl);
                    if (b > 0) {
#pragma unroll
                        for (int g = 0; g < G; ++g) sc[(Lay::s_sb + (b - 1) * NMAT + n - g) * B] = st[g].S;
                    }
                }
                if (b > 0) {
#pragma unroll
                    for (int i = 0; i < H; ++i)
                        sc[(Lay::s_d + LO - H + i) * B] = active ? Pb[i] * il0_s[LO + i] : 0.0f;
                }
            }

            // ---- cross-path reduction of this batch of B paths ----
            {
                const float v = active ? V : 0.0f;
                const float s1 = warp_sum(v), s2 = warp_sum(v * v);
                if (lane == 0) {
                    acc[0] += (double)s1;
                    acc[NOUT] += (double)s2;
                }
            }
            float *vgw = vg_s + Lay::VPAD * B;
            if (!active) {
#pragma unroll
                for (int k = 0; k < NN; ++k) vg0[k * B] = 0.0f;
            }
            __syncwarp();
            column_sums<B>(NN, vgw, warp, lane, acc, NOUT, 1 + NN);
            __syncwarp();
#pragma unroll
            for (int i = 0; i < H; ++i) vg0[i * B] = active ? Pb[i] * il0_s[i] : 0.0f;
#pragma unroll
            for (int i = 0; i < NN - H; ++i) vg0[(H + i) * B] = sc[(Lay::s_d + i) * B];
            __syncwarp();
            column_sums<B>(NN, vgw, warp, lane, acc, NOUT, 1);
            __syncwarp();
        }

        __syncthreads();
        for (int o = tid; o < 2 * NOUT; o += B) {
            double s2 = 0.0;
#pragma unroll
            for (int q = 0; q < Lay::NW; ++q) s2 += acc_s[q * 2 * NOUT + o];
            // vegas per lambda: sqrt(delta) times those per sigma, delta times their squares
            if (o < NOUT ? o >= 1 + NN : o - NOUT >= 1 + NN) s2 *= o < NOUT ? m.sqdd : m.deltad;
            w.partial[(size_t)unit * 2 * NOUT + o] = s2;
        }
    }  // units
}

template <int NN, int NMAT, bool PHILOX>
cudaError_t launch_tpq(const DevModel &m, const float *z, uint64_t seed, int64_t path0, const Work &w,
                       float *scr, cudaStream_t s)
{
    using Lay = TpqLayout<NN, NMAT>;
    auto kern = k_tpq<NN, NMAT, PHILOX>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Lay::bytes);
    if (e != cudaSuccess) return e;
    TppConst<NN, NMAT> kp;
    for (int i = 0; i < NMAT + NN; ++i)
        kp.v[i] = i < NMAT ? make_float4(0.f, 0.f, 0.f, 0.f) : m.kc_host[i - NMAT];
    const unsigned grid = (unsigned)(w.grid > 0 ? w.grid : (int64_t)m.nscen * w.items);
    kern<<<grid, Lay::B, Lay::bytes, s>>>(m, z, seed, path0, w, scr, kp);
    return cudaGetLastError();
}

template <int NN, int NMAT, bool PHILOX>
cudaError_t occ_tpq(int *blocks)
{
    using Lay = TpqLayout<NN, NMAT>;
    auto kern = k_tpq<NN, NMAT, PHILOX>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Lay::bytes);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, kern, Lay::B, Lay::bytes);
}

template <int NN, int NMAT>
cudaError_t launch_tpp(const DevModel &m, const float *z, const Work &w, cudaStream_t s)
{
    using Lay = TppLayout<NN, NMAT>;
    auto kern = k_tpp<NN, NMAT>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Lay::bytes);
    if (e != cudaSuccess) return e;
    TppConst<NN, NMAT> kp;
    for (int i = 0; i < NMAT + NN; ++i)
        kp.v[i] = i < NMAT ? make_float4(0.f, 0.f, 0.f, 0.f) : m.kc_host[i - NMAT];
    const unsigned grid = (unsigned)(w.grid > 0 ? w.grid : (int64_t)m.nscen * w.items);
    kern<<<grid, Lay::B, Lay::bytes, s>>>(m, z, w, kp);
    return cudaGetLastError();
}

template <int NN, int NMAT>
cudaError_t occ_tpp(int *blocks)
{
    using Lay = TppLayout<NN, NMAT>;
    auto kern = k_tpp<NN, NMAT>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Lay::bytes);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, kern, Lay::B, Lay::bytes);
}

}  // namespace

bool f32_tpp_supports(int nn, int nmat) { return nn == 80 && nmat == 40; }

bool f32_tpq_supports(int nn, int nmat) { return nn == 160 && nmat == 120; }

int tpq_block_threads() { return LMM_TPQ_BLOCK; }

size_t tpq_scratch_floats_per_block(int nn, int nmat, int ckpt)
{
    const int H = 40, Q = nn / H;
    const int nck = ckpt > 0 ? (nmat - 1) / ckpt : 0;
    return (size_t)(Q * nmat + (Q - 1) * nmat + 2 * (nn - H) + (size_t)nck * nn) * LMM_TPQ_BLOCK;
}

cudaError_t tpq_blocks_per_sm(bool philox, int *blocks)
{
    return philox ? occ_tpq<160, 120, true>(blocks) : occ_tpq<160, 120, false>(blocks);
}

cudaError_t launch_tpq_any(const DevModel &m, const float *z, uint64_t seed, int64_t path0, bool philox,
                           const Work &w, float *scratch, cudaStream_t s)
{
    return philox ? launch_tpq<160, 120, true>(m, z, seed, path0, w, scratch, s)
                  : launch_tpq<160, 120, false>(m, z, seed, path0, w, scratch, s);
}

int tpp_block_threads() { return LMM_TPP_BLOCK; }

cudaError_t tpp_blocks_per_sm(int *blocks) { return occ_tpp<80, 40>(blocks); }

cudaError_t launch_tpp_any(const DevModel &m, const float *z, const Work &w, cudaStream_t s)
{
    return launch_tpp<80, 40>(m, z, w, s);
}

}  // namespace lmm
