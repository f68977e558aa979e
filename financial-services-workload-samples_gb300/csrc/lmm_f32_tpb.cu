// Instances and dispatch of the rate-block kernel (lmm_f32_tpb.cuh).
#include "lmm_f32_tpb.cuh"

#include <algorithm>

namespace lmm {

// The shape whose forward/backward pair runs on a tape (k_tpb): rows of it; 0:
// the backward runs the forward again.
int tpb_tape_rows(int nn, int nmat) { return nn == 80 && nmat == 40 ? nn + nmat : 0; }

// Threads per block: registers allow 512, 384, 256 threads (16, 12, 8 warps an
// SM), the vega rows of a block's paths have to fit in shared memory. 0: no
// block fits.
int tpb_block_threads(int nn, int nmat)
{
    for (int B : {512, 384, 256, 128})
        if (tpb_layout(nn, nmat, Mode::Fused, B).bytes <= 227 * 1024) return B;
    return 0;
}

size_t tpb_scratch_floats_per_block(int nn, int nmat, int ckpt)
{
    const TpbLay L = tpb_layout(nn, nmat, Mode::Fused, 32);      // rows
    const int nck = ckpt > 0 ? (nmat - 1) / ckpt : 0;
    return (size_t)(L.s_ck + nck * kRR * L.nr) * tpb_block_threads(nn, nmat);
}

// Cells that one path walks, no-ops of partly active passes and blocks among them:
// a launch of few paths takes their latency.
int tpb_cells(int nn, int nmat)
{
    int c = 0;
    for (int lo = 0; lo < nn; lo += kFR) c += kFR * std::min(nmat, lo + kFR - 1);
    for (int lo = 0; lo < nn; lo += kRR) c += kRR * std::min(nmat, lo + kRR - 1);
    return c;
}

// Checkpoints are restored between groups of steps.
bool f32_tpb_supports(int nn, int nmat, int ckpt) { return tpb_block_threads(nn, nmat) > 0 && ckpt % kRG == 0; }

// The instances for shapes at run time (lmm_f32_tpb_wide.cu, lmm_f32_tpb_narrow.cu).
cudaError_t launch_tpb_wide(int B, const DevModel &m, Mode mode, const float *z, uint64_t seed, int64_t path0, bool philox,
                            const Work &w, float *scr, const double *vbar, cudaStream_t s);
cudaError_t launch_tpb_narrow(int B, const DevModel &m, Mode mode, const float *z, uint64_t seed, int64_t path0, bool philox,
                              const Work &w, float *scr, const double *vbar, cudaStream_t s);
cudaError_t occ_tpb_wide(int B, int nn, int nmat, Mode mode, bool philox, int *blocks);
cudaError_t occ_tpb_narrow(int B, int nn, int nmat, Mode mode, bool philox, int *blocks);

cudaError_t tpb_blocks_per_sm(int nn, int nmat, Mode mode, bool philox, int *blocks)
{
    if (nn == 80 && nmat == 40) {
        if (mode == Mode::Forward) return occ_tpb<80, 40, 512, Mode::Forward>(nn, nmat, mode, philox, blocks);
        if (mode == Mode::Backward) return occ_tpb<80, 40, 512, Mode::Backward>(nn, nmat, mode, philox, blocks);
        return occ_tpb<80, 40, 512>(nn, nmat, mode, philox, blocks);
    }
    const int B = tpb_block_threads(nn, nmat);
    return B >= 384 ? occ_tpb_wide(B, nn, nmat, mode, philox, blocks) : occ_tpb_narrow(B, nn, nmat, mode, philox, blocks);
}

cudaError_t launch_tpb_any(const DevModel &m, Mode mode, const float *z, uint64_t seed, int64_t path0, bool philox,
                           const Work &w, float *scr, float *tape, const double *vbar, cudaStream_t s)
{
    if (m.nn == 80 && m.nmat == 40) {
        if (mode != Mode::Fused && !tape) return cudaErrorInvalidValue;
        if (mode == Mode::Forward)
            return launch_tpb<80, 40, 512, Mode::Forward>(m, mode, z, seed, path0, philox, w, scr, tape, vbar, s);
        if (mode == Mode::Backward)
            return launch_tpb<80, 40, 512, Mode::Backward>(m, mode, z, seed, path0, philox, w, scr, tape, vbar, s);
        return launch_tpb<80, 40, 512>(m, mode, z, seed, path0, philox, w, scr, nullptr, vbar, s);
    }
    const int B = tpb_block_threads(m.nn, m.nmat);
    return B >= 384 ? launch_tpb_wide(B, m, mode, z, seed, path0, philox, w, scr, vbar, s)
                    : launch_tpb_narrow(B, m, mode, z, seed, path0, philox, w, scr, vbar, s);
}

}  // namespace lmm
