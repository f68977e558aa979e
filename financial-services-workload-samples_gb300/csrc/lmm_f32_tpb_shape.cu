// The rate-block kernel (lmm_f32_tpb.cuh) for shapes at run time, vega rows in
// shared memory: blocks of 512 and 384 threads.
#include "lmm_f32_tpb.cuh"

namespace lmm {

cudaError_t launch_tpb_shape(int B, const DevModel &m, Mode mode, const float *z, uint64_t seed, int64_t path0, bool philox,
                             const Work &w, float *scr, const double *vbar, cudaStream_t s)
{
    return B == 512 ? launch_tpb<0, 0, 512, false>(m, mode, z, seed, path0, philox, w, scr, nullptr, vbar, s)
                    : launch_tpb<0, 0, 384, false>(m, mode, z, seed, path0, philox, w, scr, nullptr, vbar, s);
}

cudaError_t occ_tpb_shape(int B, int nn, int nmat, Mode mode, bool philox, int *blocks)
{
    return B == 512 ? occ_tpb<0, 0, 512, false>(nn, nmat, mode, philox, blocks)
                    : occ_tpb<0, 0, 384, false>(nn, nmat, mode, philox, blocks);
}

}  // namespace lmm
