// The rate-block kernel (lmm_f32_tpb.cuh) for shapes at run time, blocks of 256 and 128 threads.
#include "lmm_f32_tpb.cuh"

namespace lmm {

cudaError_t launch_tpb_narrow(int B, const DevModel &m, Mode mode, const float *z, uint64_t seed, int64_t path0, bool philox,
                          const Work &w, float *scr, const double *vbar, cudaStream_t s)
{
    return B == 256 ? launch_tpb<0, 0, 256>(m, mode, z, seed, path0, philox, w, scr, nullptr, vbar, s)
                    : launch_tpb<0, 0, 128>(m, mode, z, seed, path0, philox, w, scr, nullptr, vbar, s);
}

cudaError_t occ_tpb_narrow(int B, int nn, int nmat, Mode mode, bool philox, int *blocks)
{
    return B == 256 ? occ_tpb<0, 0, 256>(nn, nmat, mode, philox, blocks) : occ_tpb<0, 0, 128>(nn, nmat, mode, philox, blocks);
}

}  // namespace lmm
