// pq_dst_step.cu -- The forward row DST with the CABARET predictor, the beta step and the projection.
#include "pq_dst.cuh"

namespace pq {

cudaError_t launch_dst_step(const LaunchSet& ls, int f32, cudaStream_t st) {
    return f32 ? launch_dst<float, PRO_STEP, EPI_SPEC>(ls, st) : launch_dst<double, PRO_STEP, EPI_SPEC>(ls, st);
}

}  // namespace pq
