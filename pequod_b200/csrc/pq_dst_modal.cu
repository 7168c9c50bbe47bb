// pq_dst_modal.cu -- The forward row DST with the projection onto the modes.
#include "pq_dst.cuh"

namespace pq {

cudaError_t launch_dst_modal(const LaunchSet& ls, int f32, cudaStream_t st) {
    return f32 ? launch_dst<float, PRO_MODAL, EPI_SPEC>(ls, st) : launch_dst<double, PRO_MODAL, EPI_SPEC>(ls, st);
}

}  // namespace pq
