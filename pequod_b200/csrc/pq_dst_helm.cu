// pq_dst_helm.cu -- The inverse row DST of the stand-alone solves.
#include "pq_dst.cuh"

namespace pq {

cudaError_t launch_dst_helm(const LaunchSet& ls, int f32, cudaStream_t st) {
    return f32 ? launch_dst<float, PRO_PLAIN, EPI_HELM>(ls, st) : launch_dst<double, PRO_PLAIN, EPI_HELM>(ls, st);
}

}  // namespace pq
