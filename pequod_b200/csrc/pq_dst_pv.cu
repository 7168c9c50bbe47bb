// pq_dst_pv.cu -- The inverse row DST with the back-projection to psi.
#include "pq_dst.cuh"

namespace pq {

cudaError_t launch_dst_pv(const LaunchSet& ls, int f32, cudaStream_t st) {
    return f32 ? launch_dst<float, PRO_PLAIN, EPI_PV>(ls, st) : launch_dst<double, PRO_PLAIN, EPI_PV>(ls, st);
}

}  // namespace pq
