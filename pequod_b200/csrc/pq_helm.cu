// pq_helm.cu -- the Helmholtz (PV-inversion) kernels: what they are, and their
// host entries (the kernels themselves are in pq_dst.cuh and pq_tridiag.cu).
//
// The reference solves, per vertical mode, (d_xx + d_yy - ss) psi = zeta by a
// DST-I along i (FFTPACK sint, qg3p_helmholtz.F90:1370-1591), a tridiagonal
// solve along j with precomputed reciprocal pivots (ge_local, :1028-1059),
// and the inverse DST (helm, :614-769).  Here that is three kernels:
//
//   k_dst (forward)  a CTA per few interior rows: load (optionally apply the
//                    CABARET predictor + beta step and the z_to_modes
//                    projection), scale by 0.5/(ii-1), DST every mode row in
//                    shared memory, write the spectral rows.
//   k_tridiag        a CTA per (mode, KT consecutive wavenumbers): each lane
//                    holds a chunk of one column's rows in registers, and the
//                    forward / backward Thomas recurrences are solved as
//                    chunked first-order linear recurrences (local sweep,
//                    scan of the affine chunk maps, fix-up sweep).  The
//                    same CTA accumulates the domain mean of the solution in
//                    spectral space (psiC of a closed basin is finished by the
//                    inverse DST, a channel's by the last CTA).
//   k_dst (inverse)  a CTA per few rows: inverse DST of every mode row, then
//                    the mass-corrected back-projection (modes_to_z_btcu,
//                    qg3p_diagnostics.F90:615-635) straight into psi.
//
// DST-I of length n = N - 1 (N = ii - 1 = 2^p), FFTPACK convention
// X_k = 2 sum_m x_m sin(m k pi / N): the sequence is pre-twiddled into a real
// sequence c of length N (as sint1 does), c is packed into N/2 complex points
// and transformed by a radix-8/4/2 Stockham FFT, the real-FFT
// split gives C_q = R_q + i I_q, and X_2q = -I_q, X_2q+1 = R_0/2 + sum_{p<=q} R_p
// (the odd outputs are a prefix sum, done as a block scan).
#include "pq_common.cuh"
#include "pq_dst.cuh"
#include "pq_kernels.h"

namespace pq {

int dst_lanes_default(int M, int L, int dir) { return dst_lanes_default_hd(M, L, dir); }
// Batched solves fill the GPU with many members' rows: throughput, not one
// row's latency, bounds them, so units keep 8 values per lane (fewer passes
// and shared-memory round trips per value) up to M = 256, then one warp.
int dst_lanes_batched(int M) {
    const int V = M <= 2 ? 2 : M == 4 ? 4 : M <= 256 ? 8 : M / 32;
    return M / V;
}
int dst_max_threads_host(int V) { return dst_max_threads(V); }
int dst_rows_per_cta_host(int P, int c) { return dst_rows_per_cta(P, c); }

cudaError_t launch_dst_forward(const LaunchSet& ls, int prologue, int f32, cudaStream_t st) {
    switch (prologue) {
        case PRO_PLAIN: return launch_dst_plain(ls, f32, st);
        case PRO_MODAL: return launch_dst_modal(ls, f32, st);
        default: return launch_dst_step(ls, f32, st);
    }
}

cudaError_t launch_dst_inverse(const LaunchSet& ls, int epilogue, int f32, cudaStream_t st) {
    return epilogue == EPI_HELM ? launch_dst_helm(ls, f32, st) : launch_dst_pv(ls, f32, st);
}

}  // namespace pq
