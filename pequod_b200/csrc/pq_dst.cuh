// pq_dst.cuh -- the row-DST kernels and their launch templates (pq_helm.cu says
// what they are part of).  Each pq_dst_*.cu instantiates some of them, so that
// they compile side by side.
#pragma once

#include <type_traits>

#include "pq_common.cuh"
#include "pq_kernels.h"

namespace pq {

enum { PRO_PLAIN = 0, PRO_MODAL = 1, PRO_STEP = 2 };
enum { EPI_SPEC = 0, EPI_HELM = 1, EPI_PV = 2 };

// ---------------------------------------------------------------------------
// Row DSTs: one group of P lanes per (row, mode) unit.
//
// The complex FFT of length M = N/2 is a Stockham FFT in which every lane of
// a group owns V = M / P values per pass: the row is loaded as node pairs and
// stored pre-twiddled (put_pair), each radix-8 (then 4 or 2) pass is a set of
// V/R in-register butterflies, and values cross lanes only through the unit's
// shared-memory row between passes (under __syncwarp or the unit's named
// barrier, never a block barrier).  The real-FFT split and the prefix sum
// of the odd outputs run on V contiguous wavenumbers per lane with one
// segmented warp scan.  V = 8 up to M = 256 (P = M/8 lanes), then 16, 32.
//
// Unit buffer (U scalars per unit): padded complex rows (the pre-twiddled
// sequence and the Stockham passes, index t -> t + t/8), padded real output row
// (index k -> k + 2*(k/16), so that the pair stores of the split are
// bank-conflict free).

__device__ __forceinline__ int cpad(int t) { return t + (t >> 3); }
__device__ __forceinline__ int xpad(int k) { return k + ((k >> 4) << 1); }

template <typename T2> __device__ __forceinline__ T2 c_mi(T2 a) {  // a * (-i)
    T2 r;
    r.x = a.y;
    r.y = -a.x;
    return r;
}

// The FP32 transform's products and sums are written out as the multiply-adds
// they are, so that every instance of a geometry (its lanes at compile time or
// not, one member or many) rounds alike whatever the compiler would contract
// around them: a mixed run is the same alone and merged with others.  (Other
// lanes per unit round differently: the passes' radices follow the values per
// lane, and the prefix sum of the odd outputs is grouped by lane.)
// FP64 leaves the contraction to the compiler, which folds a twiddle product
// into the butterfly's sums (two operations fewer, one rounding fewer).
__device__ __forceinline__ double mad(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float mad(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double2 tw_mul(double2 a, double2 w) { return cmul(a, w); }
__device__ __forceinline__ float2 tw_mul(float2 a, float2 w) {
    return make_float2(__fmaf_rn(a.x, w.x, -__fmul_rn(a.y, w.y)), __fmaf_rn(a.x, w.y, __fmul_rn(a.y, w.x)));
}
// e + w o
__device__ __forceinline__ double2 split_sum(double2 e, double2 w, double2 o) {
    return make_double2(e.x + (w.x * o.x - w.y * o.y), e.y + (w.x * o.y + w.y * o.x));
}
__device__ __forceinline__ float2 split_sum(float2 e, float2 w, float2 o) {
    const float2 t = tw_mul(o, w);
    return make_float2(__fadd_rn(e.x, t.x), __fadd_rn(e.y, __fmaf_rn(w.x, o.y, __fmul_rn(w.y, o.x))));
}

// In-register forward DFT of R points (R = 2, 4, 8), natural order.
template <int R, typename T2> __device__ __forceinline__ void dft_reg(T2* v) {
    if constexpr (R == 2) {
        const T2 a = cadd(v[0], v[1]), b = csub(v[0], v[1]);
        v[0] = a;
        v[1] = b;
    } else if constexpr (R == 4) {
        const T2 t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]), t2 = cadd(v[1], v[3]), t3 = c_mi(csub(v[1], v[3]));
        v[0] = cadd(t0, t2);
        v[1] = cadd(t1, t3);
        v[2] = csub(t0, t2);
        v[3] = csub(t1, t3);
    } else {
        using T = decltype(v[0].x);
        const T c8 = (T)0.70710678118654752440;  // sqrt(2)/2
        const T2 e0 = cadd(v[0], v[4]), e1 = csub(v[0], v[4]), e2 = cadd(v[2], v[6]), e3 = c_mi(csub(v[2], v[6]));
        const T2 E0 = cadd(e0, e2), E1 = cadd(e1, e3), E2 = csub(e0, e2), E3 = csub(e1, e3);
        const T2 o0 = cadd(v[1], v[5]), o1 = csub(v[1], v[5]), o2 = cadd(v[3], v[7]), o3 = c_mi(csub(v[3], v[7]));
        const T2 O0 = cadd(o0, o2), O1 = cadd(o1, o3), O3 = csub(o1, o3);
        T2 O2 = csub(o0, o2);
        // W8^1 = (1 - i)/sqrt2, W8^2 = -i, W8^3 = (-1 - i)/sqrt2
        const T s1x = O1.x + O1.y, s1y = O1.y - O1.x, s3x = O3.y - O3.x, s3y = -(O3.x + O3.y);
        O2 = c_mi(O2);
        v[0] = cadd(E0, O0);
        v[1].x = mad(c8, s1x, E1.x);
        v[1].y = mad(c8, s1y, E1.y);
        v[2] = cadd(E2, O2);
        v[3].x = mad(c8, s3x, E3.x);
        v[3].y = mad(c8, s3y, E3.y);
        v[4] = csub(E0, O0);
        v[5].x = mad(-c8, s1x, E1.x);
        v[5].y = mad(-c8, s1y, E1.y);
        v[6] = csub(E2, O2);
        v[7].x = mad(-c8, s3x, E3.x);
        v[7].y = mad(-c8, s3y, E3.y);
    }
}

// Barrier of one unit's P lanes: the warp (P <= 32) or the unit's warps by a
// named barrier (P > 32; id 1 + uid, never 0, which __syncthreads uses).
__device__ __forceinline__ void unit_sync(int P, int uid) {
    if (P <= 32)
        __syncwarp();
    else
        asm volatile("bar.sync %0, %1;\n" ::"r"(1 + uid), "r"(P) : "memory");
}

// Twiddle tables (built by the host, Member::tw / wsplit, FP32 copies beside):
//   tw      three sections of M entries, one per pass plan (radix 8, then a 4
//           or 2, for V >= 8; radix 4, then a 2, for V = 4; radix 2 for V = 2).
//           A plan's passes follow one another (the first needs none); the
//           pass on sub-transforms of length Ns holds exp(-2 pi i r k / (Ns R))
//           at (r - 1) Ns + k, so lanes with consecutive k read consecutive
//           entries.
//   wsplit  five sections of M entries, V = 2, 4, 8, 16, 32: the split weight
//           of wavenumber q = p V + e at e P + p, again one line per warp.
// (Both were indexed by the angle before: every 16-byte load of the split
// touched 32 lines and those of a pass up to 28, about 40 % of the kernel's
// L1 cycles at 1025 nodes.)
template <int V> __host__ __device__ constexpr int dst_plan() { return V >= 8 ? 0 : V == 4 ? 1 : 2; }
template <int V> __host__ __device__ constexpr int dst_split_section() { return V == 2 ? 0 : V == 4 ? 1 : V == 8 ? 2 : V == 16 ? 3 : 4; }

// One radix-R Stockham pass over the unit's M values (Ns = length of the
// sub-transforms already done).  Lane p owns butterflies j = p + P*b; its
// values v[b*R + r] are the butterfly inputs j + r*(M/R), read from and stored
// to the unit's padded complex row.  tw: this pass's table (unused at Ns = 1).
template <int V, int R, typename T2>
__device__ __forceinline__ void fft_pass(T2* z, int p, int P, int uid, int M, int Ns, int logNs,
                                         const T2* __restrict__ tw) {
    constexpr int logR = (R == 8) ? 3 : (R == 4) ? 2 : 1;
    const int MR = M >> logR;
    T2 v[V];
#pragma unroll
    for (int b = 0; b < V / R; ++b)
#pragma unroll
        for (int r = 0; r < R; ++r) v[b * R + r] = z[cpad(p + P * b + r * MR)];
#pragma unroll
    for (int b = 0; b < V / R; ++b) {
        const int k = (p + P * b) & (Ns - 1);
        if (Ns > 1) {
#pragma unroll
            for (int r = 1; r < R; ++r) v[b * R + r] = tw_mul(v[b * R + r], __ldg(&tw[((r - 1) << logNs) + k]));
        }
        dft_reg<R>(&v[b * R]);
    }
    unit_sync(P, uid);
#pragma unroll
    for (int b = 0; b < V / R; ++b) {
        const int j = p + P * b, k = j & (Ns - 1);
        const int o = ((j >> logNs) << (logNs + logR)) + k;
#pragma unroll
        for (int r = 0; r < R; ++r) z[cpad(o + r * Ns)] = v[b * R + r];
    }
    unit_sync(P, uid);
}

// The pre-twiddled sequence of a row (sint1, qg3p_helmholtz.F90:1404-1413):
// c_k = (x_k - x_{N-k}) + 2 sin(k pi / N) (x_k + x_{N-k}), c_0 = 0, stored
// packed as c_{2t} + i c_{2t+1} in the unit's padded complex row.  Pair t of
// nodes (t, N - t), t = 1..N/2-1, gives c_t and c_{N-t}; pair 0 stands for
// the middle node N/2 (xb = xa) and c_0.
__device__ __forceinline__ int cidx(int k) { return 2 * cpad(k >> 1) + (k & 1); }
template <typename T>
__device__ __forceinline__ void put_pair(T* buf, int t, int N, T xa, T xb, const T* __restrict__ was) {
    const int k = t ? t : N >> 1;
    const T w = __ldg(&was[k]);
    buf[cidx(k)] = mad(w, xa + xb, xa - xb);
    if (t)
        buf[cidx(N - k)] = mad(w, xa + xb, xb - xa);
    else
        buf[0] = (T)0;
}
// One node of the pair (odd: node N - t) by itself, given the other's value.
template <typename T>
__device__ __forceinline__ void put_node(T* buf, int t, bool odd, int N, T own, T other, const T* __restrict__ was) {
    const int k = t ? t : N >> 1;
    if (odd && !t)
        buf[0] = (T)0;
    else
        buf[cidx(odd ? N - t : k)] = mad(__ldg(&was[k]), own + other, own - other);
}
// A unit's own row, straight from global memory (fetch(k) is x_k): V pairs per lane,
// at most eight of them in flight.
template <int V, typename T, typename F>
__device__ __forceinline__ void stage_unit(T* buf, int p, int P, int N, const T* __restrict__ was, F fetch) {
    constexpr int B = V < 8 ? V : 8;
#pragma unroll
    for (int e0 = 0; e0 < V; e0 += B) {
        T xa[B], xb[B];
#pragma unroll
        for (int e = 0; e < B; ++e) {
            const int t = p + P * (e0 + e), k = t ? t : N >> 1;
            xa[e] = fetch(k);
            xb[e] = fetch(N - k);
        }
#pragma unroll
        for (int e = 0; e < B; ++e) put_pair(buf, p + P * (e0 + e), N, xa[e], xb[e], was);
    }
}

// DST-I (FFTPACK sint convention, qg3p_helmholtz.F90:1370-1426) of the row
// whose pre-twiddled sequence the unit buffer holds (put_pair), output X_k
// at buf[xpad(k)], k = 1..N-1.  Every lane of the unit must call this; uid
// names the unit's barrier, utot is P/32 scalars of scratch for units wider
// than a warp.
template <int V, int M, int Ns, typename T2>
__device__ __forceinline__ void fft_passes(T2* z, int p, int uid, const T2* __restrict__ tw) {
    if constexpr (Ns < M) {
        constexpr int rem = M / Ns, R = (V >= 8 && rem >= 8) ? 8 : (V >= 4 && rem >= 4) ? 4 : 2;
        constexpr int logNs = Ns == 1 ? 0 : 31 - __builtin_clz((unsigned)Ns);
        fft_pass<V, R>(z, p, M / V, uid, M, Ns, logNs, tw);
        fft_passes<V, M, Ns * R>(z, p, uid, tw + (Ns > 1 ? (R - 1) * Ns : 0));
    }
}
template <int V, int PC, typename T>
__device__ __forceinline__ void dst_unit(T* buf, int p, int P, int uid, T* utot, int N, int M,
                                         const typename Cplx<T>::type* __restrict__ tw,
                                         const typename Cplx<T>::type* __restrict__ wsp) {
    using T2 = typename Cplx<T>::type;
    constexpr int R0 = V >= 8 ? 8 : V;
    T2* z = reinterpret_cast<T2*>(buf);
    tw += dst_plan<V>() * M;
    wsp += dst_split_section<V>() * M;
    if constexpr (PC > 0) {
        fft_passes<V, V * PC, 1>(z, p, uid, tw);
    } else {
        int Ns = 1, logNs = 0;
        while (Ns < M) {
            const int rem = M >> logNs;
            int done = 2, ldone = 1;
            if (V >= 8 && rem >= 8) {
                if constexpr (V >= 8) fft_pass<V, 8>(z, p, P, uid, M, Ns, logNs, tw);
                done = 8;
                ldone = 3;
            } else if (R0 >= 4 && rem >= 4) {
                if constexpr (R0 >= 4) fft_pass<V, 4>(z, p, P, uid, M, Ns, logNs, tw);
                done = 4;
                ldone = 2;
            } else {
                fft_pass<V, 2>(z, p, P, uid, M, Ns, logNs, tw);
            }
            if (Ns > 1) tw += (done - 1) * Ns;
            Ns *= done;
            logNs += ldone;
        }
    }
    // Real-FFT split on V contiguous wavenumbers q = p*V + e:
    // C_q = E_q + W_q O_q, R_q = Re C_q (halved at q = 0), X_2q = -Im C_q,
    // X_{2q+1} = sum_{s <= q} R_s.
    T Xe[V], Xo[V];
    T run = (T)0;
#pragma unroll
    for (int e = 0; e < V; ++e) {
        const int q = p * V + e;
        const T2 zq = z[cpad(q)];
        const T2 zr = z[cpad((M - q) & (M - 1))];
        const T dx = zq.x - zr.x, dy = zq.y + zr.y;
        T2 E, O;
        E.x = (T)0.5 * (zq.x + zr.x);
        E.y = (T)0.5 * (zq.y - zr.y);
        O.x = (T)0.5 * dy;
        O.y = (T)-0.5 * dx;
        const T2 C = split_sum(E, __ldg(&wsp[e * P + p]), O);
        const T cx = C.x, cy = C.y;
        Xe[e] = (q == 0) ? (T)0 : -cy;
        run += (q == 0) ? (T)0.5 * cx : cx;
        Xo[e] = run;
    }
    // Segmented (width P) exclusive scan of the lanes' totals: in the warp
    // (or P-lane segment), then across the unit's warps.
    T incl = run;
    const int PW = P < 32 ? P : 32;
    for (int d = 1; d < PW; d <<= 1) {
        const T y = __shfl_up_sync(0xffffffffu, incl, d, PW);
        if ((p & (PW - 1)) >= d) incl += y;
    }
    if (P > 32) {
        if ((p & 31) == 31) utot[p >> 5] = incl;
        unit_sync(P, uid);
        T add = (T)0;
        for (int w = 0; w < (p >> 5); ++w) add += utot[w];
        incl += add;
    } else {
        unit_sync(P, uid);
    }
    const T excl = incl - run;
#pragma unroll
    for (int e = 0; e < V; ++e) {
        const int q = p * V + e;
        T2 pr;
        pr.x = Xe[e];
        pr.y = Xo[e] + excl;
        *reinterpret_cast<T2*>(buf + xpad(2 * q)) = pr;
    }
    unit_sync(P, uid);
}

// Launch geometry shared by host and device: lanes P and values V = M / P
// per unit, rows per CTA (whole warps: 32 / P rows per group for P < 32),
// scalars per unit buffer.  Default P (measured per grid size on B200): one
// warp per unit up to M = 256 (fewer values per lane, more warps in flight,
// shorter dependent chains), two warps (a named barrier between passes) from
// M = 512 in both directions (the inverse's 8-value units in a register-
// capped instance, whose back-projection otherwise held it to two CTAs per
// SM), when a row's L units fit the kernel's thread bound; dir is kept for
// callers that ask per direction.
// Threads a DST CTA may have: 320 for 16 values per lane (five layers of
// two-warp units at M = 1024), else 256, the bound the others' register
// use was tuned for.
__host__ __device__ constexpr int dst_max_threads(int V) { return V == 16 ? 320 : 256; }
__host__ __device__ inline int dst_lanes_default_hd(int M, int L, int dir) {
    (void)dir;
    if (M <= 256) return M / 2 < 32 ? (M / 2 < 1 ? 1 : M / 2) : 32;
    return L * 64 <= dst_max_threads(M / 64) ? 64 : 32;
}
__host__ __device__ inline int dst_rows_per_cta(int P, int c) {
    if (c <= 0) c = 1;  // one row group per CTA: the most CTAs, measured fastest
    return c * (P >= 32 ? 1 : 32 / P);
}
__host__ __device__ inline int dst_unit_len(int N) { return (N + N / 8 + 2 + 1) & ~1; }

// Row DST kernel.  A CTA holds R rows x L modes = L*R units of P lanes,
// ordered mode-major (unit (m, r) at index m*R + r), so that every warp's
// units share one mode.
//
// Forward (EPI_SPEC, interior rows 1..jj-2): a thread loads the layer values
// of a node pair (k, N - k) straight from global memory, projects both onto
// the modes (z_to_modes, scaled by 0.5/(ii-1); PRO_STEP first applies the
// CABARET predictor + beta update, PRO_PLAIN only scales) and stores the
// pair's two pre-twiddled values of every mode.  Each unit then transforms
// its row and writes spec(m, j, k-1) = X_k.
//
// Inverse (EPI_HELM / EPI_PV, rows 0..jj-1): each unit loads the pairs of its
// solved spectral row (zero on the boundary rows), transforms them, and the
// row is written out; for EPI_PV the correction rows corr_m (m >= 1) are
// copied into shared memory during the transform and the mass-corrected
// back-projection writes psi.
//
// What bounds it: L1 / shared-memory cycles and the latency of a CTA's chain
// (1.7 waves at 1025 nodes).  Pre-twiddling in registers, instead of staging
// the row (cp.async), projecting it in place and reading it twice more, takes
// five passes over the shared-memory row down to two; with the tables read
// line by line, FP32 units at their own width and compile-time geometries:
// 1025^2 x 3 forward 45.7 -> 29.1 us FP64, 33.4 -> 24.8 mixed, inverse 41.1 ->
// 27.6 and 36.7 -> 26.7; 2049^2 x 5 forward 271 -> 169 and 236 -> 144, inverse
// 291 -> 177 and 257 -> 156 (there two CTAs per SM instead of one).
//
// S is the storage type of the state and spectral fields.  S = float is the
// mixed form: the layer fields and the baroclinic spectral rows are FP32 and
// transformed in FP32, while the barotropic mode (m = 0) is kept in FP64
// end to end (spec64), as are the projection, the back-projection and psi.
// Scalars of shared memory (in doubles) the L*R unit buffers take: FP64, or
// for the mixed form FP64 for mode 0 and FP32 for the others.
__host__ __device__ inline size_t dst_units_len(int L, int R, int N, bool mixed) {
    const size_t U = dst_unit_len(N);
    return mixed ? R * U + (((size_t)(L - 1) * R * U + 3) / 4) * 2 : (size_t)L * R * U;
}

// The row-DST kernel's body; k_dst and k_dst_capped below are its kernels.
//
// PC > 0: the lanes per unit P at compile time (most default geometries,
// launch_dst), hence N, M and the pitch: every index of the
// transform is then a lane's base plus an immediate.
template <typename S, int V, int PC, int PRO, int EPI>
__device__ __forceinline__ void dst_body(const Member* __restrict__ mems, const int* __restrict__ prefix, int nmem,
                                         int row_offset, int c, int corr_smem, int psic_here, const Member& one,
                                         int use_one, int gemm_bc) {
    constexpr bool MX = sizeof(S) == 4;
    __shared__ Member Mb;
    __shared__ double psic_s[PQ_MAXL];                   // closed basin: psiC of the inverse
    __shared__ double psic_red[dst_max_threads(V) / 32 * PQ_MAXL];  // (at least eight warps' room)
    extern __shared__ __align__(16) double sm[];
    pdl_wait();
    int local;
    cta_member(Mb, one, use_one, mems, prefix, nmem, blockIdx.x, &local);
    __syncthreads();
    const int L = Mb.L, jj = Mb.jj;
    const int P = PC ? PC : Mb.M / V;
    const int M = P * V, N = 2 * M, n = N - 1, ii = N + 1, pitch = (ii + 31) & ~31;
    const long long ls = Mb.lstride;
    const int R = dst_rows_per_cta(P, c);
    const int U = dst_unit_len(N);
    const int j0 = row_offset + local * R;                 // first row of this CTA
    // one past the last row; a channel periodic in j transforms every row
    const int jend = (EPI == EPI_SPEC && !Mb.periodic) ? jj - 1 : jj;
    const int nthr = blockDim.x;
    double* extra = sm + dst_units_len(L, R, N, MX);        // EPI_PV: corr rows [R][L-1][pitch]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = nthr >> 5;
    // Unit (m, r) buffers: FP64 values, except the baroclinic ones of the mixed form.
    auto fp64_mode = [&](int m) { return !MX || m == 0; };
    auto ubuf = [&](int m, int r) { return sm + (size_t)(m * R + r) * U; };  // FP64 modes
    auto ubuf32 = [&](int m, int r) { return reinterpret_cast<float*>(sm + (size_t)R * U) + (size_t)((m - 1) * R + r) * U; };
    auto get = [&](int m, int r, int k) -> double { return fp64_mode(m) ? ubuf(m, r)[k] : (double)ubuf32(m, r)[k]; };
    // This thread's unit: mode um of row ju.
    const int u = threadIdx.x / P, p = threadIdx.x & (P - 1);
    const int um = u / R, ur = u - um * R;
    const int ju = j0 + ur;
    const bool interior = (Mb.periodic || (ju >= 1 && ju <= jj - 2)) && ju < jend;

    // ---------------- stage the rows --------------------------------------
    if (EPI == EPI_SPEC) {
        const double cff = 0.5 / (double)(ii - 1);
        // The pair's values xa (node k), xb (node N - k) of mode m, row r.
        auto put = [&](int m, int r, int t, double xa, double xb) {
            if (fp64_mode(m)) {
                put_pair(ubuf(m, r), t, N, xa, xb, Mb.was);
            } else if (gemm_bc) {
                // the projected node row itself, for the tensor-core DST
                if (j0 + r < jend) {
                    float* g = reinterpret_cast<float*>(Mb.gbuf) + m * ls + (long long)(j0 + r) * pitch - 1;
                    const int k = t ? t : N >> 1;
                    g[k] = (float)xa;
                    if (t) g[N - k] = (float)xb;
                }
            } else {
                put_pair(ubuf32(m, r), t, N, (float)xa, (float)xb, Mb.was_f);
            }
        };
        // The same of one node (odd: N - t), given the other's value.
        [[maybe_unused]] auto put1 = [&](int m, int r, int t, bool odd, double own, double other) {
            if (fp64_mode(m)) {
                put_node(ubuf(m, r), t, odd, N, own, other, Mb.was);
            } else if (gemm_bc) {
                if (j0 + r < jend && (t || !odd))
                    reinterpret_cast<float*>(Mb.gbuf)[m * ls + (long long)(j0 + r) * pitch - 1 + (odd ? N - t : t ? t : N >> 1)] = (float)own;
            } else {
                put_node(ubuf32(m, r), t, odd, N, (float)own, (float)other, Mb.was_f);
            }
        };
        if constexpr (PRO == PRO_PLAIN) {
            // The stand-alone helm input (helm_io) is FP64 in either form.
            const double* src = reinterpret_cast<const double*>(Mb.helm_io) + um * Mb.io_ls +
                                (long long)(ju < jend ? ju : jend - 1) * Mb.io_pitch;
            if (fp64_mode(um)) {
                stage_unit<V>(ubuf(um, ur), p, P, N, Mb.was, [&](int k) { return cff * __ldcg(src + k); });
            } else if (gemm_bc) {
                for (int t = p; t < M; t += P) put(um, ur, t, cff * __ldcg(src + (t ? t : M)), cff * __ldcg(src + N - t - (t ? 0 : M)));
            } else {
                stage_unit<V>(ubuf32(um, ur), p, P, N, Mb.was_f, [&](int k) { return (float)(cff * __ldcg(src + k)); });
            }
        } else {
            const double dt = Mb.sc->dt, ta = Mb.sc->tweight_a;
            const S* __restrict__ zin = reinterpret_cast<const S*>(Mb.zeta);
            const S* __restrict__ zo = reinterpret_cast<const S*>(Mb.zeta_old[Mb.cur]);
            const S* __restrict__ rs = reinterpret_cast<const S*>(Mb.res);
            const S* __restrict__ rbo = reinterpret_cast<const S*>(Mb.res_beta_other);
            S* __restrict__ rb = reinterpret_cast<S*>(Mb.res_beta);
            const S* __restrict__ ui = reinterpret_cast<const S*>(Mb.ui);
            S* __restrict__ zp = reinterpret_cast<S*>(Mb.zeta);
            // Layer counts up to five run with the loops unrolled to the exact
            // count and z2m (and beta) in registers, larger ones under predicates.
            auto rows = [&](auto lc, auto exact) {
                constexpr int LC = decltype(lc)::value;
                constexpr bool EX = decltype(exact)::value;
                // Node pairs a thread loads before it uses any of them.
                constexpr int UN = PRO == PRO_STEP ? 1 : LC <= 2 ? 3 : LC == 3 ? 2 : 1;
                // z2m in registers up to three layers, else read from shared memory.
                constexpr bool ZR = EX && LC <= 3;
                constexpr int LZ = ZR ? LC : 1;
                double zm[LZ][LZ];
                if constexpr (ZR) {
#pragma unroll
                    for (int m = 0; m < LC; ++m)
#pragma unroll
                        for (int l = 0; l < LC; ++l) zm[m][l] = Mb.z2m[m * PQ_MAXL + l];
                }
                auto has = [&](int l) { return EX || l < L; };
                // cabaret_predictor (qg3p_aux.F90:1012-1018) and cabaret_beta
                // (:1051-1059) at node k of row j: every load first, then the
                // arithmetic and the stores of res_beta and zeta.
                auto step_node = [&](int j, int k, bool ok, double (&z)[LC]) {
                    const long long o = (long long)j * pitch + k;
                    S a0[LC], a1[LC], a2[LC], a3[LC], a4[LC];  // (widened at their use: no load waits)
#pragma unroll
                    for (int l = 0; l < LC; ++l) {
                        if (has(l) && ok) {
                            const long long ol = o + l * ls;
                            a0[l] = zo[ol];
                            a1[l] = rs[ol];
                            a2[l] = ui[ol];
                            a3[l] = ui[ol + 1];
                            a4[l] = rbo[ol];
                        }
                    }
#pragma unroll
                    for (int l = 0; l < LC; ++l) {
                        double zz = 0.0;
                        if (has(l) && ok) {
                            const long long ol = o + l * ls;
                            zz = (double)a0[l] + 0.5 * dt * (double)a1[l];
                            const double rbn = dt * (0.5 * ((double)a3[l] + (double)a2[l]) * Mb.beta[l]);
                            zz = zz + (1.0 + ta) * rbn - ta * (double)a4[l];
                            rb[ol] = (S)rbn;
                            zp[ol] = (S)zz;
                            if (MX) zz = (double)(S)zz;  // the stored (FP32) value
                        }
                        z[l] = zz;
                    }
                };
                auto project = [&](int r, int t, const double (&za)[LC], const double (&zb)[LC]) {
                    // z_to_modes, qg3p_diagnostics.F90:545-549
#pragma unroll ZR ? LC : 1
                    for (int m = 0; m < LC; ++m) {
                        if (!has(m)) break;
                        double sa = 0.0, sb = 0.0;
#pragma unroll
                        for (int l = 0; l < LC; ++l) {
                            if (has(l)) {
                                const double w = ZR ? zm[ZR ? m : 0][ZR ? l : 0] : Mb.z2m[m * PQ_MAXL + l];
                                sa += w * za[l];
                                sb += w * zb[l];
                            }
                        }
                        put(m, r, t, cff * sa, cff * sb);
                    }
                };
                // Two values per lane: the rows of units narrower than a warp (G of
                // them) side by side, so that their loads are in flight together
                // (33 x 33 x 3 mixed: 12.8 us one row after the other, 10.8).
                constexpr bool FLAT = V == 2 && PC < 32;
                const int G = FLAT && P < 32 ? 32 / P : 1;
                auto row_of = [&](int r0, int i) { return FLAT ? r0 + (PC ? i / M : i >> Mb.logM) : r0; };
                auto pair_of = [&](int i) { return FLAT ? i & (M - 1) : i; };
                if constexpr (PRO == PRO_STEP && !EX && V <= 16) {
                    // More than five layers: a node per lane, its pair's other
                    // from the next lane, so that the predictor's loads of a
                    // node (five per layer) and one projection fit the registers
                    // (1025^2 x 8, pairs: 235 us FP64 and 280 mixed; 169, 166).
                    // (Whole warps: the shuffle below, also where 2 M < 32.)
                    for (int r0 = 0; r0 < R; r0 += G) {
                        for (int t0 = threadIdx.x; t0 < ((2 * G * M + 31) & ~31); t0 += nthr) {
                            const bool in = t0 < 2 * G * M, odd = t0 & 1;
                            const int i = in ? t0 >> 1 : 0, r = row_of(r0, i), t = pair_of(i);
                            const int j = min(j0 + r, jend - 1), k = odd ? N - t : t ? t : M;
                            double z[LC];
                            step_node(j, k, in && j0 + r < jend && (t || !odd), z);
#pragma unroll 1
                            for (int m = 0; m < L; ++m) {
                                double sum = 0.0;
#pragma unroll
                                for (int l = 0; l < LC; ++l)
                                    if (has(l)) sum += Mb.z2m[m * PQ_MAXL + l] * z[l];
                                const double own = cff * sum, next = __shfl_xor_sync(0xffffffffu, own, 1);
                                if (in) put1(m, r, t, odd, own, t ? next : own);
                            }
                        }
                    }
                    return;
                }
                for (int r0 = 0; r0 < R; r0 += G) {
                    const bool ok0 = j0 + r0 < jend;
                    const int jr0 = ok0 ? j0 + r0 : jend - 1;
                    [[maybe_unused]] const S* row0 = zin + (long long)jr0 * pitch;
                    for (int t0 = threadIdx.x; t0 < G * M; t0 += nthr * UN) {
                        double za[UN][LC], zb[UN][LC];
                        if constexpr (PRO == PRO_STEP) {
                            const int t = pair_of(t0), k = t ? t : M;
                            const bool ok = FLAT ? j0 + row_of(r0, t0) < jend : ok0;
                            const int j = FLAT ? min(j0 + row_of(r0, t0), jend - 1) : jr0;
                            step_node(j, k, ok, za[0]);
                            if (LC > 2) asm volatile("" ::: "memory");  // one node's loads at a time
                            if (t) {
                                step_node(j, N - k, ok, zb[0]);
                            } else {
#pragma unroll
                                for (int l = 0; l < LC; ++l) zb[0][l] = za[0][l];
                            }
                        } else {
                            S va[UN][LC], vb[UN][LC];
#pragma unroll
                            for (int q = 0; q < UN; ++q) {
                                const int i = t0 + q * nthr, t = pair_of(i), k = t ? t : M;
                                const S* row = FLAT ? zin + (long long)min(j0 + row_of(r0, i), jend - 1) * pitch : row0;
#pragma unroll
                                for (int l = 0; l < LC; ++l) {
                                    const bool in = has(l) && i < G * M;
                                    va[q][l] = in ? __ldcg(row + l * ls + k) : (S)0;
                                    vb[q][l] = in ? __ldcg(row + l * ls + N - k) : (S)0;
                                }
                            }
#pragma unroll
                            for (int q = 0; q < UN; ++q)
#pragma unroll
                                for (int l = 0; l < LC; ++l) {
                                    za[q][l] = (double)va[q][l];
                                    zb[q][l] = (double)vb[q][l];
                                }
                        }
#pragma unroll
                        for (int q = 0; q < UN; ++q)
                            if (t0 + q * nthr < G * M) project(row_of(r0, t0 + q * nthr), pair_of(t0 + q * nthr), za[q], zb[q]);
                    }
                }
            };
            switch (L) {
                case 1: rows(std::integral_constant<int, 1>{}, std::true_type{}); break;
                case 2: rows(std::integral_constant<int, 2>{}, std::true_type{}); break;
                case 3: rows(std::integral_constant<int, 3>{}, std::true_type{}); break;
                case 4: rows(std::integral_constant<int, 4>{}, std::true_type{}); break;
                case 5: rows(std::integral_constant<int, 5>{}, std::true_type{}); break;
                default: rows(std::integral_constant<int, PQ_MAXL>{}, std::false_type{});
            }
        }
    } else {
        if (EPI == EPI_PV && corr_smem) {
            const double* corr = Mb.corr;
            const int cw = pitch >> 1;
            for (int rm = warp; rm < R * (L - 1); rm += nwarp) {
                const int r = rm / (L - 1), m = 1 + rm - r * (L - 1);
                const int j = j0 + r;
                const bool ok = j < jend;
                const double* g = corr + m * ls + (long long)(ok ? j : 0) * pitch;
                double* d = extra + (size_t)rm * pitch;
                for (int q = lane; q < cw; q += 32) cp16(d + 2 * q, g + 2 * q, ok);
            }
        }
        const int KT = 8 / tri_warps(jj), tpm = (n + KT - 1) / KT;
        // psiC's sum runs on psic_here "threads" (this CTA's, or 256 of which
        // each warp stands for several warps): the first terms, in flight
        // with the rows.
        double acc[PQ_MAXL];
        auto part = [&](int mm, int vt) {
            double t = 0.0;
            for (int q = vt; q < tpm; q += psic_here) t += __ldcg(Mb.partials + (long long)mm * tpm + q);
            return t;
        };
        if (EPI == EPI_PV && psic_here) {
#pragma unroll
            for (int mm = 0; mm < PQ_MAXL; ++mm)
                acc[mm] = (mm < L && (int)threadIdx.x < tpm) ? __ldcg(Mb.partials + (long long)mm * tpm + threadIdx.x) : 0.0;
        }
        // x_k = spec(m, j, k-1); the boundary rows of a closed basin are zero.
        const long long ro = um * ls + (long long)(interior ? ju : 1) * pitch - 1;
        if (fp64_mode(um)) {
            const double* g = (MX ? Mb.spec64 : reinterpret_cast<const double*>(Mb.spec)) + ro;
            stage_unit<V>(ubuf(um, ur), p, P, N, Mb.was, [&](int k) { return interior ? __ldcg(g + k) : 0.0; });
        } else if (gemm_bc) {
            // Rows the tensor-core DST already took back to node values:
            // straight to the positions the back-projection reads.
            const float* g = reinterpret_cast<const float*>(Mb.gbuf) + ro;
            float* d = ubuf32(um, ur);
            for (int k = 1 + p; k <= n; k += P) d[xpad(k)] = interior ? __ldcg(g + k) : 0.f;
        } else {
            const float* g = reinterpret_cast<const float*>(Mb.spec) + ro;
            stage_unit<V>(ubuf32(um, ur), p, P, N, Mb.was_f, [&](int k) { return interior ? __ldcg(g + k) : 0.f; });
        }
        if (EPI == EPI_PV && psic_here) {
            // psiC_m = (sum of the tridiagonal CTAs' partial means of mode m)
            // / (g_ii_int g_jj_int) (modes_to_z_correct_mass,
            // qg3p_aux.F90:482-521), summed in the same fixed order by every
            // CTA (one pass for all modes); the member's
            // first CTA publishes it and flags a NaN (the reference aborts,
            // :504-510) or a value above 1e100 (it warns, :511-517).
            for (int vw = warp; vw < psic_here / 32; vw += nwarp)
#pragma unroll
                for (int mm = 0; mm < PQ_MAXL; ++mm) {
                    if (mm < L) {
                        double t;
                        if (vw == warp) {
                            t = acc[mm];
                            for (int q = threadIdx.x + psic_here; q < tpm; q += psic_here)
                                t += __ldcg(Mb.partials + (long long)mm * tpm + q);
                        } else {
                            t = part(mm, 32 * vw + lane);
                        }
                        t = warp_sum(t);
                        if (lane == 0) psic_red[vw * PQ_MAXL + mm] = t;
                    }
                }
            __syncthreads();
            if (threadIdx.x < L) {
                const int mm = threadIdx.x;
                double t = 0.0;
                for (int w = 0; w < psic_here / 32; ++w) t += psic_red[w * PQ_MAXL + mm];
                const double pc = t * Mb.mean_scale;
                psic_s[mm] = pc;
                if (local == 0) {
                    Mb.sc->psiC[mm] = pc;
                    if (pc != pc)
                        atomicOr(Mb.status, (int)ST_NAN_PSIC);
                    else if (fabs(pc) > 1.0e100)
                        atomicOr(Mb.status, (int)ST_LARGE_PSIC);
                }
            }
        }
    }
    // Rows staged by the whole CTA (the projection), or by the unit itself.
    if (EPI == EPI_SPEC && PRO != PRO_PLAIN)
        __syncthreads();
    else
        unit_sync(P, u);

    // ---------------- per-unit transform ----------------------------------
    __shared__ double utot[8][2];  // cross-warp scan totals of units wider than a warp
    // With gemm_bc the baroclinic rows (a whole warp's or unit's mode) are
    // transformed by the tensor-core DST instead (pq_dst_mma.cu).
    if (fp64_mode(um))
        dst_unit<V, PC, double>(ubuf(um, ur), p, P, u, utot[u & 7], N, M, Mb.tw, Mb.wsplit);
    else if (!gemm_bc)
        dst_unit<V, PC, float>(ubuf32(um, ur), p, P, u, reinterpret_cast<float*>(utot[u & 7]), N, M, Mb.tw_f, Mb.wsplit_f);
    if (EPI == EPI_PV && corr_smem) cp_commit_wait_all();
    pdl_release();

    if (EPI == EPI_SPEC) {
        if (ju < jend) {
            if (fp64_mode(um)) {
                double* spec = (MX ? Mb.spec64 : reinterpret_cast<double*>(Mb.spec)) + um * ls +
                               (long long)ju * pitch - 1;
                const double* buf = ubuf(um, ur);
                for (int k = 1 + p; k <= n; k += P) spec[k] = buf[xpad(k)];
            } else if (!gemm_bc) {
                float* spec = reinterpret_cast<float*>(Mb.spec) + um * ls + (long long)ju * pitch - 1;
                const float* fb = ubuf32(um, ur);
                for (int k = 1 + p; k <= n; k += P) spec[k] = fb[xpad(k)];
            }
        }
    } else if (EPI == EPI_HELM) {
        // helm's in-place output: interior entries of interior rows, row
        // i = ii zeroed (:758-761); ge_local zeroes psi(2:ii-1, 1)
        // (:1055-1057).  helm_io is FP64 in either form (the mixed form's
        // FP32 units are widened).
        double* io = reinterpret_cast<double*>(Mb.helm_io) + um * Mb.io_ls + (long long)ju * Mb.io_pitch;
        if (interior) {
            if (fp64_mode(um)) {
                const double* buf = ubuf(um, ur);
                for (int k = 1 + p; k <= n; k += P) io[k] = buf[xpad(k)];
            } else {
                const float* fb = ubuf32(um, ur);
                for (int k = 1 + p; k <= n; k += P) io[k] = (double)fb[xpad(k)];
            }
            if (p == 0) io[ii - 1] = 0.0;
        } else if (ju == 0 && !Mb.periodic) {
            for (int k = 1 + p; k <= n; k += P) io[k] = 0.0;
        }
    } else {
        // psi_l = phi_1 - psiC_1 + sum_{m>=2} m2z(l,m) (phi_m - psiC_m corr_m)
        // (modes_to_z_btcu, qg3p_diagnostics.F90:615-635) on every node of the
        // row; phi is zero on the boundary (apply_dirichlet_bc(0),
        // qg3p_aux.F90:470).
        __syncthreads();
        // A channel (modes_to_z_correct_momentum + modes_to_z, qg3p_aux.F90:
        // 524-575) subtracts psiC_m corr_m + psiC2_m corr2_m from the
        // baroclinic modes; its psiC_0 is zero.
        const double* psiC = Mb.sc->psiC;
        const double* psiC2 = Mb.sc->psiC2;
        double pc[PQ_MAXL], pc2[PQ_MAXL];
#pragma unroll
        for (int m = 0; m < PQ_MAXL; ++m) {
            pc[m] = (m < L) ? (psic_here ? psic_s[m] : psiC[m]) : 0.0;
            pc2[m] = (m < L && Mb.periodic) ? psiC2[m] : 0.0;
        }
        double* psi = Mb.psi;
        // Exact layer counts up to five (every configuration here) run with
        // the loops unrolled to L and m2z in registers: the loops below,
        // unrolled to PQ_MAXL under predicates, issue several times the
        // instructions and shared-memory loads (measured 0.6-0.8 us per node
        // row pass at 513 x 513 x 3 against ~0.1 us for L = 3).
        auto exact = [&](auto lc) {
            constexpr int LC = decltype(lc)::value;
            double mz[LC][LC];
#pragma unroll
            for (int l = 0; l < LC; ++l)
#pragma unroll
                for (int m = 1; m < LC; ++m) mz[l][m] = Mb.m2z[l * PQ_MAXL + m];
            const double* c2b = Mb.corr2;
            for (int r = 0; r < R; ++r) {
                const int j = j0 + r;
                if (j >= jend) break;
                const double* crs = extra + ((long long)r * (LC - 1) - 1) * pitch;  // staged corr rows
                const double* crg = Mb.corr + (long long)j * pitch;
                for (int i = threadIdx.x; i < ii; i += nthr) {
                    const bool inner = (Mb.periodic || (j >= 1 && j <= jj - 2)) && i >= 1 && i <= n;
                    double ph[LC];
#pragma unroll
                    for (int m = 0; m < LC; ++m) ph[m] = inner ? get(m, r, xpad(i)) : 0.0;
#pragma unroll
                    for (int m = 1; m < LC; ++m)
                        ph[m] -= pc[m] * (corr_smem ? crs[m * (long long)pitch + i] : crg[m * ls + i]);
                    if (Mb.periodic) {
                        const double* c2 = c2b + (long long)j * pitch + i;
#pragma unroll
                        for (int m = 1; m < LC; ++m) ph[m] -= pc2[m] * c2[m * ls];
                    }
                    const double b0 = ph[0] - pc[0];
                    const long long o = (long long)j * pitch + i;
#pragma unroll
                    for (int l = 0; l < LC; ++l) {
                        double dot = 0.0;
#pragma unroll
                        for (int m = 1; m < LC; ++m) dot += mz[l][m] * ph[m];
                        psi[o + l * ls] = b0 + dot;
                    }
                }
            }
        };
        switch (L) {
            case 1: exact(std::integral_constant<int, 1>{}); return;
            case 2: exact(std::integral_constant<int, 2>{}); return;
            case 3: exact(std::integral_constant<int, 3>{}); return;
            case 4: exact(std::integral_constant<int, 4>{}); return;
            case 5: exact(std::integral_constant<int, 5>{}); return;
            default: break;
        }
        for (int r = 0; r < R; ++r)
            for (int i = threadIdx.x; i < ii; i += nthr) {
                const int j = j0 + r;
                if (j >= jend) break;
                const bool inner = (Mb.periodic || (j >= 1 && j <= jj - 2)) && i >= 1 && i <= n;
                // corr_m at cr[m * cst] (staged rows, or the field itself)
                const double* cr = corr_smem ? extra + ((long long)r * (L - 1) - 1) * pitch + i
                                             : Mb.corr + (long long)j * pitch + i;
                const long long cst = corr_smem ? (long long)pitch : ls;
                double ph[PQ_MAXL];
#pragma unroll
                for (int m = 0; m < PQ_MAXL; ++m)
                    if (m < L) ph[m] = inner ? get(m, r, xpad(i)) : 0.0;
#pragma unroll
                for (int m = 1; m < PQ_MAXL; ++m)
                    if (m < L) ph[m] -= pc[m] * cr[m * cst];
                if (Mb.periodic) {
                    const double* c2 = Mb.corr2 + (long long)j * pitch + i;
#pragma unroll
                    for (int m = 1; m < PQ_MAXL; ++m)
                        if (m < L) ph[m] -= pc2[m] * c2[m * ls];
                }
                const double b0 = ph[0] - pc[0];
                const long long o = (long long)j * pitch + i;
#pragma unroll
                for (int l = 0; l < PQ_MAXL; ++l) {
                    if (l < L) {
                        double dot = 0.0;
#pragma unroll
                        for (int m = 1; m < PQ_MAXL; ++m)
                            if (m < L) dot += Mb.m2z[l * PQ_MAXL + m] * ph[m];
                        psi[o + l * ls] = b0 + dot;
                    }
                }
            }
    }
}

// MINB > 0: registers capped so that MINB CTAs of the bound's threads fit an
// SM (dst_min_ctas); the bodies' widest layer counts would otherwise set the
// register count of all.
template <typename S, int V, int PC, int PRO, int EPI>
__global__ void __launch_bounds__(dst_max_threads(V))
    k_dst(const Member* __restrict__ mems, const int* __restrict__ prefix, int nmem, int row_offset, int c,
          int corr_smem, int psic_here, const __grid_constant__ Member one, int use_one, int gemm_bc) {
    dst_body<S, V, PC, PRO, EPI>(mems, prefix, nmem, row_offset, c, corr_smem, psic_here, one, use_one, gemm_bc);
}
template <typename S, int V, int PC, int PRO, int EPI, int MINB>
__global__ void __launch_bounds__(dst_max_threads(V), MINB)
    k_dst_capped(const Member* __restrict__ mems, const int* __restrict__ prefix, int nmem, int row_offset, int c,
                 int corr_smem, int psic_here, const __grid_constant__ Member one, int use_one, int gemm_bc) {
    dst_body<S, V, PC, PRO, EPI>(mems, prefix, nmem, row_offset, c, corr_smem, psic_here, one, use_one, gemm_bc);
}
// CTAs per SM the registers must allow (0: no bound; the bound's CTAs have 256
// threads, 320 with 16 values): the forward DST three up to 8 values per lane,
// the inverse of 64-lane units of 8 values three, 16 values two.  With the predictor
// two up to 8 values (513^2 x 4 FP64 20.9 us, 27.0 without a bound; 1025^2 x 4 65, 78;
// the smallest grids lose 2 us at eight layers) and one with 16, which lets its
// loads take the registers (1025^2 x 5 FP64 98.9 us, 123 without).
template <int V, int PC, int PRO, int EPI>
__host__ __device__ constexpr int dst_min_ctas() {
    if (PRO == PRO_STEP) return V <= 8 ? 2 : V == 16 ? 1 : 0;
    if (V == 16) return 2;
    if (EPI == EPI_SPEC && PRO == PRO_MODAL) return V <= 8 ? 3 : 0;
    return (EPI == EPI_PV && V == 8 && PC == 64) ? 3 : 0;
}

// psiC's order of summation changes where a member has more row CTAs than this.
constexpr int PSIC_CTAS = 592;

template <typename S, int V, int PC, int PRO, int EPI>
static cudaError_t launch_dst_v(const LaunchSet& ls, cudaStream_t st) {
    const int M = ls.maxN / 2, L = ls.maxL;
    const int R = dst_rows_per_cta(M / V, ls.dst_group);
    const int threads = L * R * (M / V);
    size_t bytes = dst_units_len(L, R, ls.maxN, sizeof(S) == 4) * sizeof(double);
    const size_t cbytes = (size_t)R * (L - 1) * ls.maxPitch * sizeof(double);
    constexpr int MINB = dst_min_ctas<V, PC, PRO, EPI>();
    // corr rows in shared memory while as many CTAs fit an SM beside them as the
    // registers allow: four; two of more than 192 threads with 128 registers
    // (513^2 x 8 FP64: 41.0 us without, 30.9 with); one of 32 values (2049 x 257 x 6: 94, 83).
    const size_t room = (V == 32 ? 200 : (MINB == 0 && threads > 192) ? 100 : 56) * 1024;
    const int corr_smem = (EPI == EPI_PV && !ls.periodic && bytes + cbytes <= room) ? 1 : 0;
    if (corr_smem) bytes += cbytes;
    // The number of strided sums psiC is taken in: a CTA's threads (one pass), or
    // 256 when a member has more than PSIC_CTAS CTAs of rows.  Either order is
    // the one such a problem has always had; which one it is depends on the
    // member's own rows alone, so that a run merged with others, on any device,
    // adds as it does alone (every member of a launch has ls.maxJ rows).
    const int psic_here =
        (EPI == EPI_PV && !ls.periodic) ? ((ls.maxJ + R - 1) / R <= PSIC_CTAS ? threads : 256) : 0;
    void (*kern)(const Member*, const int*, int, int, int, int, int, Member, int, int);
    if constexpr (MINB > 0)
        kern = k_dst_capped<S, V, PC, PRO, EPI, MINB>;
    else
        kern = k_dst<S, V, PC, PRO, EPI>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    const int dir = (EPI == EPI_SPEC) ? 0 : 1;
    return launch_step_kernel(ls.pdl, kern, dim3(ls.ctas_dst[dir]), dim3(threads), bytes, st,
                              ls.members, ls.prefix_dst[dir], ls.nmem, (EPI == EPI_SPEC && !ls.periodic) ? 1 : 0,
                              ls.dst_group, corr_smem, psic_here, member_arg(ls), member_arg_used(ls),
                              sizeof(S) == 4 ? ls.gemm_bc : 0);
}

// The compile-time geometries: what the defaults select (dst_lanes_default
// for a step, dst_lanes_batched for the stand-alone solves) from 65 (33) to 2049
// nodes, but for a step of five or more layers at 1025 nodes, of six or more at 2049,
// and a stand-alone solve at 2049: one-warp units of 16 and 32 values.
template <typename S, int PRO, int EPI>
static cudaError_t launch_dst(const LaunchSet& ls, cudaStream_t st) {
    const int P = ls.dst_lanes[EPI == EPI_SPEC ? 0 : 1], V = ls.maxN / 2 / P;
    constexpr bool STEP = PRO != PRO_PLAIN || EPI == EPI_PV;
    constexpr bool HELM = EPI == EPI_HELM || (PRO == PRO_PLAIN && EPI == EPI_SPEC);
    if constexpr (STEP) {
        if (V == 2 && P == 16) return launch_dst_v<S, 2, 16, PRO, EPI>(ls, st);
        if (V == 2 && P == 32) return launch_dst_v<S, 2, 32, PRO, EPI>(ls, st);
        if (V == 4 && P == 32) return launch_dst_v<S, 4, 32, PRO, EPI>(ls, st);
        if (V == 8 && P == 64) return launch_dst_v<S, 8, 64, PRO, EPI>(ls, st);
        if (V == 16 && P == 64) return launch_dst_v<S, 16, 64, PRO, EPI>(ls, st);
    }
    if constexpr (HELM) {
        if (V == 8 && P == 4) return launch_dst_v<S, 8, 4, PRO, EPI>(ls, st);
        if (V == 8 && P == 8) return launch_dst_v<S, 8, 8, PRO, EPI>(ls, st);
        if (V == 8 && P == 16) return launch_dst_v<S, 8, 16, PRO, EPI>(ls, st);
        if (V == 16 && P == 32) return launch_dst_v<S, 16, 32, PRO, EPI>(ls, st);
    }
    if constexpr (STEP || HELM) {
        if (V == 8 && P == 32) return launch_dst_v<S, 8, 32, PRO, EPI>(ls, st);
    }
    switch (V) {
        case 2: return launch_dst_v<S, 2, 0, PRO, EPI>(ls, st);
        case 4: return launch_dst_v<S, 4, 0, PRO, EPI>(ls, st);
        case 8: return launch_dst_v<S, 8, 0, PRO, EPI>(ls, st);
        case 16:  // (the stand-alone solves have 16 values only with 32 lanes, above)
            if constexpr (STEP) return launch_dst_v<S, 16, 0, PRO, EPI>(ls, st);
            return cudaErrorInvalidValue;
        case 32: return launch_dst_v<S, 32, 0, PRO, EPI>(ls, st);
        default: return cudaErrorInvalidValue;
    }
}

// One launcher per prologue / epilogue, each in a source of its own (pq_dst_*.cu).
cudaError_t launch_dst_plain(const LaunchSet& ls, int f32, cudaStream_t st);
cudaError_t launch_dst_modal(const LaunchSet& ls, int f32, cudaStream_t st);
cudaError_t launch_dst_step(const LaunchSet& ls, int f32, cudaStream_t st);
cudaError_t launch_dst_helm(const LaunchSet& ls, int f32, cudaStream_t st);
cudaError_t launch_dst_pv(const LaunchSet& ls, int f32, cudaStream_t st);

}  // namespace pq
