// pq_tridiag.cu -- the tridiagonal solves of the PV inversion (pq_helm.cu).
#include "pq_common.cuh"
#include "pq_kernels.h"

namespace pq {

constexpr int TRI_THREADS = 256;
// CTAs per SM the tridiagonal kernel's registers must allow, by chunk length
// and storage: 64 registers while they hold a chunk, then 80 (mixed: 1025^2 x 3
// 142.2 us per step, 145.5 with 128) or 128 (FP64: 174.5, 178.3 with 80, 182 with 64).
__host__ __device__ constexpr int tri_min_ctas(int RR, bool f32) {
    return f32 ? (RR <= 8 ? 4 : RR <= 16 ? 3 : 2) : (RR <= 6 ? 4 : RR <= 8 ? 3 : 2);
}

// ---------------------------------------------------------------------------
// Tridiagonal solves along j for KT = 8 / W wavenumbers of one mode (W warps
// per column, tri_warps).
//
// A lane owns one column's chunk of R <= RR consecutive rows, in registers from
// its loads to its stores (FULL: R = RR): lane = KT * (chunk in the warp) + column,
// the 32 W chunks of a column over the CTA's warps.  So a warp's access to row
// t of its chunks is 32 / KT segments of KT values (32-byte sectors in FP64,
// KT = 4) -- the transpose needs no shared memory.  The forward and backward
// Thomas recurrences run as first-order affine recurrences: a local sweep, a
// scan of the column's affine chunk maps (handed over in shared memory, one chunk per lane
// of W warps), and a fix-up sweep.  Rows past the column's end are padding of
// value and pivot 0.  The CTA also accumulates the domain mean of the solution
// in spectral space.
//
// Pivots: explicit up to len (few rows except for the smallest wavenumbers),
// then the fixed point; a warp beyond len takes the fixed point without a load,
// the others read theirs from shared memory (loaded beside the rows).
//
// What bounds it: the latency of the chain, load to store, in one to three
// waves.  Against the strip staged in shared memory by cp.async (126 registers
// and two CTAs per SM at 1025 nodes, shared-memory sweeps unless a chunk had 4,
// 8 or 16 rows), us per step: 2049^2 x 5 1125 -> 1093 FP64, 842 -> 793 mixed;
// 1025 x 769 x 3 153 -> 143, 1025^2 x 3 179 -> 175 FP64, 142.5 -> 140 mixed.  At
// 25 to 31 rows a chunk the mixed form's kernel is 13 % slower on 2049 columns
// (2049 x 1540 x 3: 84 -> 94 us) and 20 % faster on 257 (28.5 -> 23.4).  The chunks, their scan's order and the sums are that
// kernel's, so the results are too, bit for bit; chunks spread over more warps and scanned
// in the warp that holds them measured 2 % faster in the mixed form and lose that.
//
// S = float: the mixed form, whose baroclinic spectral rows are FP32 (solved in
// FP64); the barotropic mode (m = 0) comes from spec64.
//
// Doubles between two columns' pivots in shared memory (g(0) .. g(rows)): one
// of padding per 16, and 16 / KT modulo 16, so that the 16 / KT chunks of KT
// columns that a half-warp reads hit 16 bank pairs (16-row chunks).
__host__ __device__ inline int tri_pitch(int rows, int KT) { return (rows + (rows >> 4) + 16) / 16 * 16 + 16 / KT; }

// A CTA's partial means (wpart, wpart2: its warps' sums), and for a channel the
// member's coefficients by the last CTA.  Every thread takes part, after a
// barrier behind the last write of wpart.
__device__ __forceinline__ void publish_means(const Member& Mb, int local, int tiles_per_mode, double* wpart,
                                              double* wpart2, int* is_last) {
    if (threadIdx.x == 0) {
        double t = 0.0, t2 = 0.0;
        for (int w = 0; w < 8; ++w) {
            t += wpart[w];
            t2 += wpart2[w];
        }
        Mb.partials[local] = t;
        if (Mb.periodic) Mb.partials[Mb.ntiles_tri + local] = t2;
    }
    // A closed basin's inverse DST sums the partials itself (psiC_m, while its
    // rows load), so that no CTA here waits on a counter (1025^2 x 3: 137.9 ->
    // 135.4 us per step mixed, 180.5 -> 178.2 FP64).
    if (!Mb.periodic) return;
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned prev = atomicAdd(&Mb.counters[0], 1u);
        *is_last = (prev == (unsigned)(Mb.ntiles_tri - 1));
    }
    __syncthreads();
    if (!*is_last) return;
    // Last CTA of this channel, every sum in a fixed order so that the result
    // is independent of CTA timing (modes_to_z_correct_momentum,
    // qg3p_aux.F90:524-575): the baroclinic modes' coefficients of the two
    // correction functions, inv_corr_a times the wall PV means; the
    // barotropic mode is not corrected.
    __threadfence();
    for (int mm = 0; mm < Mb.L; ++mm) {
        const double t = block_sum_l2(Mb.partials + (long long)mm * tiles_per_mode, tiles_per_mode, 1, wpart);
        const double t2 =
            block_sum_l2(Mb.partials + Mb.ntiles_tri + (long long)mm * tiles_per_mode, tiles_per_mode, 1, wpart2);
        if (threadIdx.x == 0) {
            const double* M2 = Mb.inv_corr_a + 4 * mm;
            const double pc = mm == 0 ? 0.0 : M2[0] * t + M2[2] * t2, pc2 = mm == 0 ? 0.0 : M2[1] * t + M2[3] * t2;
            Mb.sc->psiC[mm] = pc;
            Mb.sc->psiC2[mm] = pc2;
            if (pc != pc || pc2 != pc2) atomicOr(Mb.status, (int)ST_NAN_PSIC);
            else if (fabs(pc) > 1.0e100 || fabs(pc2) > 1.0e100) atomicOr(Mb.status, (int)ST_LARGE_PSIC);
        }
    }
    if (threadIdx.x == 0) Mb.counters[0] = 0u;
}

template <typename S, int RR, int KT, bool FULL, bool ONE>
__global__ void __launch_bounds__(TRI_THREADS, tri_min_ctas(RR, sizeof(S) == 4)) k_tridiag(const Member* __restrict__ mems, const int* __restrict__ prefix,
                                                  int nmem, int do_mean, const __grid_constant__ Member one,
                                                  int use_one) {
    constexpr int W = 8 / KT, NQ = 32 * W;  // warps that scan a column's chunk maps, chunks of a column
    __shared__ Member Mb_s;
    __shared__ double maps[2][KT][NQ + 1];  // the chunks' affine maps (A, c); their carries in [0]
    __shared__ double tot[2][8][2];         // per scanning warp: affine totals (forward, backward)
    __shared__ double wpart[8], wpart2[8];
    __shared__ double ends[2][KT];          // channel: the solution's first and last open row
    __shared__ int is_last;
    extern __shared__ __align__(16) double pivs[];  // [KT][tri_pitch]
    pdl_wait();
    int local = blockIdx.x;
    if constexpr (!ONE) {
        cta_member(Mb_s, one, use_one, mems, prefix, nmem, blockIdx.x, &local);
        __syncthreads();
    }
    const Member& Mb = member_ref<ONE>(Mb_s, one);
    const int n = Mb.n, jj = Mb.jj, pitch = Mb.pitch;
    const int tiles_per_mode = (n + KT - 1) / KT;
    const int m = local / tiles_per_mode, tile = local - m * tiles_per_mode;
    const int Mr = jj - 2, R = FULL ? RR : (Mr + NQ - 1) / NQ;  // rows of a chunk, at most RR
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = lane & (KT - 1), q = warp * (32 / KT) + lane / KT;  // column and chunk
    const int kk = tile * KT + c;                                     // 0-based wavenumber index
    const bool active = kk < n;
    const int a = q * R + 1, b = a + R - 1;  // the chunk's row positions (1-based)
    const bool f32 = sizeof(S) == 4 && m > 0;  // this mode's rows are FP32
    // Column kk of this mode's spectral field (row j at sp + j pitch), FP32 or FP64.
    char* const sp = f32 ? reinterpret_cast<char*>(reinterpret_cast<float*>(Mb.spec) + (long long)m * Mb.lstride + (active ? kk : 0))
                         : reinterpret_cast<char*>(((sizeof(S) == 4) ? Mb.spec64 : reinterpret_cast<double*>(Mb.spec)) +
                                                   (long long)m * Mb.lstride + (active ? kk : 0));
    auto ld = [&](int row) -> double {
        return f32 ? (double)reinterpret_cast<const float*>(sp)[(long long)row * pitch]
                   : reinterpret_cast<const double*>(sp)[(long long)row * pitch];
    };
    // Pivot table entries first: the explicit pivots depend on them.
    int len = 0, off = 0;
    double fix = 0.0, wm = 0.0;
    if (active) {
        const int mk = m * n + kk;
        off = __ldg(&Mb.piv_off[mk]);
        len = __ldg(&Mb.piv_len[mk]);
        fix = __ldg(&Mb.piv_fix[mk]);
    }
    // The scanning warp's column weight of the mean, in flight with the rows.
    if (do_mean && tile * KT + warp % KT < n)
        wm = __ldg((Mb.periodic ? Mb.wwall : Mb.wmean) + tile * KT + warp % KT);
    double v[RR];
    if (f32) {
        float w[RR];
#pragma unroll
        for (int t = 0; t < RR; ++t)
            w[t] = (active && t < R && a + t <= Mr) ? reinterpret_cast<const float*>(sp)[(long long)(a + t) * pitch] : 0.f;
#pragma unroll
        for (int t = 0; t < RR; ++t) v[t] = (double)w[t];
    } else {
#pragma unroll
        for (int t = 0; t < RR; ++t)
            v[t] = (active && t < R && a + t <= Mr) ? reinterpret_cast<const double*>(sp)[(long long)(a + t) * pitch] : 0.0;
    }
    // g(p) at gs[p + p / 16] (0 outside the column), for the warps that read
    // it: those that start at or before the longest explicit table, and from
    // the warp that holds the column's end on.
    len = min(len, Mr);
    double* const gs = pivs + c * tri_pitch(NQ * R, KT);
    const double* const piv = Mb.piv + off;
    const int WR = 32 / KT * R;  // rows of a warp
    const int most = __reduce_max_sync(0xffffffffu, len), e0 = min(Mr, (most / WR + 1) * WR);
    for (int p = threadIdx.x / KT; p <= e0; p += TRI_THREADS / KT) {
        double* d = gs + p + (p >> 4);
        if (p >= 1 && p <= len)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(d)),
                         "l"(piv + p - 1)
                         : "memory");
        else
            *d = p == 0 ? 0.0 : fix;
    }
    for (int p = max(e0 + 1, Mr / WR * WR) + threadIdx.x / KT; p <= NQ * R; p += TRI_THREADS / KT)
        gs[p + (p >> 4)] = p <= Mr ? fix : 0.0;
    cp_commit_wait_all();
    __syncthreads();
    auto G = [&](int p) -> double { return gs[p + (p >> 4)]; };
    auto F = [&](int) -> double { return fix; };
    const bool flat = __all_sync(0xffffffffu, a - 1 > len && b <= Mr);

    // (Roundings written out: every instance gives the same bits.)
    // Forward elimination, local: y~_a = f_a, y~_p = f_p - g_{p-1} y~_{p-1};
    // y_p = y~_p + A_p y_{a-1}, A_a = -g_{a-1}, A_p = -g_{p-1} A_{p-1}.
    double A, y;
    auto forward = [&](auto g) {
        A = -g(a - 1);
        y = v[0];
#pragma unroll
        for (int t = 1; t < RR; ++t) {
            if (t < R) {
                const double gp = g(a + t - 1);
                y = __fma_rn(-gp, y, v[t]);
                v[t] = y;
                A = __dmul_rn(-gp, A);
            }
        }
    };
    if (flat)
        forward(F);
    else
        forward(G);
    // Scans run one chunk per lane: warp -> column wc, its half h (of W).
    const int wc = warp % KT, h = warp / KT, ch = 32 * h + lane;
    // Inclusive scan of the affine chunk maps y_out = c + A y_in in the warp,
    // then the column's earlier warps' totals composed in order.
    maps[0][c][q] = A;
    maps[1][c][q] = y;
    __syncthreads();
    {
        double sA = maps[0][wc][ch], sc = maps[1][wc][ch];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double pA = __shfl_up_sync(0xffffffffu, sA, o);
            const double pc = __shfl_up_sync(0xffffffffu, sc, o);
            if (lane >= o) {
                sc = __fma_rn(sA, pc, sc);
                sA = __dmul_rn(sA, pA);
            }
        }
        double y0 = 0.0;  // y entering this warp's first chunk
        if (W > 1) {
            if (lane == 31) {
                tot[0][warp][0] = sA;
                tot[0][warp][1] = sc;
            }
            __syncthreads();
            for (int hh = 0; hh < h; ++hh) y0 = __fma_rn(tot[0][hh * KT + wc][0], y0, tot[0][hh * KT + wc][1]);
        }
        const double eA = __shfl_up_sync(0xffffffffu, sA, 1), ec = __shfl_up_sync(0xffffffffu, sc, 1);
        maps[0][wc][ch] = (lane == 0) ? y0 : __fma_rn(eA, y0, ec);
    }
    __syncthreads();
    const double yin = maps[0][c][q];
    // Fix-up of y, then the local back substitution from the chunk end:
    // x~_b = y_b g_b, x~_p = (y_p - x~_{p+1}) g_p; x_p = x~_p + B_p x_{b+1},
    // B_b = -g_b, B_p = -g_p B_{p+1}.
    double B, x;
    auto backward = [&](auto g) {
        double Ap = -g(a - 1);
        v[0] = __fma_rn(Ap, yin, v[0]);
#pragma unroll
        for (int t = 1; t < RR; ++t) {
            if (t < R) {
                Ap = __dmul_rn(-g(a + t - 1), Ap);
                v[t] = __fma_rn(Ap, yin, v[t]);
            }
        }
        x = 0.0;
        B = -1.0;  // B_b = -g_b
#pragma unroll
        for (int t = RR - 1; t >= 0; --t) {
            if (t < R) {
                const double gp = g(a + t);
                x = __dmul_rn(__dsub_rn(v[t], x), gp);
                v[t] = x;
                B = t == R - 1 ? -gp : __dmul_rn(-gp, B);
            }
        }
    };
    if (flat)
        backward(F);
    else
        backward(G);
    // Reverse inclusive scan of x_start = c + B x_next, then the column's
    // later warps' totals composed in order.
    __syncthreads();  // every lane has read its carry
    maps[0][c][q] = B;
    maps[1][c][q] = x;
    __syncthreads();
    {
        double rB = maps[0][wc][ch], rc = maps[1][wc][ch];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double nB = __shfl_down_sync(0xffffffffu, rB, o);
            const double nc = __shfl_down_sync(0xffffffffu, rc, o);
            if (lane + o < 32) {
                rc = __fma_rn(rB, nc, rc);
                rB = __dmul_rn(rB, nB);
            }
        }
        double x0 = 0.0;  // x entering this warp's last chunk from above
        if (W > 1) {
            if (lane == 0) {
                tot[1][warp][0] = rB;
                tot[1][warp][1] = rc;
            }
            __syncthreads();
            for (int hh = W - 1; hh > h; --hh) x0 = __fma_rn(tot[1][hh * KT + wc][0], x0, tot[1][hh * KT + wc][1]);
        }
        const double nB = __shfl_down_sync(0xffffffffu, rB, 1), nc = __shfl_down_sync(0xffffffffu, rc, 1);
        maps[0][wc][ch] = (lane == 31) ? x0 : __fma_rn(nB, x0, nc);
    }
    __syncthreads();
    const double xin = maps[0][c][q];
    double lsum = 0.0;
    auto finish = [&](auto g) {
        double Bp = -1.0;
#pragma unroll
        for (int t = RR - 1; t >= 0; --t) {
            if (t < R) {
                const double gp = g(a + t);
                Bp = t == R - 1 ? -gp : __dmul_rn(-gp, Bp);
                v[t] = __fma_rn(Bp, xin, v[t]);
                lsum = __dadd_rn(lsum, v[t]);
            }
        }
    };
    if (flat)
        finish(F);
    else
        finish(G);
    if (Mb.periodic) {
        // periodic_ge (qg3p_helmholtz.F90:565-610): the cyclic closure
        // through the rows 1 and jj, which the Thomas solve above leaves
        // out, as two rank-one corrections with the precomputed b, c.
        if (q == 0) ends[0][c] = v[0];                   // row 2 (1-based) after the solve
#pragma unroll
        for (int t = 0; t < RR; ++t)
            if (t < R && a + t == Mr) ends[1][c] = v[t];  // row jj-1
        double z1i = 0.0, zji = 0.0;  // rows 1 and jj of this mode's spectral field
        if (active) {
            z1i = ld(0);
            zji = ld(jj - 1);
        }
        __syncthreads();  // every warp has read rows 1 and jj before they are written
        if (active) {
            const double* pb = Mb.pb + (long long)m * jj * n + kk;
            const double* pc = Mb.pc + (long long)m * jj * n + kk;
            const double z1 = (z1i - ends[0][c]) / __ldg(&pb[0]);
            const double zj = ((zji - ends[1][c]) - z1 * __ldg(&pb[(long long)(jj - 1) * n])) /
                              __ldg(&pc[(long long)(jj - 1) * n]);
            lsum = 0.0;  // the column sum over every row of the closed solution
#pragma unroll
            for (int t = 0; t < RR; ++t) {
                if (t < R && a + t <= Mr) {
                    const long long row = a + t;  // 0-based grid row
                    v[t] = (v[t] - z1 * __ldg(&pb[row * n])) - zj * __ldg(&pc[row * n]);
                    lsum += v[t];
                }
            }
            if (q == 0) {
                const double r0 = z1 - zj * __ldg(&pc[0]);
                if (f32) {
                    reinterpret_cast<float*>(sp)[0] = (float)r0;
                    reinterpret_cast<float*>(sp)[(long long)(jj - 1) * pitch] = (float)zj;
                } else {
                    reinterpret_cast<double*>(sp)[0] = r0;
                    reinterpret_cast<double*>(sp)[(long long)(jj - 1) * pitch] = zj;
                }
                lsum += r0 + zj;
            }
        }
    }
    if (active) {
        if (!f32) {
            double* p = reinterpret_cast<double*>(sp) + (long long)a * pitch;
#pragma unroll
            for (int t = 0; t < RR; ++t)
                if (t < R && a + t <= Mr) p[(long long)t * pitch] = v[t];
        } else {
            float* p = reinterpret_cast<float*>(sp) + (long long)a * pitch;
#pragma unroll
            for (int t = 0; t < RR; ++t)
                if (t < R && a + t <= Mr) p[(long long)t * pitch] = (float)v[t];
        }
    }
    pdl_release();
    if (!do_mean) return;
    // Closed basin: the domain mean of the mode (wmean weights).  Channel:
    // the mean PV of the two walls (zeta_boundary of the solved mode,
    // qg3p_aux.F90:289-379), linear in the column sums: sum_j phi(i, j) =
    // 2 sum_k sin(i k pi / N) C_k, so wall i = 0 gets wwall[k] C_k and wall
    // ii - 1 gets (-1)^(k+1) wwall[k] C_k.
    maps[1][c][q] = lsum;  // (its last readers passed a barrier)
    __syncthreads();
    {
        const double cs = warp_sum(maps[1][wc][ch]);
        if (lane == 0) {
            double t = 0.0, t2 = 0.0;
            if (tile * KT + wc < n) {
                t = cs * wm;
                t2 = (wc & 1) ? -t : t;  // the tile's first column is even
            }
            wpart[warp] = t;
            wpart2[warp] = t2;
        }
    }
    __syncthreads();
    publish_means(Mb, local, tiles_per_mode, wpart, wpart2, &is_last);
}

// ---------------------------------------------------------------------------
// The same solves for columns of more than 32 rows per chunk (more than 2050
// grid rows), whose chunks no longer fit registers.
//
// The CTA's KT columns are staged in shared memory by cp.async and swept there:
// row t of chunk q of column c at c CS + q RS + t, RS = R | 1 odd, so that the
// 32 chunks of a column that a warp sweeps lie in 32 banks.  What bounds it: the
// chain of shared-memory sweeps, on three CTAs per SM at 2051 rows and one from
// 3600.  Instances of k_tridiag with 64 and 128 rows in registers spilled 2 to
// 12 KB per thread; us per solve with them and here: 257 x 2561 x 3 57 -> 30 FP64,
// 71 -> 29 mixed, 257 x 4500 x 3 358 -> 45 and 274 -> 45, 2049 x 2561 x 3 349 -> 126
// and 390 -> 119, 2049 x 4097 x 3 324 -> 225 and 263 -> 218.  Chunks of up to 32 rows
// stay in registers (257 x 2049 x 3: 20 us, 33 for a strip).  A strip laid out by
// thread (no transpose) took 1.4 to 2 times as long.  The arithmetic is
// k_tridiag's, operation for operation.
//
// Column stride of the strip: NQ RS plus a pad that makes the 16 threads of a
// half-warp of the staging and write-back phases (KT columns x 16 / KT chunks
// each) hit 16 distinct 8-byte bank pairs: NQ RS is a multiple of 16, so
// c CS + q RS = RS (c 16 / KT + q) (mod 16) with RS odd.
__host__ __device__ inline int tri_cs(int NQ, int RS, int KT) { return NQ * RS + (RS * (16 / KT)) % 16; }

template <typename S>
__global__ void __launch_bounds__(TRI_THREADS) k_tridiag_strip(const Member* __restrict__ mems,
                                                                const int* __restrict__ prefix, int nmem, int do_mean,
                                                                const __grid_constant__ Member one, int use_one) {
    __shared__ Member Mb;
    __shared__ double wpart[8], wpart2[8];
    __shared__ double tot[2][8][2];  // per warp: affine totals (forward, backward)
    __shared__ int is_last;
    extern __shared__ __align__(16) double strip[];
    pdl_wait();
    int local;
    cta_member(Mb, one, use_one, mems, prefix, nmem, blockIdx.x, &local);
    __syncthreads();
    const int n = Mb.n, jj = Mb.jj, pitch = Mb.pitch;
    const int W = tri_warps(jj), KT = 8 / W, NQ = 32 * W;
    const int tiles_per_mode = (n + KT - 1) / KT;
    const int m = local / tiles_per_mode, tile = local - m * tiles_per_mode;
    const int k0 = tile * KT;  // the tile's first column (0-based)
    const int Mr = jj - 2, R = (Mr + NQ - 1) / NQ, RS = R | 1, CS = tri_cs(NQ, RS, KT);
    const bool f32 = sizeof(S) == 4 && m > 0;  // this mode's rows are FP32
    double* const spec = (sizeof(S) == 4 ? Mb.spec64 : reinterpret_cast<double*>(Mb.spec)) + (long long)m * Mb.lstride;
    float* const specf = reinterpret_cast<float*>(Mb.spec) + (long long)m * Mb.lstride;

    // Stage: thread -> (column, chunk), a copy per row; columns past n are zeros.
    {
        const int c = threadIdx.x % KT, q = threadIdx.x / KT;
        const bool ok = k0 + c < n;
        const long long go = (long long)(q * R + 1) * pitch + (ok ? k0 + c : 0);
        double* const d = strip + c * CS + q * RS;
        const int Rq = min(R, Mr - q * R);
        if (!f32) {
            const unsigned da = (unsigned)__cvta_generic_to_shared(d);
            for (int t = 0; t < Rq; ++t)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(da + 8u * t),
                             "l"(spec + go + (long long)t * pitch), "r"(ok ? 8 : 0)
                             : "memory");
            cp_commit_wait_all();
        } else {
            // FP32 rows into the upper half of the chunk's slots (float t at
            // float RS + t), then widened in place: double t covers floats 2t
            // and 2t + 1 < RS + t, so each float is read before it is overwritten.
            const unsigned fa = (unsigned)__cvta_generic_to_shared(reinterpret_cast<float*>(d) + RS);
            for (int t = 0; t < Rq; ++t)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(fa + 4u * t),
                             "l"(specf + go + (long long)t * pitch), "r"(ok ? 4 : 0)
                             : "memory");
            cp_commit_wait_all();
            const float* const f = reinterpret_cast<const float*>(d) + RS;
            for (int t = 0; t < Rq; ++t) d[t] = (double)f[t];
        }
    }
    __syncthreads();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = warp % KT, h = warp / KT;  // column, and which W-th of it
    const int q = h * 32 + lane, kk = k0 + c;
    const bool active = kk < n;
    const int a = q * R + 1, cnt = max(0, min(R, Mr - q * R)), b = a + cnt - 1;  // row positions (1-based)
    double* const s = strip + c * CS + q * RS;  // s[t] is position a + t
    const double* piv = nullptr;
    int len = 0;
    double fix = 0.0;
    if (active) {
        const int mk = m * n + kk;
        piv = Mb.piv + __ldg(&Mb.piv_off[mk]);
        len = __ldg(&Mb.piv_len[mk]);
        fix = __ldg(&Mb.piv_fix[mk]);
    }
    auto G = [&](int p) -> double { return p <= len ? __ldg(piv + p - 1) : fix; };

    // Forward elimination and its scan (k_tridiag).
    double A = 1.0, y = 0.0;
    if (active && cnt > 0) {
        A = (a > 1) ? -G(a - 1) : 0.0;
        y = s[0];
        for (int t = 1; t < cnt; ++t) {
            const double gp = G(a + t - 1);
            y = __fma_rn(-gp, y, s[t]);
            s[t] = y;
            A = __dmul_rn(-gp, A);
        }
    }
    double sA = A, sc = y;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double pA = __shfl_up_sync(0xffffffffu, sA, o);
        const double pc = __shfl_up_sync(0xffffffffu, sc, o);
        if (lane >= o) {
            sc = __fma_rn(sA, pc, sc);
            sA = __dmul_rn(sA, pA);
        }
    }
    if (lane == 31) {
        tot[0][warp][0] = sA;
        tot[0][warp][1] = sc;
    }
    __syncthreads();
    double y0 = 0.0;  // y entering this warp's first chunk
    for (int hh = 0; hh < h; ++hh) y0 = __fma_rn(tot[0][hh * KT + c][0], y0, tot[0][hh * KT + c][1]);
    const double eA = __shfl_up_sync(0xffffffffu, sA, 1), ec = __shfl_up_sync(0xffffffffu, sc, 1);
    const double yin = (lane == 0) ? y0 : __fma_rn(eA, y0, ec);
    // Fix-up of y, local back substitution, its reverse scan.
    double B = 1.0, x = 0.0;
    if (active && cnt > 0) {
        double Ap = (a > 1) ? -G(a - 1) : 0.0;
        const double gb = G(b);
        s[0] = __fma_rn(Ap, yin, s[0]);
        for (int t = 1; t < cnt; ++t) {
            Ap = __dmul_rn(-G(a + t - 1), Ap);
            s[t] = __fma_rn(Ap, yin, s[t]);
        }
        x = __dmul_rn(s[cnt - 1], gb);
        s[cnt - 1] = x;
        B = -gb;
        for (int t = cnt - 2; t >= 0; --t) {
            const double gp = G(a + t);
            x = __dmul_rn(__dsub_rn(s[t], x), gp);
            s[t] = x;
            B = __dmul_rn(-gp, B);
        }
    }
    double rB = B, rc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double nB = __shfl_down_sync(0xffffffffu, rB, o);
        const double nc = __shfl_down_sync(0xffffffffu, rc, o);
        if (lane + o < 32) {
            rc = __fma_rn(rB, nc, rc);
            rB = __dmul_rn(rB, nB);
        }
    }
    if (lane == 0) {
        tot[1][warp][0] = rB;
        tot[1][warp][1] = rc;
    }
    __syncthreads();
    double x0 = 0.0;  // x entering this warp's last chunk from above
    for (int hh = W - 1; hh > h; --hh) x0 = __fma_rn(tot[1][hh * KT + c][0], x0, tot[1][hh * KT + c][1]);
    const double nB = __shfl_down_sync(0xffffffffu, rB, 1), nc = __shfl_down_sync(0xffffffffu, rc, 1);
    const double xin = (lane == 31) ? x0 : __fma_rn(nB, x0, nc);
    double lsum = 0.0;
    if (active && cnt > 0) {
        double Bp = -G(b);
        double u = __fma_rn(Bp, xin, s[cnt - 1]);
        s[cnt - 1] = u;
        lsum = __dadd_rn(lsum, u);
        for (int t = cnt - 2; t >= 0; --t) {
            Bp = __dmul_rn(-G(a + t), Bp);
            u = __fma_rn(Bp, xin, s[t]);
            s[t] = u;
            lsum = __dadd_rn(lsum, u);
        }
    }
    if (Mb.periodic) {
        // The cyclic closure (k_tridiag).
        __syncthreads();
        double z1 = 0.0, zj = 0.0;
        const double* const pb = Mb.pb + (long long)m * jj * n + kk;
        const double* const pc = Mb.pc + (long long)m * jj * n + kk;
        if (active) {
            const int ql = (Mr - 1) / R;  // row jj-1's chunk
            const double z1i = f32 ? (double)specf[kk] : spec[kk];
            const double zji = f32 ? (double)specf[(long long)(jj - 1) * pitch + kk] : spec[(long long)(jj - 1) * pitch + kk];
            z1 = (z1i - strip[c * CS]) / __ldg(&pb[0]);
            zj = ((zji - strip[c * CS + ql * RS + (Mr - 1) - ql * R]) - z1 * __ldg(&pb[(long long)(jj - 1) * n])) /
                 __ldg(&pc[(long long)(jj - 1) * n]);
        }
        __syncthreads();  // every warp has read rows 1 and jj, and the strip's ends, before they are written
        if (active) {
            lsum = 0.0;  // the column sum over every row of the closed solution
            for (int t = 0; t < cnt; ++t) {
                const long long row = a + t;  // 0-based grid row
                const double u = (s[t] - z1 * __ldg(&pb[row * n])) - zj * __ldg(&pc[row * n]);
                s[t] = u;
                lsum += u;
            }
            if (q == 0) {
                const double r0 = z1 - zj * __ldg(&pc[0]);
                if (f32) {
                    specf[kk] = (float)r0;
                    specf[(long long)(jj - 1) * pitch + kk] = (float)zj;
                } else {
                    spec[kk] = r0;
                    spec[(long long)(jj - 1) * pitch + kk] = zj;
                }
                lsum += r0 + zj;
            }
        }
    }
    if (do_mean) {
        const double cs = warp_sum(lsum);
        if (lane == 0) {
            const double t = active ? cs * __ldg((Mb.periodic ? Mb.wwall : Mb.wmean) + kk) : 0.0;
            wpart[warp] = t;
            wpart2[warp] = (kk & 1) ? -t : t;
        }
    }
    pdl_release();
    __syncthreads();
    {
        const int cc = threadIdx.x % KT, qq = threadIdx.x / KT;
        if (k0 + cc < n) {
            const long long go = (long long)(qq * R + 1) * pitch + k0 + cc;
            const double* const d = strip + cc * CS + qq * RS;
            const int Rq = min(R, Mr - qq * R);
            if (!f32) {
                for (int t = 0; t < Rq; ++t) spec[go + (long long)t * pitch] = d[t];
            } else {
                for (int t = 0; t < Rq; ++t) specf[go + (long long)t * pitch] = (float)d[t];
            }
        }
    }
    if (do_mean) publish_means(Mb, local, tiles_per_mode, wpart, wpart2, &is_last);
}

template <typename S, int RR, int KT>
static cudaError_t launch_tri(const LaunchSet& ls, int do_mean, cudaStream_t st) {
    constexpr int NQ = 256 / KT;
    const int R = (ls.maxJ - 2 + NQ - 1) / NQ;
    const size_t bytes = (size_t)KT * tri_pitch(NQ * R, KT) * sizeof(double);
    void (*kern)(const Member*, const int*, int, int, Member, int);
    if (R == RR)
        kern = member_arg_used(ls) ? k_tridiag<S, RR, KT, true, true> : k_tridiag<S, RR, KT, true, false>;
    else
        kern = member_arg_used(ls) ? k_tridiag<S, RR, KT, false, true> : k_tridiag<S, RR, KT, false, false>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    return launch_step_kernel(ls.pdl, kern, dim3(ls.ctas_tri), dim3(TRI_THREADS), bytes, st, ls.members,
                              ls.prefix_tri, ls.nmem, do_mean, member_arg(ls), member_arg_used(ls));
}

constexpr int TRI_MAX_ROWS = 8192;

template <typename S>
static cudaError_t launch_tri_strip(const LaunchSet& ls, int do_mean, cudaStream_t st) {
    const int W = tri_warps(ls.maxJ), KT = 8 / W, NQ = 32 * W, R = (ls.maxJ - 2 + NQ - 1) / NQ;
    const size_t bytes = (size_t)KT * tri_cs(NQ, R | 1, KT) * sizeof(double);
    cudaError_t e =
        cudaFuncSetAttribute(k_tridiag_strip<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    return launch_step_kernel(ls.pdl, k_tridiag_strip<S>, dim3(ls.ctas_tri), dim3(TRI_THREADS), bytes, st, ls.members,
                              ls.prefix_tri, ls.nmem, do_mean, member_arg(ls), member_arg_used(ls));
}

// The instance that holds chunks of R rows (every member of a launch has
// ls.maxJ rows per column); longer chunks are swept in shared memory, of columns
// of up to TRI_MAX_ROWS.
template <typename S>
static cudaError_t launch_tri_rows(const LaunchSet& ls, int do_mean, cudaStream_t st) {
    const int W = tri_warps(ls.maxJ), R = (ls.maxJ - 2 + 32 * W - 1) / (32 * W);
    if (W == 1) return launch_tri<S, 2, 8>(ls, do_mean, st);
    if (R <= 3) return launch_tri<S, 3, 4>(ls, do_mean, st);
    if (R <= 4) return launch_tri<S, 4, 4>(ls, do_mean, st);
    if (R <= 6) return launch_tri<S, 6, 4>(ls, do_mean, st);
    if (R <= 8) return launch_tri<S, 8, 4>(ls, do_mean, st);
    if (R <= 12) return launch_tri<S, 12, 4>(ls, do_mean, st);
    if (R <= 16) return launch_tri<S, 16, 4>(ls, do_mean, st);
    if (R <= 20) return launch_tri<S, 20, 4>(ls, do_mean, st);
    if (R <= 24) return launch_tri<S, 24, 4>(ls, do_mean, st);
    if (W == 2 && R <= 32) return launch_tri<S, 32, 4>(ls, do_mean, st);
    return ls.maxJ - 2 <= TRI_MAX_ROWS ? launch_tri_strip<S>(ls, do_mean, st) : cudaErrorInvalidValue;
}

cudaError_t launch_tridiag(const LaunchSet& ls, int do_mean, int f32, cudaStream_t st) {
    return f32 ? launch_tri_rows<float>(ls, do_mean, st) : launch_tri_rows<double>(ls, do_mean, st);
}

}  // namespace pq
