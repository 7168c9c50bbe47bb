// pq_cabaret.cu -- the CABARET advection step after the PV inversion, fused.
//
// Everything between the PV inversion and the next step's predictor, in the
// reference's order (qg3.F90:641-957), in one pass over the fields:
//   rel_from_zeta_and_psi + apply_rel_bc     qg3p_aux.F90:738-915
//   update_zeta_bc                           :643-734
//   cabaret_forcing                          :1065-1164
//   cabaret_cell_boundaries_time_integrated  :1235-1313
//   cabaret_extrapolator (+ limiter)         :1317-1544
//   cabaret_flux                             :1547-1594
//   cabaret_corrector + set(zeta_old, zeta)  :1597-1642, qg3.F90:957
// writing back only the fields the next step needs.  Halo values are
// recomputed, never exchanged.  Fields read at nodes or faces owned by another
// warp (zeta_old, uimo, ujmo, zeta_fi, zeta_fj) are ping-ponged.
#include <algorithm>

#include "pq_common.cuh"
#include "pq_kernels.h"

namespace pq {

// Sweep decomposition: a warp owns one layer of a strip of 32 NC columns --
// NC consecutive columns per lane, cab_sw(NC) = 32 NC - 4 output columns plus
// 2 halo columns on each side -- and marches down a band of Mb.cab_sh output
// rows (a tuning parameter).  Every per-lane quantity lives in registers as
// a rolling window over rows; the i-neighbours come from the lane's own
// columns or, across a lane boundary, from warp shuffles.  At iteration k
// (s = j0 + k - 2) the warp takes psi row s and the inputs of rows s, s-1, s-2,
// and produces
//   rel(s), zeta after BC/forcing at row s-1, uj on face row s, ui on row s-1,
//   zeta_fj on face row s-1, zeta_fi on row s-1, and res / zeta_old at row s-2.
// NC = 2 (FP32 fields only, pq_tuning.cab_kernel = 2): each row access of a
// field is one 8-byte vector per lane (16 bytes for psi) and one shuffle
// serves two columns; it needs more registers (two CTAs per SM instead of
// three), so it pays on large grids (2049^2 x 5).
//
// What bounds it: instruction issue and latency at 12 warps per SM (issue
// active 45-50 %, DRAM 45-65 % of its peak), and the end of the sweep queue.
// 1025^2 x 3, us per launch, FP64 / mixed: 133 / 98 with a copy and an address
// per lane and field, one cp.async each; 121 / 93 with the descriptor read from the kernel's
// parameters (field bases in uniform registers), one-sided shuffles and FP64
// max / min as selects; 120 / 90 with edge sweeps on the same iteration and
// 16-byte copies; 107 / 75 with every wall sweep claimed first, bands sized to
// the resident warps and the step finished by the last warp.  Bulk copies
// (cp.async.bulk, a row of a field each) were slower (134 / 122): one lane's
// operands at a time.  More CTAs per SM (4, 5) gave nothing at FP64 (125, 170)
// and 2 % mixed.  513^2 x 3: 58 / 43 (tiles) -> 42 / 32; 2049^2 x 5 631 / 405 ->
// 599 / 373.
constexpr int CAB_WARPS = 4;
constexpr int CAB_D = 4;  // depth of the per-warp cp.async row pipeline
__host__ __device__ constexpr int cab_sw(int nc) { return 32 * nc - 4; }  // output columns per warp

__device__ __forceinline__ double shup(double v, int d) { return __shfl_up_sync(0xffffffffu, v, d); }
__device__ __forceinline__ double shdn(double v, int d) { return __shfl_down_sync(0xffffffffu, v, d); }
__device__ __forceinline__ float shup(float v, int d) { return __shfl_up_sync(0xffffffffu, v, d); }
__device__ __forceinline__ float shdn(float v, int d) { return __shfl_down_sync(0xffffffffu, v, d); }

// Neighbours of a lane's NC columns: o[c] = v at column (c - 1), (c + 1),
// (c - 2), (c + 2) of the lane's frame.  Every lane must call them (shuffles).
template <int NC, typename V>
__device__ __forceinline__ void col_up(const V (&v)[NC], V (&o)[NC]) {
    const V t = shup(v[NC - 1], 1);
#pragma unroll
    for (int c = NC - 1; c > 0; --c) o[c] = v[c - 1];
    o[0] = t;
}
template <int NC, typename V>
__device__ __forceinline__ void col_dn(const V (&v)[NC], V (&o)[NC]) {
    const V t = shdn(v[0], 1);
#pragma unroll
    for (int c = 0; c < NC - 1; ++c) o[c] = v[c + 1];
    o[NC - 1] = t;
}
template <int NC, typename V>
__device__ __forceinline__ void col_up2(const V (&v)[NC], V (&o)[NC]) {
    if constexpr (NC == 1) {
        o[0] = shup(v[0], 2);
    } else {
        const V t0 = shup(v[NC - 2], 1), t1 = shup(v[NC - 1], 1);
#pragma unroll
        for (int c = NC - 1; c > 1; --c) o[c] = v[c - 2];
        o[0] = t0;
        o[1] = t1;
    }
}
template <int NC, typename V>
__device__ __forceinline__ void col_dn2(const V (&v)[NC], V (&o)[NC]) {
    if constexpr (NC == 1) {
        o[0] = shdn(v[0], 2);
    } else {
        const V t0 = shdn(v[0], 1), t1 = shdn(v[1], 1);
#pragma unroll
        for (int c = 0; c < NC - 2; ++c) o[c] = v[c + 2];
        o[NC - 2] = t0;
        o[NC - 1] = t1;
    }
}
// NC consecutive values: one vector access (shared or global memory).
template <int NC, typename V>
__device__ __forceinline__ void vld(const V* p, V (&v)[NC]) {
    if constexpr (NC == 1) {
        v[0] = p[0];
    } else if constexpr (sizeof(V) == 8) {
        const double2 t = *reinterpret_cast<const double2*>(p);
        v[0] = t.x;
        v[1] = t.y;
    } else {
        const float2 t = *reinterpret_cast<const float2*>(p);
        v[0] = t.x;
        v[1] = t.y;
    }
}
template <int NC, typename V>
__device__ __forceinline__ void vst(V* p, const V (&v)[NC]) {
    if constexpr (NC == 1) {
        p[0] = v[0];
    } else if constexpr (sizeof(V) == 8) {
        *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
    } else {
        *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
    }
}
// z + f r, the forcing added to zeta.  FP32 written out, so that a mixed run
// does not depend on what the compiler contracts: the product rounded first,
// as in the tile kernel.  `once` rounds the sum only: the second column of a
// two-column edge sweep has always done so, and is kept bit for bit.
__device__ __forceinline__ double add_scaled(double z, double f, double r, bool) { return z + f * r; }
__device__ __forceinline__ float add_scaled(float z, float f, float r, bool once) {
    return once ? __fmaf_rn(f, r, z) : __fadd_rn(z, __fmul_rn(f, r));
}
// max / min as one comparison and a select: FP64 fmax is a sequence around the
// NaN rules, which the limiter does not need (a NaN in any of its inputs is in
// zeta too and poisons the next inversion).
__device__ __forceinline__ double mx(double a, double b) { return a > b ? a : b; }
__device__ __forceinline__ double mn(double a, double b) { return a < b ? a : b; }
__device__ __forceinline__ float mx(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ float mn(float a, float b) { return fminf(a, b); }
// The input rows of an iteration come in 16-byte chunks (cp.async.cg: no line of the L1 cache
// is held while a copy is in flight; a field's row copied 8 bytes per lane holds
// three lines, and the L1 cache left beside the rings bounds how many fly).  The rows of an iteration lie one after another in a ring stage --
// first the FP64 ones, then the T ones -- and instruction q of a class copies
// chunks 32 q .. 32 q + 31 of them: a lane's chunk belongs to one field for
// the whole sweep, so its address is one pointer that moves a row down per
// iteration.  T = float rows start two columns early and are four values
// longer, so that every chunk starts on 16 bytes (i0 is a multiple of 28 or 60).
enum { G_PSI = 0, G_PSIM, G_PSIP, G_WIND, G_N64 };
enum { G_ZPB = 0, G_ZO, G_UIMO, G_UJMO, G_FIO, G_FJ, G_RB, G_NT };
template <typename T, int NC> struct CabRing {
    static constexpr int LEAD = sizeof(T) == 4 ? 2 : 0;
    static constexpr int B64 = 32 * NC * 8, BT = (32 * NC + 2 * LEAD) * (int)sizeof(T);  // bytes of a row
    static constexpr int C64 = G_N64 * B64 / 16, CT = G_NT * BT / 16;                    // chunks of a stage
    static constexpr int Q64 = (C64 + 31) / 32, QT = (CT + 31) / 32;                     // copy instructions
    static constexpr int STAGE = G_N64 * B64 + G_NT * BT;
    __host__ __device__ static constexpr int bytes() { return CAB_D * STAGE; }
};
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
template <int OFF>
__device__ __forceinline__ void cp_chunk(unsigned dst, const void* src, unsigned bytes) {  // bytes 0: zeros
    asm volatile("cp.async.cg.shared.global [%0+%2], [%1], 16, %3;\n" ::"r"(dst), "l"(src), "n"(OFF), "r"(bytes)
                 : "memory");
}

// One warp's sweep over layer l of the strip starting at column i0 and the
// band of rows j0 .. j0+SH-1.  EDGE = false is the specialisation for warps
// whose whole footprint (columns i0-2 .. i0+32NC-3, rows j0-4 .. j0+SH+3) lies
// at least two nodes inside the domain; EDGE = true runs the same iteration
// and replaces what differs at the walls (rows by warp-uniform branches, the
// columns of a strip that touches a wall per lane), masking values outside
// the domain to zero.  PRED = true also applies the next step's
// cabaret_predictor and cabaret_beta (fixed dt) to every interior
// node it finishes, writing the next step's inversion input zeta_next and
// res_beta_other.  T is the type of the CABARET fields (double, or float in
// the mixed form); psi is FP64 and everything computed from psi differences
// (the rel coupling, the boundary rel, the corner streamfunction and the face
// velocities before the time weighting) is evaluated in FP64.  Returns the
// largest |u| of the faces it wrote.
template <bool EDGE, bool PRED, typename T, int NC>
__device__ __forceinline__ double cab_sweep(const Member& Mb, int l, int i0, int j0, int SH, int lane, char* ring) {
    static_assert(NC == 1 || NC == 2, "one or two columns per lane");
    using RG = CabRing<T, NC>;
    const int L = Mb.L, pitch = Mb.pitch, ii = Mb.ii, jj = Mb.jj;
    const long long ls = Mb.lstride;
    constexpr int HL = 2 / NC;  // halo lanes on each side
    const bool out_lane = lane >= HL && lane < 32 - HL;
    const int cur = Mb.cur, nxt = cur ^ 1;
    const double dt64 = Mb.sc->dt;
    const T dt = (T)dt64, tu = (T)Mb.sc->tweight_u;
    const bool avg = cab_average_gate(Mb);
    const T hdt = (T)0.5 * dt;
    const T ta = (T)Mb.sc->tweight_a, beta_l = (T)Mb.beta[l];
    const bool has_wind = (l == 0 && Mb.wind);
    const T nu = (T)Mb.viscosity, vb = (T)Mb.visc_bot;
    const double s1 = Mb.s1[l], s2 = Mb.s2[l];
    const bool lim = Mb.limiter != 0;
    const bool top = (l == 0), bottom = (l == L - 1);
    T umax = 0;  // |u| is exact in T: widened once at the end
    const int ib = i0 - 2 + NC * lane;  // the lane's first column
    // Column masks (true inside): nodes, interior nodes, i-faces a = i.
    auto in_i = [&](int c) { return !EDGE || (ib + c >= 0 && ib + c < ii); };
    auto int_i = [&](int c) { return !EDGE || (ib + c >= 1 && ib + c <= ii - 2); };
    auto fac_i = [&](int c) { return !EDGE || (ib + c >= 1 && ib + c <= ii - 1); };
    auto in_j = [&](int j) { return !EDGE || (j >= 0 && j < jj); };
    auto int_j = [&](int j) { return !EDGE || (j >= 1 && j <= jj - 2); };
    const bool walls = EDGE && (i0 - 2 <= 0 || i0 + 32 * NC - 3 >= ii - 1);  // the strip holds a wall column
    const int bc = Mb.bc_type;
    const double cffbc = Mb.alpha / (Mb.alpha + 3.0);

    // This lane's chunks: their addresses at the next row to copy, and 16 or,
    // where the field does not exist, 0 bytes.
    const int n = SH + 4;
    const char *c64[RG::Q64], *cT[RG::QT];
    unsigned b64[RG::Q64], bT[RG::QT];
    int r64[RG::Q64], rT[RG::QT];  // EDGE: the row the chunk comes from at the next copy
#pragma unroll
    for (int q = 0; q < RG::Q64; ++q) {
        const int c = 32 * q + lane, f = c * 16 / RG::B64, col = (c * 16 % RG::B64) / 8;
        const bool on = f == G_PSI || (f == G_PSIM && !top) || (f == G_PSIP && !bottom) || (f == G_WIND && has_wind);
        const int layer = f == G_WIND ? 0 : f == G_PSIM ? l - 1 : f == G_PSIP ? l + 1 : l;
        const double* base = f == G_WIND ? Mb.wind : Mb.psi;
        r64[q] = j0 - 2 - (f == G_WIND ? 1 : 0);
        // Outside the row (a chunk lies wholly inside or outside it): zeros.
        const bool ok = on && (!EDGE || (i0 - 2 + col >= 0 && i0 - 2 + col < pitch));
        b64[q] = ok ? 16u : 0u;
        c64[q] = reinterpret_cast<const char*>(ok ? base + layer * ls + (long long)r64[q] * pitch + (i0 - 2 + col)
                                                  : Mb.psi);
    }
#pragma unroll
    for (int q = 0; q < RG::QT; ++q) {
        const int c = 32 * q + lane, f = c * 16 / RG::BT, col = (c * 16 % RG::BT) / (int)sizeof(T);
        const void* base = f == G_ZPB    ? Mb.zeta
                           : f == G_ZO   ? Mb.zeta_old[cur]
                           : f == G_UIMO ? Mb.uimo[cur]
                           : f == G_UJMO ? Mb.ujmo[cur]
                           : f == G_FIO  ? Mb.zfi[cur]
                           : f == G_FJ   ? Mb.zfj[cur]
                                         : Mb.res_beta;
        const int d = f == G_RB ? 2 : (f == G_ZO || f == G_UIMO || f == G_FIO) ? 1 : 0;  // rows above s
        const bool on = f < G_RB || (f == G_RB && PRED);
        rT[q] = j0 - 2 - d;
        const int gc = i0 - 2 - RG::LEAD + col;
        const bool ok = on && (!EDGE || (gc >= 0 && gc < pitch));
        bT[q] = ok ? 16u : 0u;
        cT[q] = reinterpret_cast<const char*>(ok ? static_cast<const T*>(base) + l * ls + (long long)rT[q] * pitch + gc
                                                 : static_cast<const T*>(Mb.zeta));
    }
    const unsigned p64 = (unsigned)pitch * 8u, pT = (unsigned)pitch * (unsigned)sizeof(T);
    const unsigned ring_a = smem_addr(ring) + 16u * lane;
    auto issue = [&](int k) {
        const unsigned dst = ring_a + (unsigned)(k % CAB_D) * RG::STAGE;
        // chunk 32 q + lane of each class, the last instruction's lanes past its end left out
#define PQ_CP64(q)                                                                     \
    if constexpr (q < RG::Q64) {                                                       \
        const bool in = !EDGE || (r64[q] >= 0 && r64[q] < jj);                         \
        if (32 * q + 32 <= RG::C64 || 32 * q + lane < RG::C64)                         \
            cp_chunk<512 * q>(dst, in ? c64[q] : reinterpret_cast<const char*>(Mb.psi), in ? b64[q] : 0u); \
        c64[q] += b64[q] ? p64 : 0u;                                                   \
        ++r64[q];                                                                      \
    }
#define PQ_CPT(q)                                                                      \
    if constexpr (q < RG::QT) {                                                        \
        const bool in = !EDGE || (rT[q] >= 0 && rT[q] < jj);                           \
        if (32 * q + 32 <= RG::CT || 32 * q + lane < RG::CT)                           \
            cp_chunk<G_N64 * RG::B64 + 512 * q>(dst, in ? cT[q] : reinterpret_cast<const char*>(Mb.psi), \
                                                in ? bT[q] : 0u);                      \
        cT[q] += bT[q] ? pT : 0u;                                                      \
        ++rT[q];                                                                       \
    }
        PQ_CP64(0) PQ_CP64(1) PQ_CP64(2) PQ_CP64(3)
        PQ_CPT(0) PQ_CPT(1) PQ_CPT(2) PQ_CPT(3)
#undef PQ_CP64
#undef PQ_CPT
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    static_assert(RG::Q64 <= 4 && RG::QT <= 4, "copy instructions per stage");
    for (int k = 0; k < CAB_D - 1; ++k) issue(k);  // n > CAB_D - 1 (SH >= 1)

    // Output addresses: element (row, this lane's first column) of a field.
    const long long lo = l * ls + ib;
    T* const p_res = reinterpret_cast<T*>(Mb.res_out) + lo;
    T* const p_zn = reinterpret_cast<T*>(Mb.zeta_old[nxt]) + lo;
    T* const p_rbn = reinterpret_cast<T*>(Mb.res_beta_other) + lo;
    T* const p_zpn = reinterpret_cast<T*>(Mb.zeta_next) + lo;
    T* const p_ui = reinterpret_cast<T*>(Mb.ui) + lo;
    T* const p_uimon = reinterpret_cast<T*>(Mb.uimo[nxt]) + lo;
    T* const p_fin = reinterpret_cast<T*>(Mb.zfi[nxt]) + lo;
    T* const p_uj = reinterpret_cast<T*>(Mb.uj) + lo;
    T* const p_ujmon = reinterpret_cast<T*>(Mb.ujmo[nxt]) + lo;
    T* const p_fjn = reinterpret_cast<T*>(Mb.zfj[nxt]) + lo;
    double* const p_av = Mb.psi_av + lo;
    const double* const p_psi = Mb.psi + lo;

    // rel_from_zeta_and_psi coupling.
    auto rel_int = [&](T z, double p, double pm, double pp) -> T {
        if (L == 1) return z;
        if (top) return (T)((double)z + s2 * (p - pp));
        if (bottom) return (T)((double)z + s1 * (p - pm));
        return (T)((double)z + s1 * (p - pm) + s2 * (p - pp));
    };
    // Limited upwind extrapolation (cabaret_extrapolator, interior branch).
    // The upwind side only selects the inputs and the sign of the gradient
    // term, so both directions evaluate one instance (no divergent branch).
    auto extrap = [&](T u1, T u2, T fi1, T fi2, T psi_n, T psi_o, bool pos) -> T {
        const T v0 = (u1 + u2) / (T)2;
        const T dfi = pos ? fi1 - fi2 : fi2 - fi1;
        const T d_f = -(psi_n - psi_o) * (T)2 - dt * v0 * dfi;
        T v = (T)2 * psi_n - fi2;
        if (lim) {
            const T fmx = mx(mx(fi1, fi2), psi_n) - d_f;
            const T fmn = mn(mn(fi1, fi2), psi_n) - d_f;
            if (v > fmx) v = fmx;
            if (v < fmn) v = fmn;
        }
        return v;
    };

    // The wall branch: upwind node on the boundary.
    auto extrap_wall = [&](T fi1, T psi_n, T psi_o) -> T {
        const T fi2 = psi_n;
        const T d_f = -(psi_n - psi_o);
        T v = (T)2 * psi_n - fi2;
        if (lim) {
            const T fmx = mx(mx(fi1, fi2), psi_n) - d_f;
            const T fmn = mn(mn(fi1, fi2), psi_n) - d_f;
            if (v > fmx) v = fmx;
            if (v < fmn) v = fmn;
        }
        return v;
    };
    // apply_rel_bc from the wall node and the two nodes inward.
    auto rel_wall = [&](double p, double q1, double q2) -> T {
        if (bc == 3) return (T)0;
        return (T)((bc == 1) ? cffbc * (-3.5 * p + 4.0 * q1 - 0.5 * q2) : 2.0 * (q1 - p));
    };

    // Rolling windows.
    double P1[NC], P2[NC];  // psi rows s-1, s
    T Rm2[NC], Rm1[NC];    // rel rows s-2, s-1
    T ZFm2[NC];            // zeta after forcing, row s-2
    T ZOm2[NC];            // zeta_old row s-2
    T UJm2[NC], UJm1[NC];  // uj faces s-2, s-1
    T FJm2[NC], FJm1[NC];  // zeta_fj (old) faces s-2, s-1
    T FLJm2[NC];           // flux_j face s-2
    T FLI[NC];             // flux_i row s-2 (face a = i)
    T UIm2[NC];            // ui row s-2 (face a = i)
    T zpb_prev[NC];
    double pe_prev[NC];
    [[maybe_unused]] double pm_prev[NC], pp_prev[NC];  // EDGE: psi of the neighbour layers, row s-1
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        P2[c] = (in_j(j0 - 3) && in_i(c)) ? p_psi[(long long)(j0 - 3) * pitch + c] : 0.0;
        Rm2[c] = Rm1[c] = ZFm2[c] = ZOm2[c] = UJm2[c] = UJm1[c] = FJm2[c] = FJm1[c] = FLJm2[c] = FLI[c] = UIm2[c] =
            zpb_prev[c] = 0;
        pe_prev[c] = pm_prev[c] = pp_prev[c] = 0;
    }
    // The left neighbour of P1 (psi row s-1) is, for the lane's first column,
    // the previous row's left neighbour of P2 (carried over, so the corner
    // needs no second shuffle), for the others the lane's own column.
    double up1_prev0 = shup(P2[NC - 1], 1);

#pragma unroll 1
    for (int k = 0; k < n; ++k) {
        const int s = j0 + k - 2;
        // Row k's copies have landed: this lane's (wait), then everyone's (the
        // barrier, which also ends the reads of the stage refilled next).
        asm volatile("cp.async.wait_group %0;\n" ::"n"(CAB_D - 2) : "memory");
        __syncwarp();
        if (k + CAB_D - 1 < n)
            issue(k + CAB_D - 1);
        else
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        const char* st = ring + (k % CAB_D) * RG::STAGE;
        auto get64 = [&](int f, double(&v)[NC]) { vld<NC>(reinterpret_cast<const double*>(st + f * RG::B64) + NC * lane, v); };
        auto gett = [&](int f, T(&v)[NC]) {
            vld<NC>(reinterpret_cast<const T*>(st + G_N64 * RG::B64 + f * RG::BT) + RG::LEAD + NC * lane, v);
        };
        T zpb_s[NC], zo_1[NC], uimo_1[NC], ujmo_s[NC], fio_1[NC], fj_s[NC], w_1[NC], rb_2[NC];
        double pm_s[NC], pp_s[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) P1[c] = P2[c];
        get64(G_PSI, P2);
        get64(G_PSIM, pm_s);  // not read by a layer without that neighbour
        get64(G_PSIP, pp_s);
        gett(G_ZPB, zpb_s);
        gett(G_ZO, zo_1);
        gett(G_UIMO, uimo_1);
        gett(G_UJMO, ujmo_s);
        gett(G_FIO, fio_1);
        gett(G_FJ, fj_s);
        if (has_wind) {
            double w[NC];
            get64(G_WIND, w);
#pragma unroll
            for (int c = 0; c < NC; ++c) w_1[c] = (T)w[c];
        } else {
#pragma unroll
            for (int c = 0; c < NC; ++c) w_1[c] = (T)0;
        }
        if (PRED) {
            gett(G_RB, rb_2);
        } else {
#pragma unroll
            for (int c = 0; c < NC; ++c) rb_2[c] = (T)0;
        }

        // ---- rel(s): rel_from_zeta_and_psi + apply_rel_bc -------------------
        double up1[NC];
        col_up(P2, up1);
        T rel_s[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) rel_s[c] = rel_int(zpb_s[c], P2[c], pm_s[c], pp_s[c]);
        if constexpr (EDGE) {
            // Walls (apply_rel_bc; the corners take the j-wall's formula,
            // which the reference applies last).
            if (s == 0 || s == jj - 1) {
                const long long d = s == 0 ? pitch : -(long long)pitch;
#pragma unroll
                for (int c = 0; c < NC; ++c)
                    if (in_i(c)) {
                        const double* p = p_psi + (long long)s * pitch + c;
                        rel_s[c] = rel_wall(P2[c], p[d], p[2 * d]);
                    }
            } else if (walls) {
                double up2[NC], dn1[NC], dn2[NC];
                col_up2(P2, up2);
                col_dn(P2, dn1);
                col_dn2(P2, dn2);
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    if (ib + c == 0) rel_s[c] = rel_wall(P2[c], dn1[c], dn2[c]);
                    if (ib + c == ii - 1) rel_s[c] = rel_wall(P2[c], up1[c], up2[c]);
                }
            }
#pragma unroll
            for (int c = 0; c < NC; ++c)
                if (!(in_j(s) && in_i(c))) rel_s[c] = 0;
        }

        // ---- zeta at row s-1 after update_zeta_bc and cabaret_forcing -------
        const int s1r = s - 1;
        T rl_up[NC], rl_dn[NC];
        col_up(Rm1, rl_up);
        col_dn(Rm1, rl_dn);
        T zf_1[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const T lap = (T)-4 * Rm1[c] + rl_up[c] + rl_dn[c] + Rm2[c] + rel_s[c];
            T fr, f = dt;  // the forcing is f * fr
            if (L == 1) {
                fr = w_1[c] - vb * Rm1[c] + nu * lap;
            } else if (top) {
                fr = w_1[c] + nu * lap;
            } else if (bottom) {
                fr = -vb * Rm1[c] + nu * lap;
            } else {
                f = dt * nu;
                fr = lap;
            }
            zf_1[c] = add_scaled(zpb_prev[c], f, fr, EDGE && c == 1);
            if (EDGE && !(int_j(s1r) && int_i(c))) {
                if (!(in_j(s1r) && in_i(c)))
                    zf_1[c] = 0;
                else if (L == 1)
                    zf_1[c] = Rm1[c];
                else if (top)
                    zf_1[c] = (T)((double)Rm1[c] - s2 * (P1[c] - pp_prev[c]));
                else if (bottom)
                    zf_1[c] = (T)((double)Rm1[c] - s1 * (P1[c] - pm_prev[c]));
                else
                    zf_1[c] = (T)((double)Rm1[c] - s1 * (P1[c] - pm_prev[c]) - s2 * (P1[c] - pp_prev[c]));
            }
        }

        // ---- corner psi and face velocities ------------------------------------
        // pe_here: corner between nodes (i-1, i) x (s-1, s).
        double left1[NC], pe_here[NC], pe_dn[NC];  // left1: psi row s-1, column i-1
        left1[0] = up1_prev0;
#pragma unroll
        for (int c = 1; c < NC; ++c) left1[c] = P1[c - 1];
#pragma unroll
        for (int c = 0; c < NC; ++c) pe_here[c] = 0.25 * (P2[c] + P1[c] + up1[c] + left1[c]);
        col_dn(pe_here, pe_dn);
        T uj_s[NC], ujm_s[NC], ui_1[NC], uim_1[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            ujm_s[c] = (T)(pe_dn[c] - pe_here[c]);  // face b = s
            uj_s[c] = ((T)1 + tu) * ujm_s[c] - tu * ujmo_s[c];
            uim_1[c] = (T)(-pe_here[c] + pe_prev[c]);  // row s-1, face a = i
            ui_1[c] = ((T)1 + tu) * uim_1[c] - tu * uimo_1[c];
            if (EDGE && !(s >= 1 && s <= jj - 1 && int_i(c))) uj_s[c] = ujm_s[c] = 0;
            if (EDGE && !(int_j(s1r) && fac_i(c))) ui_1[c] = uim_1[c] = 0;
        }

        // ---- extrapolator, j-faces: face b = s-1 -------------------------------
        T fjn[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const T u1 = UJm1[c];
            const bool pos = u1 >= (T)0;
            fjn[c] = extrap(u1, pos ? UJm2[c] : uj_s[c], FJm1[c], pos ? FJm2[c] : fj_s[c], pos ? ZFm2[c] : zf_1[c],
                            pos ? ZOm2[c] : zo_1[c], pos);
            if (EDGE) {
                if (s1r == 1 && pos) fjn[c] = extrap_wall(FJm1[c], ZFm2[c], ZOm2[c]);
                if (s1r == jj - 1 && !pos) fjn[c] = extrap_wall(FJm1[c], zf_1[c], zo_1[c]);
                if (!(s1r >= 1 && s1r <= jj - 1 && int_i(c))) fjn[c] = 0;
            }
        }

        // ---- extrapolator, i-faces on row s-1: face a = i ------------------------
        T fin[NC], flj_1[NC], fli_1[NC];
        if constexpr (NC == 1) {
            // The upwind side only: one shuffle from the lane that holds it.
            const bool pos = ui_1[0] >= (T)0;
            const int sf = pos ? lane - 1 : lane + 1, sn = pos ? lane - 1 : lane;
            const T u2 = __shfl_sync(0xffffffffu, ui_1[0], sf), f2 = __shfl_sync(0xffffffffu, fio_1[0], sf);
            const T zn = __shfl_sync(0xffffffffu, zf_1[0], sn), zo = __shfl_sync(0xffffffffu, zo_1[0], sn);
            fin[0] = extrap(ui_1[0], u2, fio_1[0], f2, zn, zo, pos);
            if (EDGE) {
                if (walls && ((ib == 1 && pos) || (ib == ii - 1 && !pos))) fin[0] = extrap_wall(fio_1[0], zn, zo);
                if (!(int_j(s1r) && fac_i(0))) fin[0] = 0;
            }
        } else {
            T ui_up[NC], ui_dn[NC], fi_up[NC], fi_dn[NC], zf_up[NC], zo_up[NC];
            col_up(ui_1, ui_up);
            col_dn(ui_1, ui_dn);
            col_up(fio_1, fi_up);
            col_dn(fio_1, fi_dn);
            col_up(zf_1, zf_up);
            col_up(zo_1, zo_up);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const T u1 = ui_1[c];
                const bool pos = u1 >= (T)0;
                fin[c] = extrap(u1, pos ? ui_up[c] : ui_dn[c], fio_1[c], pos ? fi_up[c] : fi_dn[c],
                                pos ? zf_up[c] : zf_1[c], pos ? zo_up[c] : zo_1[c], pos);
                if (EDGE) {
                    if (walls && ((ib + c == 1 && pos) || (ib + c == ii - 1 && !pos)))
                        fin[c] = extrap_wall(fio_1[c], pos ? zf_up[c] : zf_1[c], pos ? zo_up[c] : zo_1[c]);
                    if (!(int_j(s1r) && fac_i(c))) fin[c] = 0;
                }
            }
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            flj_1[c] = UJm1[c] * fjn[c];  // flux_j on face s-1
            fli_1[c] = ui_1[c] * fin[c];  // flux_i on row s-1, face i
        }

        // ---- corrector at row o = s-2 -----------------------------------------
        const int o = s - 2;
        T fli_dn[NC], ui_e[NC];  // flux_i and (PRED) ui on face a = i + 1, row o
        col_dn(FLI, fli_dn);
        if (PRED) col_dn(UIm2, ui_e);
        const bool row_o = o >= j0 && in_j(o), row_i = s1r >= j0 && s1r < j0 + SH, row_j = s >= j0 && s < j0 + SH;
        if (row_o) {
            T z[NC], rr[NC], zz[NC], rbn[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                rr[c] = -(fli_dn[c] - FLI[c] + flj_1[c] - FLJm2[c]);
                z[c] = ZFm2[c];
                if (int_j(o) && int_i(c)) z[c] = z[c] + hdt * rr[c];
                if (PRED) {
                    // Next step: cabaret_predictor (qg3p_aux.F90:1012-1018) and
                    // cabaret_beta (:1051-1059) with this step's ui.
                    zz[c] = z[c] + hdt * rr[c];
                    rbn[c] = dt * ((T)0.5 * (ui_e[c] + UIm2[c]) * beta_l);
                    zz[c] = zz[c] + ((T)1 + ta) * rbn[c] - ta * rb_2[c];
                }
            }
            const long long ro = (long long)o * pitch;
            if (out_lane && !EDGE) {
                vst<NC>(p_res + ro, rr);
                if (PRED) {
                    vst<NC>(p_rbn + ro, rbn);
                    vst<NC>(p_zpn + ro, zz);
                }
                vst<NC>(p_zn + ro, z);
            }
            if (out_lane && EDGE) {
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    if (!in_i(c)) continue;
                    if (int_j(o) && int_i(c)) {
                        p_res[ro + c] = rr[c];
                        if (PRED) {
                            p_rbn[ro + c] = rbn[c];
                            p_zpn[ro + c] = zz[c];
                        }
                    }
                    p_zn[ro + c] = z[c];
                }
            }
            if (avg && out_lane) {
#pragma unroll
                for (int c = 0; c < NC; ++c)
                    if (in_i(c)) p_av[ro + c] += dt64 * p_psi[ro + c];
            }
        }
        // ---- owned face writes ---------------------------------------------------
        if (out_lane) {
            const long long ri = (long long)s1r * pitch;
            if (!EDGE) {
                if (row_i) {
                    vst<NC>(p_ui + ri, ui_1);
                    vst<NC>(p_uimon + ri, uim_1);
                    vst<NC>(p_fin + ri, fin);
                    vst<NC>(p_fjn + ri, fjn);
                }
                if (row_j) {
                    vst<NC>(p_uj + ri + pitch, uj_s);
                    vst<NC>(p_ujmon + ri + pitch, ujm_s);
                }
            } else {
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    if (row_i && int_j(s1r) && fac_i(c)) {
                        p_ui[ri + c] = ui_1[c];
                        p_uimon[ri + c] = uim_1[c];
                        p_fin[ri + c] = fin[c];
                    }
                    if (row_i && s1r >= 1 && s1r <= jj - 1 && int_i(c)) p_fjn[ri + c] = fjn[c];
                    if (row_j && s >= 1 && s <= jj - 1 && int_i(c)) {
                        p_uj[ri + pitch + c] = uj_s[c];
                        p_ujmon[ri + pitch + c] = ujm_s[c];
                    }
                }
            }
            // (EDGE: faces outside the domain are zero)
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                if (row_i) umax = fmax(umax, fabs(ui_1[c]));
                if (row_j) umax = fmax(umax, fabs(uj_s[c]));
            }
        }
        // ---- shift the windows ---------------------------------------------------
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            Rm2[c] = Rm1[c];
            Rm1[c] = rel_s[c];
            ZFm2[c] = zf_1[c];
            ZOm2[c] = zo_1[c];
            UJm2[c] = UJm1[c];
            UJm1[c] = uj_s[c];
            FJm2[c] = FJm1[c];
            FJm1[c] = fj_s[c];
            FLJm2[c] = flj_1[c];
            FLI[c] = fli_1[c];
            UIm2[c] = ui_1[c];
            zpb_prev[c] = zpb_s[c];
            pe_prev[c] = pe_here[c];
            if (EDGE) {
                pm_prev[c] = pm_s[c];
                pp_prev[c] = pp_s[c];
            }
        }
        up1_prev0 = up1[0];
    }
    return (double)umax;
}

template <typename T, int NC>
__host__ __device__ constexpr int cab_ring_bytes() {  // of a warp
    return (CabRing<T, NC>::bytes() + 127) / 128 * 128;
}

// End of a member's step, by the thread that counted last: the CFL number,
// model time, and when adaptive stepping is on dt and the time
// weights for the next step (cabaret_cfl / cabaret_adapt_dt,
// qg3p_aux.F90:920-990).
__device__ __forceinline__ void finish_step(const Member& Mb) {
    // max |u|, taken out for the next step
    const double mu = __longlong_as_double((long long)atomicExch(Mb.maxu, 0ull));
    Scalars* sc = Mb.sc;
    if (cab_average_gate(Mb)) sc->diag_time += sc->dt;
    sc->max_u = mu;
    sc->cfl = mu * sc->dt;
    sc->dt_last = sc->dt;
    sc->tweight_a_last = sc->tweight_a;
    sc->tweight_u_last = sc->tweight_u;
    sc->model_time += sc->dt;
    if (Mb.adapt_dt) {
        const double old_dt = sc->dt;
        double ndt = old_dt;
        const double tol = 10.0 * fmax(fabs(mu) * 2.220446049250313e-16, 2.220446049250313e-16);
        if (fabs(mu) > tol) {
            ndt = Mb.target_cfl / mu;
            ndt = fmin(fmin(ndt, old_dt * Mb.max_dt_increase), Mb.max_dt);
        }
        sc->dt = ndt;
        sc->tweight_a = 0.5 * ndt / old_dt;
        sc->tweight_u = ndt / (old_dt + ndt);
        if (ndt < 1.0e-6) atomicOr(Mb.status, (int)ST_SMALL_DT);
    }
    Mb.counters[1] = 0u;
    Mb.counters[3] = 0u;  // the sweep queue of k_cabaret_fused
}
// One thread per unit of work (a warp or a CTA, `units` of them per member)
// reports its largest |u|: an integer maximum on the bits of the non-negative
// value, so the result does not depend on the order.  True for the last one.
// (Partial maxima per CTA, reduced by the last CTA, left the GPU idle for
// 4 us at the end of every step at 1025 nodes.)
__device__ __forceinline__ bool count_done(const Member& Mb, double umax, unsigned units) {
    if (umax > 0.0) atomicMax(Mb.maxu, (unsigned long long)__double_as_longlong(umax));
    __threadfence();
    return atomicAdd(&Mb.counters[1], 1u) == units - 1u;
}

// Three CTAs per SM (at most 168 registers) with one column per lane:
// measured 16 % faster than the unconstrained allocation (two CTAs) at
// 1025 x 1025 x 3 FP64, 15 % at 2049 x 2049 x 5; four CTAs spill heavily
// and are slower.  Two columns per lane: two CTAs per SM, no spills.
//
// Persistent: a member's CTAs (at most the resident ones, cabaret_ctas) share
// its (layer, strip, band) sweeps through a counter (counters[3]); each warp
// claims the next sweep when it finishes one, so warps run until the queue is
// empty instead of idling in partly filled CTAs and waves.  The sweeps at a
// wall (slower) are claimed first, so the last sweeps claimed are interior
// ones.  The last warp of a member resets the counter (finish_step).
template <bool PRED, typename T, int NC, bool ONE>
__global__ void __launch_bounds__(CAB_WARPS * 32, NC == 2 ? 2 : 3)
    k_cabaret_fused(const Member* __restrict__ mems, const int* __restrict__ prefix, int nmem,
                    const __grid_constant__ Member one, int use_one) {
    __shared__ Member Mb_s;
    extern __shared__ __align__(128) char cab_smem[];  // [CAB_WARPS][cab_ring_bytes<T, NC>()]
    pdl_wait();
    int local = blockIdx.x;
    if constexpr (!ONE) {
        cta_member(Mb_s, one, use_one, mems, prefix, nmem, blockIdx.x, &local);
        __syncthreads();
    }
    const Member& Mb = member_ref<ONE>(Mb_s, one);
    const int ii = Mb.ii, jj = Mb.jj, L = Mb.L;
    const int SH = Mb.cab_sh;
    constexpr int SW = cab_sw(NC);
    const int nstrips = (ii + SW - 1) / SW, nbands = (jj + SH - 1) / SH;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ntasks = nstrips * nbands * L;
    // Interior sweeps: footprint columns i0-2 .. i0+32NC-3, rows j0-4 ..
    // j0+SH+3 at least two nodes inside the domain -- strips sA .. sA+nsi-1
    // of bands bA .. bA+nbi-1; the nedge others (per layer) are claimed first.
    const int sA = (4 + SW - 1) / SW, bA = (6 + SH - 1) / SH;
    const int nsi = max(0, (ii - 32 * NC) / SW - sA + 1) * (ii >= 32 * NC), nbi = max(0, (jj - 6 - SH) / SH - bA + 1) * (jj >= 6 + SH);
    const int nedge = nsi * nbi ? nstrips * nbands - nsi * nbi : nstrips * nbands;
    char* ring = cab_smem + warp * cab_ring_bytes<T, NC>();
    double umax = 0.0;
    for (;;) {
        int task = 0;
        if (lane == 0) task = (int)atomicAdd(&Mb.counters[3], 1u);
        task = __shfl_sync(0xffffffffu, task, 0);
        if (task >= ntasks) break;
        const int l = task % L;
        int sb = task / L, strip, band;
        const bool interior = sb >= nedge;
        if (interior) {
            sb -= nedge;
            strip = sA + sb % nsi;
            band = bA + sb / nsi;
        } else if (sb < (nbands - nbi) * nstrips) {  // bands at the j-walls
            const int q = sb / nstrips;
            strip = sb - q * nstrips;
            band = q < bA ? q : q + nbi;
        } else {  // strips at the i-walls
            sb -= (nbands - nbi) * nstrips;
            const int q = sb / nbi;
            strip = q < sA ? q : q + nsi;
            band = bA + sb - q * nbi;
        }
        const int i0 = strip * SW, j0 = band * SH;
        const double u = interior ? cab_sweep<false, PRED, T, NC>(Mb, l, i0, j0, SH, lane, ring)
                                  : cab_sweep<true, PRED, T, NC>(Mb, l, i0, j0, min(SH, jj - j0), lane, ring);
        umax = fmax(umax, u);
        __syncwarp();  // the ring's last reads before the next sweep's copies
    }
    pdl_release();

    // Max |u| of the new face velocities (cabaret_cfl / cabaret_adapt_dt);
    // the last warp of the member finishes the step.
    umax = warp_max(umax);
    if (lane == 0 && count_done(Mb, umax, (unsigned)(CAB_WARPS * Mb.ntiles_cab))) finish_step(Mb);
}

// ---------------------------------------------------------------------------
// Tile formulation of the same fused step: one CTA (8 warps) per (layer,
// CT_X x CT_Y tile of output nodes).  Every stage is computed once per node
// or face of the tile's footprint into shared memory, stages separated by
// block barriers; lane = column, warps stride over rows.  All footprint
// arrays share one 32-column frame whose column 0 is node i0-2 and row 0 is
// node j0-2 (a face a sits in the column of node a, a corner between columns
// c-1 and c in column c).  For outputs i in [i0, i0+CT_X), j in [j0, j0+CT_Y):
//   psi (3 layers), zeta, rel   nodes [i0-2, i0+CT_X+1] x [j0-2, j0+CT_Y+1]
//   corner psi                  columns [i0-1, i0+CT_X+1], rows [j0-1, j0+CT_Y+1]
//   zeta after forcing, zeta_old   nodes [i0-1, i0+CT_X] x [j0-1, j0+CT_Y]
//   ui, zeta_fi (old)           faces a in [i0-1, i0+CT_X+1], rows [j0, j0+CT_Y)
//   uj, zeta_fj (old)           faces b in [j0-1, j0+CT_Y+1], columns [i0, i0+CT_X)
//   flux_i / flux_j             faces a in [i0, i0+CT_X] / b in [j0, j0+CT_Y]
// Each output node owns face a = i (ui, uimo, zeta_fi) and face b = j (uj,
// ujmo, zeta_fj), as in the sweep.  EDGE = false: the whole footprint is at
// least one node inside the domain, so no bounds checks or boundary branches.
constexpr int CT_X = 28, CT_Y = 16, CT_THREADS = 256, CT_W = 32, CT_H = CT_Y + 4;
constexpr int CT_N = CT_W * CT_H;  // entries of one frame array

template <typename T>
struct TileSmem {
    // doubles: psi, psi above, psi below, corner psi; T: zeta, rel, zf, zo,
    // ui, fio, uj, fj.  The fluxes reuse the psi-above / psi-below space.
    static constexpr size_t bytes() { return 4 * CT_N * sizeof(double) + 8 * CT_N * sizeof(T); }
};

// rows handled by a warp in a frame row range of length h: ceil(h / 8)
__host__ __device__ constexpr int ct_rows(int h) { return (h + 7) / 8; }

template <bool PRED, bool EDGE, typename T>
// FP64: the CTA's CFL partial and its count towards the last-CTA step finish
// are issued right after the face velocities (stage 3), so that the
// counter's round trip overlaps the extrapolation and the corrector (+1 % per
// step at 513^2 x 3, +2.6 % at 257^2); every scalar the later stages need is
// read before (the last CTA may advance them once every CTA has counted).
// FP32 (64-80 registers, where the extra live values cost more: -5 % at 513^2)
// counts at the end.
__device__ __forceinline__ void cab_tile(const Member& Mb, int l, int i0, int j0, char* smem, double* red) {
    const int ii = Mb.ii, jj = Mb.jj, L = Mb.L, pitch = Mb.pitch;
    const long long ls = Mb.lstride;
    const int cur = Mb.cur, nxt = cur ^ 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const T dt = (T)Mb.sc->dt, tu = (T)Mb.sc->tweight_u, ta = (T)Mb.sc->tweight_a;
    constexpr bool EARLY = sizeof(T) == 8;
    const bool avg_early = EARLY && cab_average_gate(Mb);
    const double dt64_early = EARLY ? Mb.sc->dt : 0.0;
    const T hdt = (T)0.5 * dt;
    const double s1 = Mb.s1[l], s2 = Mb.s2[l];
    const int bc = Mb.bc_type;
    const double cffbc = Mb.alpha / (Mb.alpha + 3.0);
    const bool lim = Mb.limiter != 0;
    const bool top = (l == 0), bottom = (l == L - 1);
    const T nu = (T)Mb.viscosity, vb = (T)Mb.visc_bot, beta_l = (T)Mb.beta[l];
    const long long lo = l * ls;
    // This lane's column: node i0 - 2 + lane; the row of frame row r is j0 - 2 + r.
    const int ic = i0 - 2 + lane;
    const long long gcol = lo + ic;
    auto grow = [&](int r) { return (long long)(j0 - 2 + r) * pitch; };
    const bool col_in = !EDGE || (ic >= 0 && ic < ii);
    const bool col_int = !EDGE || (ic > 0 && ic < ii - 1);
    auto row_in = [&](int r) { return !EDGE || (j0 - 2 + r >= 0 && j0 - 2 + r < jj); };
    auto row_int = [&](int r) { return !EDGE || (j0 - 2 + r > 0 && j0 - 2 + r < jj - 1); };
    const bool ui_col = !EDGE || (ic >= 1 && ic <= ii - 1);   // face a = ic can exist
    const bool uj_col = !EDGE || (ic >= 1 && ic <= ii - 2);   // column ic can carry j-faces
    auto ui_row = [&](int r) { return !EDGE || (j0 - 2 + r >= 1 && j0 - 2 + r <= jj - 2); };
    auto uj_row = [&](int r) { return !EDGE || (j0 - 2 + r >= 1 && j0 - 2 + r <= jj - 1); };

    double* sPsi = reinterpret_cast<double*>(smem);
    double* sPm = sPsi + CT_N;
    double* sPp = sPm + CT_N;
    double* sPe = sPp + CT_N;
    T* sZpb = reinterpret_cast<T*>(sPe + CT_N);
    T* sRel = sZpb + CT_N;
    T* sZf = sRel + CT_N;
    T* sZo = sZf + CT_N;
    T* sUi = sZo + CT_N;
    T* sFio = sUi + CT_N;
    T* sUj = sFio + CT_N;
    T* sFj = sUj + CT_N;
    T* sFli = reinterpret_cast<T*>(sPm);  // after the face velocities
    T* sFlj = sFli + CT_N;
    auto X = [&](int r, int c) { return r * CT_W + c; };  // frame index

    // Limited upwind extrapolation (cabaret_extrapolator, interior branch).
    auto extrap = [&](T u1, T u2, T fi1, T fi2, T psi_n, T psi_o, bool pos) -> T {
        const T v0 = (u1 + u2) / (T)2;
        const T d_f = pos ? -(psi_n - psi_o) * (T)2 - dt * v0 * (fi1 - fi2)
                          : -(psi_n - psi_o) * (T)2 - dt * v0 * (fi2 - fi1);
        T v = (T)2 * psi_n - fi2;
        if (lim) {
            const T fmx = fmax(fmax(fi1, fi2), psi_n) - d_f;
            const T fmn = fmin(fmin(fi1, fi2), psi_n) - d_f;
            if (v > fmx) v = fmx;
            if (v < fmn) v = fmn;
        }
        return v;
    };
    // The wall branch: upwind node on the boundary.
    auto extrap_wall = [&](T fi1, T psi_n, T psi_o) -> T {
        const T fi2 = psi_n;
        const T d_f = -(psi_n - psi_o);
        T v = (T)2 * psi_n - fi2;
        if (lim) {
            const T fmx = fmax(fmax(fi1, fi2), psi_n) - d_f;
            const T fmn = fmin(fmin(fi1, fi2), psi_n) - d_f;
            if (v > fmx) v = fmx;
            if (v < fmn) v = fmn;
        }
        return v;
    };

    const T* zpb = reinterpret_cast<const T*>(Mb.zeta);
    const double* wind = (top && Mb.wind) ? Mb.wind : nullptr;
    // ---- loads used by later stages, issued first (held in registers) -----
    // frame rows: zf 1..CT_Y+2, ui rows 2..CT_Y+1, uj rows 1..CT_Y+3, outputs 2..CT_Y+1
    constexpr int NZ = ct_rows(CT_Y + 2), NU = ct_rows(CT_Y), NV = ct_rows(CT_Y + 3);
    T rWind[NZ], rUimo[NU], rUjmo[NV], rRb[NU];
    {
        const T* uimo = reinterpret_cast<const T*>(Mb.uimo[cur]);
        const T* ujmo = reinterpret_cast<const T*>(Mb.ujmo[cur]);
        const T* rb = reinterpret_cast<const T*>(Mb.res_beta);
#pragma unroll
        for (int k = 0; k < NZ; ++k) {
            const int r = 1 + warp + 8 * k;
            rWind[k] = (wind && r < CT_Y + 3 && lane >= 1 && lane <= CT_X + 2 && col_int && row_int(r))
                           ? (T)wind[grow(r) + ic]
                           : (T)0;
        }
#pragma unroll
        for (int k = 0; k < NU; ++k) {
            const int r = 2 + warp + 8 * k;
            const bool ok = r < CT_Y + 2;
            rUimo[k] = (ok && lane >= 1 && lane <= CT_X + 3 && ui_col && ui_row(r)) ? uimo[grow(r) + gcol] : (T)0;
            rRb[k] = (PRED && ok && lane >= 2 && lane < CT_X + 2 && col_int && row_int(r)) ? rb[grow(r) + gcol] : (T)0;
        }
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const int r = 1 + warp + 8 * k;
            rUjmo[k] = (r < CT_Y + 4 && lane >= 2 && lane < CT_X + 2 && uj_col && uj_row(r)) ? ujmo[grow(r) + gcol]
                                                                                             : (T)0;
        }
    }

    // ---- stage 1: psi (three layers), zeta, zeta_old, old face values ------
    {
        constexpr int NP = ct_rows(CT_H);
        const double* psi = Mb.psi;
        const long long om = (l > 0) ? -ls : 0, op = (l < L - 1) ? ls : 0;
        const T* zold = reinterpret_cast<const T*>(Mb.zeta_old[cur]);
        const T* fio = reinterpret_cast<const T*>(Mb.zfi[cur]);
        const T* fjo = reinterpret_cast<const T*>(Mb.zfj[cur]);
        double vP[NP], vM[NP], vQ[NP];
        T vZ[NP], vO[NZ], vF[NU], vG[NV];
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            const int r = warp + 8 * k;
            const bool ok = r < CT_H && col_in && row_in(r);
            const long long o = grow(r) + gcol;
            vP[k] = ok ? psi[o] : 0.0;
            vM[k] = (ok && L > 1) ? psi[o + om] : 0.0;
            vQ[k] = (ok && L > 1) ? psi[o + op] : 0.0;
            vZ[k] = (ok && col_int && row_int(r)) ? zpb[o] : (T)0;
        }
#pragma unroll
        for (int k = 0; k < NZ; ++k) {
            const int r = 1 + warp + 8 * k;
            vO[k] = (r < CT_Y + 3 && lane >= 1 && lane <= CT_X + 2 && col_in && row_in(r)) ? zold[grow(r) + gcol]
                                                                                           : (T)0;
        }
#pragma unroll
        for (int k = 0; k < NU; ++k) {
            const int r = 2 + warp + 8 * k;
            vF[k] = (r < CT_Y + 2 && lane >= 1 && lane <= CT_X + 3 && ui_col && ui_row(r)) ? fio[grow(r) + gcol]
                                                                                          : (T)0;
        }
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const int r = 1 + warp + 8 * k;
            vG[k] = (r < CT_Y + 4 && lane >= 2 && lane < CT_X + 2 && uj_col && uj_row(r)) ? fjo[grow(r) + gcol]
                                                                                          : (T)0;
        }
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            const int r = warp + 8 * k;
            if (r < CT_H) {
                sPsi[X(r, lane)] = vP[k];
                sPm[X(r, lane)] = vM[k];
                sPp[X(r, lane)] = vQ[k];
                sZpb[X(r, lane)] = vZ[k];
            }
        }
#pragma unroll
        for (int k = 0; k < NZ; ++k) {
            const int r = 1 + warp + 8 * k;
            if (r < CT_Y + 3) sZo[X(r, lane)] = vO[k];
        }
#pragma unroll
        for (int k = 0; k < NU; ++k) {
            const int r = 2 + warp + 8 * k;
            if (r < CT_Y + 2) sFio[X(r, lane)] = vF[k];
        }
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const int r = 1 + warp + 8 * k;
            if (r < CT_Y + 4) sFj[X(r, lane)] = vG[k];
        }
    }
    __syncthreads();

    // ---- stage 2: rel (rel_from_zeta_and_psi + apply_rel_bc), corner psi ---
#pragma unroll
    for (int k = 0; k < ct_rows(CT_H); ++k) {
        const int r = warp + 8 * k;
        if (r >= CT_H) break;
        const int q = X(r, lane);
        T rel = (T)0;
        if (col_in && row_in(r)) {
            const int j = j0 - 2 + r;
            const double p = sPsi[q];
            const bool bj = EDGE && (j == 0 || j == jj - 1), bi = EDGE && (ic == 0 || ic == ii - 1);
            if (bj || bi) {
                // Corners take the j-boundary formula, which the reference applies last.
                if (bc != 3) {
                    double q1, q2;
                    if (bj) {
                        const int d = (j == 0) ? CT_W : -CT_W;
                        q1 = sPsi[q + d];
                        q2 = sPsi[q + 2 * d];
                    } else {
                        const int d = (ic == 0) ? 1 : -1;
                        q1 = sPsi[q + d];
                        q2 = sPsi[q + 2 * d];
                    }
                    rel = (T)((bc == 1) ? cffbc * (-3.5 * p + 4.0 * q1 - 0.5 * q2) : 2.0 * (q1 - p));
                }
            } else {
                const T z = sZpb[q];
                if (L == 1)
                    rel = z;
                else if (top)
                    rel = (T)((double)z + s2 * (p - sPp[q]));
                else if (bottom)
                    rel = (T)((double)z + s1 * (p - sPm[q]));
                else
                    rel = (T)((double)z + s1 * (p - sPm[q]) + s2 * (p - sPp[q]));
            }
        }
        sRel[q] = rel;
    }
#pragma unroll
    for (int k = 0; k < ct_rows(CT_Y + 3); ++k) {
        const int r = 1 + warp + 8 * k;  // corner between rows r-1 and r
        if (r >= CT_H) break;
        if (lane >= 1) {
            const int q = X(r, lane);     // corner between columns lane-1 and lane
            sPe[q] = 0.25 * (sPsi[q] + sPsi[q - CT_W] + sPsi[q - 1] + sPsi[q - CT_W - 1]);
        }
    }
    __syncthreads();

    // ---- stage 3: zeta after update_zeta_bc + forcing; face velocities -----
    double umax = 0.0;
#pragma unroll
    for (int k = 0; k < NZ; ++k) {
        const int r = 1 + warp + 8 * k;
        if (r >= CT_Y + 3) break;
        if (lane < 1 || lane > CT_X + 2) continue;
        const int q = X(r, lane);
        T zf = (T)0;
        if (col_in && row_in(r)) {
            const T R = sRel[q];
            if (EDGE && !(col_int && row_int(r))) {
                const double p = sPsi[q];
                if (L == 1)
                    zf = R;
                else if (top)
                    zf = (T)((double)R - s2 * (p - sPp[q]));
                else if (bottom)
                    zf = (T)((double)R - s1 * (p - sPm[q]));
                else
                    zf = (T)((double)R - s1 * (p - sPm[q]) - s2 * (p - sPp[q]));
            } else {
                const T lap = (T)-4 * R + sRel[q - 1] + sRel[q + 1] + sRel[q - CT_W] + sRel[q + CT_W];
                const T w = rWind[k];
                T rv;
                if (L == 1)
                    rv = dt * (w - vb * R + nu * lap);
                else if (top)
                    rv = dt * (w + nu * lap);
                else if (bottom)
                    rv = dt * (-vb * R + nu * lap);
                else
                    rv = dt * nu * lap;
                zf = sZpb[q] + rv;
            }
        }
        sZf[q] = zf;
    }
    T* ui_g = reinterpret_cast<T*>(Mb.ui);
    T* uimo_n = reinterpret_cast<T*>(Mb.uimo[nxt]);
    T* uj_g = reinterpret_cast<T*>(Mb.uj);
    T* ujmo_n = reinterpret_cast<T*>(Mb.ujmo[nxt]);
    const bool own_col = lane >= 2 && lane < CT_X + 2;  // columns of the tile's outputs
#pragma unroll
    for (int k = 0; k < NU; ++k) {
        const int r = 2 + warp + 8 * k;  // face a = ic on row r
        if (r >= CT_Y + 2) break;
        if (lane < 1 || lane > CT_X + 3) continue;
        const int q = X(r, lane);
        T u = (T)0;
        if (ui_col && ui_row(r)) {
            // corners (a, rows r-1|r) and (a, rows r|r+1)
            const T um = (T)(sPe[q] - sPe[q + CT_W]);
            u = ((T)1 + tu) * um - tu * rUimo[k];
            if (own_col) {
                const long long o = grow(r) + gcol;
                ui_g[o] = u;
                uimo_n[o] = um;
                umax = fmax(umax, (double)fabs(u));
            }
        }
        sUi[q] = u;
    }
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int r = 1 + warp + 8 * k;  // face b = row r, column ic
        if (r >= CT_Y + 4) break;
        if (!own_col) continue;
        const int q = X(r, lane);
        T u = (T)0;
        if (uj_col && uj_row(r)) {
            // corners (columns ic|ic+1, rows r-1|r) and (ic-1|ic, r-1|r)
            const T um = (T)(sPe[q + 1] - sPe[q]);
            u = ((T)1 + tu) * um - tu * rUjmo[k];
            if (r >= 2 && r < CT_Y + 2) {
                const long long o = grow(r) + gcol;
                uj_g[o] = u;
                ujmo_n[o] = um;
                umax = fmax(umax, (double)fabs(u));
            }
        }
        sUj[q] = u;
    }
    bool last = false;
    auto count = [&]() {
        umax = warp_max(umax);
        if (lane == 0) red[warp] = umax;
        __syncthreads();
        if (threadIdx.x == 0) {
            double m = 0.0;
            for (int w = 0; w < CT_THREADS / 32; ++w) m = fmax(m, red[w]);
            last = count_done(Mb, m, (unsigned)Mb.ntiles_cab);
        }
    };
    if constexpr (EARLY)
        count();
    else
        __syncthreads();

    // ---- stage 4: extrapolated face values (cabaret_extrapolator) and fluxes
    T* fin_g = reinterpret_cast<T*>(Mb.zfi[nxt]);
    T* fjn_g = reinterpret_cast<T*>(Mb.zfj[nxt]);
#pragma unroll
    for (int k = 0; k < NU; ++k) {
        const int r = 2 + warp + 8 * k;  // face a = ic on row r, a in [i0, i0+CT_X]
        if (r >= CT_Y + 2) break;
        if (lane < 2 || lane > CT_X + 2) continue;
        const int q = X(r, lane);
        T flux = (T)0;
        if (ui_col && ui_row(r)) {
            const T u1 = sUi[q];
            T f;
            if (u1 >= (T)0)
                f = (!EDGE || ic > 1) ? extrap(u1, sUi[q - 1], sFio[q], sFio[q - 1], sZf[q - 1], sZo[q - 1], true)
                                      : extrap_wall(sFio[q], sZf[q - 1], sZo[q - 1]);
            else
                f = (!EDGE || ic < ii - 1) ? extrap(u1, sUi[q + 1], sFio[q], sFio[q + 1], sZf[q], sZo[q], false)
                                           : extrap_wall(sFio[q], sZf[q], sZo[q]);
            if (own_col) fin_g[grow(r) + gcol] = f;
            flux = u1 * f;
        }
        sFli[q] = flux;
    }
#pragma unroll
    for (int k = 0; k < ct_rows(CT_Y + 1); ++k) {
        const int r = 2 + warp + 8 * k;  // face b = row r in [j0, j0+CT_Y], column ic
        if (r >= CT_Y + 3) break;
        if (!own_col) continue;
        const int q = X(r, lane);
        const int b = j0 - 2 + r;
        T flux = (T)0;
        if (uj_col && uj_row(r)) {
            const T u1 = sUj[q];
            T f;
            if (u1 >= (T)0)
                f = (!EDGE || b > 1)
                        ? extrap(u1, sUj[q - CT_W], sFj[q], sFj[q - CT_W], sZf[q - CT_W], sZo[q - CT_W], true)
                        : extrap_wall(sFj[q], sZf[q - CT_W], sZo[q - CT_W]);
            else
                f = (!EDGE || b < jj - 1) ? extrap(u1, sUj[q + CT_W], sFj[q], sFj[q + CT_W], sZf[q], sZo[q], false)
                                          : extrap_wall(sFj[q], sZf[q], sZo[q]);
            if (r < CT_Y + 2) fjn_g[grow(r) + gcol] = f;
            flux = u1 * f;
        }
        sFlj[q] = flux;
    }
    __syncthreads();

    // ---- stage 5: cabaret_corrector (+ the next step's predictor and beta) --
    T* res_g = reinterpret_cast<T*>(Mb.res_out);
    T* zn_g = reinterpret_cast<T*>(Mb.zeta_old[nxt]);
    T* rbn_g = reinterpret_cast<T*>(Mb.res_beta_other);
    T* zpn_g = reinterpret_cast<T*>(Mb.zeta_next);
    const bool avg = EARLY ? avg_early : cab_average_gate(Mb);
    const double dt64 = EARLY ? dt64_early : Mb.sc->dt;
#pragma unroll
    for (int k = 0; k < NU; ++k) {
        const int r = 2 + warp + 8 * k;
        if (r >= CT_Y + 2) break;
        if (!own_col || !(col_in && row_in(r))) continue;
        const int q = X(r, lane);
        const long long o = grow(r) + gcol;
        if (avg) Mb.psi_av[o] += dt64 * sPsi[q];
        T z = sZf[q];
        if (col_int && row_int(r)) {
            const T rr = -(sFli[q + 1] - sFli[q] + sFlj[q + CT_W] - sFlj[q]);
            res_g[o] = rr;
            z = z + hdt * rr;
            if (PRED) {
                // cabaret_predictor (qg3p_aux.F90:1012-1018) and cabaret_beta
                // (:1051-1059) of the next step with this step's ui.
                T zz = z + hdt * rr;
                const T rbn = dt * ((T)0.5 * (sUi[q + 1] + sUi[q]) * beta_l);
                zz = zz + ((T)1 + ta) * rbn - ta * rRb[k];
                rbn_g[o] = rbn;
                zpn_g[o] = zz;
            }
        }
        zn_g[o] = z;
    }
    if constexpr (!EARLY) count();
    if (last) finish_step(Mb);
}

// MINB: CTAs per SM the register allocation must allow.  Three (80
// registers): the FP32 form always, FP64 on grids of many waves, where the
// extra resident CTA hides more latency than the tighter allocation costs
// (measured -8 % at 513 x 513 x 3); one for short FP64 grids.
template <bool PRED, typename T, int MINB>
__global__ void __launch_bounds__(CT_THREADS, MINB) k_cabaret_tile(const Member* __restrict__ mems,
                                                              const int* __restrict__ prefix, int nmem,
                                                              const __grid_constant__ Member one, int use_one) {
    __shared__ Member Mb;
    __shared__ double red[CT_THREADS / 32];
    extern __shared__ __align__(16) char tsm[];
    pdl_wait();
    int local;
    cta_member(Mb, one, use_one, mems, prefix, nmem, blockIdx.x, &local);
    __syncthreads();
    const int ii = Mb.ii, jj = Mb.jj, L = Mb.L;
    const int tx = (ii + CT_X - 1) / CT_X;
    const int l = local % L;
    const int tile = local / L;
    const int i0 = (tile % tx) * CT_X, j0 = (tile / tx) * CT_Y;
    // Interior tiles: footprint [i0-2, i0+CT_X+1] x [j0-2, j0+CT_Y+1] inside
    // the interior nodes.
    const bool inner = i0 - 2 >= 1 && i0 + CT_X + 1 <= ii - 2 && j0 - 2 >= 1 && j0 + CT_Y + 1 <= jj - 2;
    if (inner)
        cab_tile<PRED, false, T>(Mb, l, i0, j0, tsm, red);
    else
        cab_tile<PRED, true, T>(Mb, l, i0, j0, tsm, red);
    pdl_release();
}

// CTAs of k_cabaret_fused resident on the current device at once (at least 1).
template <typename T, int NC>
static int cabaret_resident_t() {
    const size_t bytes = (size_t)CAB_WARPS * cab_ring_bytes<T, NC>();
    int dev = 0, sms = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaFuncSetAttribute(k_cabaret_fused<true, T, NC, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_cabaret_fused<true, T, NC, true>, CAB_WARPS * 32, bytes) !=
            cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    return std::max(1, per * sms);
}

static int cabaret_resident(int nc, bool f32) {
    return !f32 ? cabaret_resident_t<double, 1>() : nc == 2 ? cabaret_resident_t<float, 2>() : cabaret_resident_t<float, 1>();
}

// Band height: the one whose greedy schedule ends first.  A sweep of SH rows
// costs SH + 4 iterations and about one more to start; one at a wall costs
// up to 1.5 times an interior one (measured, 513 and 1025 nodes) and is claimed
// earlier.  With W resident warps, floor(nE / W) or one more edge sweep each,
// the interior sweeps then fill whole rounds: the end is the first time at
// which every round begun so far holds them all.  At most 40 rows: taller
// bands measured slower at 2049^2 x 5 (86 rows 661 us, 29 rows 601), where
// the L2 cache no longer holds a row from one band to the next.
int cabaret_band(int ii, int jj, int L, bool f32) {
    const long long W = (long long)CAB_WARPS * cabaret_resident(1, f32);
    const int sw = cab_sw(1), ns = (ii + sw - 1) / sw;
    double best = 1e300;
    int band = 4;
    for (int sh = 4; sh <= 40; ++sh) {
        const int nb = (jj + sh - 1) / sh;
        const int nsi = ii < 32 ? 0 : std::max(0, (ii - 32) / sw - (4 + sw - 1) / sw + 1);
        const int nbi = jj < 6 + sh ? 0 : std::max(0, (jj - 6 - sh) / sh - (6 + sh - 1) / sh + 1);
        const long long nI = (long long)nsi * nbi * L, nE = (long long)ns * nb * L - nI;
        const double c = sh + 5, e = 1.5 * c;
        const double a0 = e * (double)(nE / W), a1 = a0 + e;  // W - g1 warps are free at a0, g1 at a1
        const long long g1 = nE % W, g0 = W - g1;
        double t = g1 ? a1 : a0;
        if (nI > 0) {
            for (long long k0 = 0, k1 = 0; g0 * k0 + g1 * k1 < nI;) {
                if (a0 + c * (double)(k0 + 1) <= a1 + c * (double)(k1 + 1))
                    t = std::max(t, a0 + c * (double)++k0);
                else
                    t = std::max(t, a1 + c * (double)++k1);
            }
        }
        if (t <= best) {
            best = t;
            band = sh;
        }
    }
    return band;
}

int cabaret_ctas(int ii, int jj, int L, int sh, int nc, bool f32) {
    const int sw = cab_sw(nc);
    const int nstrips = (ii + sw - 1) / sw, nbands = (jj + sh - 1) / sh;
    const int need = (nstrips * nbands * L + CAB_WARPS - 1) / CAB_WARPS;
    const int resident = cabaret_resident(nc, f32);
    return std::min(need, resident);
}

int cabaret_tile_ctas(int ii, int jj, int L) {
    return ((ii + CT_X - 1) / CT_X) * ((jj + CT_Y - 1) / CT_Y) * L;
}

template <bool PRED, typename T, int NC>
static cudaError_t launch_sweeps(const LaunchSet& ls, cudaStream_t st) {
    const size_t bytes = (size_t)CAB_WARPS * cab_ring_bytes<T, NC>();
    auto kern = member_arg_used(ls) ? k_cabaret_fused<PRED, T, NC, true> : k_cabaret_fused<PRED, T, NC, false>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    return launch_step_kernel(ls.pdl, kern, dim3(ls.ctas_cab), dim3(CAB_WARPS * 32), bytes, st, ls.members,
                              ls.prefix_cab, ls.nmem, member_arg(ls), member_arg_used(ls));
}

template <bool PRED, typename T>
static cudaError_t launch_cab(const LaunchSet& ls, cudaStream_t st) {
    if (ls.cab_kernel == 0) {
        const size_t tb = TileSmem<T>::bytes();
        // CTAs per SM the registers must allow (measured on B200): FP64 three
        // on grids of many waves, else one; FP32 four on grids of more than two
        // CTAs per SM (40 KB of shared memory each: +2.9 % per step at
        // 513^2 x 3, +5.1 % at 257^2; -4.8 % on 129^2's 135 CTAs), else three.
        void (*kern)(const Member*, const int*, int, Member, int);
        if constexpr (sizeof(T) == 4)
            kern = ls.ctas_cab > 2 * ls.sm_count ? k_cabaret_tile<PRED, T, 4> : k_cabaret_tile<PRED, T, 3>;
        else
            kern = ls.ctas_cab > 4 * ls.sm_count ? k_cabaret_tile<PRED, T, 3> : k_cabaret_tile<PRED, T, 1>;
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tb);
        if (e != cudaSuccess) return e;
        return launch_step_kernel(ls.pdl, kern, dim3(ls.ctas_cab), dim3(CT_THREADS), tb, st, ls.members,
                                  ls.prefix_cab, ls.nmem, member_arg(ls), member_arg_used(ls));
    }
    if constexpr (sizeof(T) == 4) {
        if (ls.cab_kernel == 2) return launch_sweeps<PRED, T, 2>(ls, st);
    }
    return launch_sweeps<PRED, T, 1>(ls, st);
}


// ---------------------------------------------------------------------------
// The channel (periodic in j) CABARET step: the same sub-steps as the fused
// closed-basin kernels (qg3.F90:640-807, 940-956), as four node-parallel
// kernels.  Every row is interior in j; rows, j-faces and corners wrap
// modulo jj (the reference's halo rows and seam faces, qg3p_base.F90:
// 1887-1956, 2964-3003, hold exactly the wrapped values); the walls are the
// columns i = 0 and ii - 1.  One thread per (column, row) with all layers;
// face a (i-faces) and face b (j-faces) belong to node (a, b).  Arithmetic
// in FP64, fields stored as T.
namespace {

struct ChannelIdx {
    int ii, jj, pitch;
    long long ls;
    __device__ __forceinline__ long long at(int i, int j, int l) const {
        j = j < 0 ? j + jj : (j >= jj ? j - jj : j);
        return (long long)j * pitch + i + l * ls;
    }
};

// rel_from_zeta_and_psi + apply_rel_bc, then update_zeta_bc on the walls.
// rel is also kept in FP64 (in helm_io, free during a step) for the forcing's
// Laplacian, whose differences would lose the mixed form's FP32 digits.
template <typename T>
__global__ void k_ch_rel(const Member* __restrict__ mems, const int* __restrict__ prefix, int nmem) {
    int local;
    const int mi = find_member(prefix, nmem, blockIdx.y, &local);
    const Member& Mb = mems[mi];
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = local;
    if (i >= Mb.ii) return;
    const long long o = (long long)j * Mb.pitch + i;
    T* z = reinterpret_cast<T*>(Mb.zeta);
    T* rel = reinterpret_cast<T*>(Mb.rel);
    double* rel64 = reinterpret_cast<double*>(Mb.helm_io);
    auto ps = [&](int a, int b, int l) { return Mb.psi[(long long)b * Mb.pitch + a + l * Mb.lstride]; };
    const bool wall = (i == 0 || i == Mb.ii - 1);
    // psi_av += dt * psi once model time passes the threshold (qg3.F90:672-680).
    double* av = cab_average_gate(Mb) ? Mb.psi_av : nullptr;
    const double dt = Mb.sc->dt;
    for (int l = 0; l < Mb.L; ++l) {
        const long long ol = o + l * Mb.lstride;
        const double r = rel_node(Mb, ps, (double)z[ol], i, j, l);
        rel[ol] = (T)r;
        rel64[ol] = r;
        if (wall) z[ol] = (T)zeta_bc_node(Mb, ps, r, i, j, l);
        if (av) av[ol] = av[ol] + dt * Mb.psi[ol];
    }
}

// cabaret_forcing (qg3p_aux.F90:1065-1164) on the interior columns, and the
// time-integrated cell-boundary velocities (cabaret_cell_boundaries_
// time_integrated, :1235-1313) of the faces a = i (i-faces) and b = j
// (j-faces) of this node.
template <typename T>
__global__ void k_ch_force_cell(const Member* __restrict__ mems, const int* __restrict__ prefix, int nmem) {
    int local;
    const int mi = find_member(prefix, nmem, blockIdx.y, &local);
    const Member& Mb = mems[mi];
    const int ii = Mb.ii, L = Mb.L, i = blockIdx.x * blockDim.x + threadIdx.x, j = local;
    if (i >= ii) return;
    const ChannelIdx X{ii, Mb.jj, Mb.pitch, Mb.lstride};
    const int cur = Mb.cur, nxt = cur ^ 1;
    const double dt = Mb.sc->dt, tu = Mb.sc->tweight_u;
    T* z = reinterpret_cast<T*>(Mb.zeta);
    const double* rel = reinterpret_cast<const double*>(Mb.helm_io);  // FP64 rel of k_ch_rel
    const double* psi = Mb.psi;
    const double nu = Mb.viscosity, vb = Mb.visc_bot;
    if (i >= 1 && i <= ii - 2) {
        for (int l = 0; l < L; ++l) {
            auto rp = [&](int a, int b) { return rel[X.at(a, b, l)]; };
            const double lap = -4.0 * rp(i, j) + rp(i - 1, j) + rp(i + 1, j) + rp(i, j - 1) + rp(i, j + 1);
            const double wnd = (l == 0 && Mb.wind) ? Mb.wind[X.at(i, j, 0)] : 0.0;
            double rv;
            if (L == 1)
                rv = dt * (wnd - vb * rp(i, j) + nu * lap);
            else if (l == 0)
                rv = dt * (wnd + nu * lap);
            else if (l < L - 1)
                rv = dt * nu * lap;
            else
                rv = dt * (-vb * rp(i, j) + nu * lap);
            const long long o = X.at(i, j, l);
            z[o] = (T)((double)z[o] + rv);
        }
    }
    // psi_edge(a, b): the corner between nodes a-1, a and rows b-1, b.
    auto pe = [&](int a, int b, int l) {
        return 0.25 * (psi[X.at(a, b, l)] + psi[X.at(a, b - 1, l)] + psi[X.at(a - 1, b, l)] + psi[X.at(a - 1, b - 1, l)]);
    };
    T* ui = reinterpret_cast<T*>(Mb.ui);
    T* uj = reinterpret_cast<T*>(Mb.uj);
    const T* uimo = reinterpret_cast<const T*>(Mb.uimo[cur]);
    const T* ujmo = reinterpret_cast<const T*>(Mb.ujmo[cur]);
    T* uimn = reinterpret_cast<T*>(Mb.uimo[nxt]);
    T* ujmn = reinterpret_cast<T*>(Mb.ujmo[nxt]);
    for (int l = 0; l < L; ++l) {
        const long long o = X.at(i, j, l);
        if (i >= 1) {  // i-face a = i, row j
            const double uim = -pe(i, j + 1, l) + pe(i, j, l);
            ui[o] = (T)((1.0 + tu) * uim - tu * (double)uimo[o]);
            uimn[o] = (T)uim;
        }
        if (i >= 1 && i <= ii - 2) {  // j-face b = j of column i
            const double ujm = pe(i + 1, j, l) - pe(i, j, l);
            uj[o] = (T)((1.0 + tu) * ujm - tu * (double)ujmo[o]);
            ujmn[o] = (T)ujm;
        }
    }
}

// cabaret_extrapolator (qg3p_aux.F90:1317-1544) for the faces of this node;
// the j-faces of a channel always take the interior branch.
template <typename T>
__global__ void k_ch_extrap(const Member* __restrict__ mems, const int* __restrict__ prefix, int nmem) {
    int local;
    const int mi = find_member(prefix, nmem, blockIdx.y, &local);
    const Member& Mb = mems[mi];
    const int ii = Mb.ii, L = Mb.L, i = blockIdx.x * blockDim.x + threadIdx.x, j = local;
    if (i < 1 || i >= ii) return;
    const ChannelIdx X{ii, Mb.jj, Mb.pitch, Mb.lstride};
    const int cur = Mb.cur, nxt = cur ^ 1;
    const double dt = Mb.sc->dt;
    const bool lim = Mb.limiter != 0;
    const T* z = reinterpret_cast<const T*>(Mb.zeta);
    const T* zo = reinterpret_cast<const T*>(Mb.zeta_old[cur]);
    const T* ui = reinterpret_cast<const T*>(Mb.ui);
    const T* uj = reinterpret_cast<const T*>(Mb.uj);
    const T* fio = reinterpret_cast<const T*>(Mb.zfi[cur]);
    const T* fjo = reinterpret_cast<const T*>(Mb.zfj[cur]);
    T* fin = reinterpret_cast<T*>(Mb.zfi[nxt]);
    T* fjn = reinterpret_cast<T*>(Mb.zfj[nxt]);
    auto limit = [&](double v, double fi1, double fi2, double psi_n, double d_f) {
        if (lim) {
            const double fmx = fmax(fmax(fi1, fi2), psi_n) - d_f;
            const double fmn = fmin(fmin(fi1, fi2), psi_n) - d_f;
            if (v > fmx) v = fmx;
            if (v < fmn) v = fmn;
        }
        return v;
    };
    for (int l = 0; l < L; ++l) {
        const long long o = X.at(i, j, l);
        {  // i-face a = i between nodes i-1 and i
            const double u1 = ui[o], fi1 = fio[o];
            double fi2, psi_n, psi_o, d_f;
            if (u1 >= 0.0) {
                psi_n = z[o - 1];
                psi_o = zo[o - 1];
                if (i > 1) {
                    const double u2 = ui[o - 1];
                    fi2 = fio[o - 1];
                    const double v0 = (u1 + u2) / 2.0;
                    d_f = -(psi_n - psi_o) * 2.0 - dt * v0 * (fi1 - fi2);
                } else {
                    fi2 = psi_n;
                    d_f = -(psi_n - psi_o);
                }
            } else {
                psi_n = z[o];
                psi_o = zo[o];
                if (i < ii - 1) {
                    const double u2 = ui[o + 1];
                    fi2 = fio[o + 1];
                    const double v0 = (u1 + u2) / 2.0;
                    d_f = -(psi_n - psi_o) * 2.0 - dt * v0 * (fi2 - fi1);
                } else {
                    fi2 = psi_n;
                    d_f = -(psi_n - psi_o);
                }
            }
            fin[o] = (T)limit(2.0 * psi_n - fi2, fi1, fi2, psi_n, d_f);
        }
        if (i <= ii - 2) {  // j-face b = j between rows j-1 and j of column i
            const double u1 = uj[o], fi1 = fjo[o];
            double u2, fi2, psi_n, psi_o, d_f;
            if (u1 >= 0.0) {
                const long long om = X.at(i, j - 1, l);
                u2 = uj[om];
                fi2 = fjo[om];
                psi_n = z[om];
                psi_o = zo[om];
                d_f = -(psi_n - psi_o) * 2.0 - dt * ((u1 + u2) / 2.0) * (fi1 - fi2);
            } else {
                const long long op = X.at(i, j + 1, l);
                u2 = uj[op];
                fi2 = fjo[op];
                psi_n = z[o];
                psi_o = zo[o];
                d_f = -(psi_n - psi_o) * 2.0 - dt * ((u1 + u2) / 2.0) * (fi2 - fi1);
            }
            fjn[o] = (T)limit(2.0 * psi_n - fi2, fi1, fi2, psi_n, d_f);
        }
    }
}

// cabaret_flux + cabaret_corrector (qg3p_aux.F90:1547-1642), zeta_old =
// zeta; the largest |u| of this node's faces, and the last CTA's
// cabaret_cfl / cabaret_adapt_dt / model time (finish_step).
template <typename T>
__global__ void __launch_bounds__(128) k_ch_corrector(const Member* __restrict__ mems, const int* __restrict__ prefix,
                                                       int nmem) {
    __shared__ double red[4];
    int local;
    const int mi = find_member(prefix, nmem, blockIdx.y, &local);
    const Member& Mb = mems[mi];
    const int ii = Mb.ii, L = Mb.L, i = blockIdx.x * blockDim.x + threadIdx.x, j = local;
    const ChannelIdx X{ii, Mb.jj, Mb.pitch, Mb.lstride};
    const int nxt = Mb.cur ^ 1;
    double umax = 0.0;
    if (i < ii) {
        const double hdt = 0.5 * Mb.sc->dt;
        const T* z = reinterpret_cast<const T*>(Mb.zeta);
        const T* ui = reinterpret_cast<const T*>(Mb.ui);
        const T* uj = reinterpret_cast<const T*>(Mb.uj);
        const T* fin = reinterpret_cast<const T*>(Mb.zfi[nxt]);
        const T* fjn = reinterpret_cast<const T*>(Mb.zfj[nxt]);
        T* res = reinterpret_cast<T*>(Mb.res_out);
        T* zn = reinterpret_cast<T*>(Mb.zeta_old[nxt]);
        for (int l = 0; l < L; ++l) {
            const long long o = X.at(i, j, l);
            if (i >= 1) umax = fmax(umax, fabs((double)ui[o]));
            if (i >= 1 && i <= ii - 2) umax = fmax(umax, fabs((double)uj[o]));
            double zz = z[o];
            if (i >= 1 && i <= ii - 2) {
                const long long op = X.at(i, j + 1, l);
                const double fl0 = (double)ui[o] * (double)fin[o], fl1 = (double)ui[o + 1] * (double)fin[o + 1];
                const double fj0 = (double)uj[o] * (double)fjn[o], fj1 = (double)uj[op] * (double)fjn[op];
                const double r = -(fl1 - fl0 + fj1 - fj0);
                res[o] = (T)r;
                zz = zz + hdt * r;
            }
            zn[o] = (T)zz;
        }
    }
    umax = warp_max(umax);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) red[warp] = umax;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < 4; ++w) t = fmax(t, red[w]);
        if (count_done(Mb, t, (unsigned)Mb.ntiles_cab)) finish_step(Mb);
    }
}

}  // namespace

cudaError_t launch_cabaret_channel(const LaunchSet& ls, int f32, cudaStream_t st) {
    const dim3 g((ls.maxI + 127) / 128, ls.maxJ * ls.nmem);
    if (f32) {
        k_ch_rel<float><<<g, 128, 0, st>>>(ls.members, ls.prefix_rows_all, ls.nmem);
        k_ch_force_cell<float><<<g, 128, 0, st>>>(ls.members, ls.prefix_rows_all, ls.nmem);
        k_ch_extrap<float><<<g, 128, 0, st>>>(ls.members, ls.prefix_rows_all, ls.nmem);
        k_ch_corrector<float><<<g, 128, 0, st>>>(ls.members, ls.prefix_rows_all, ls.nmem);
    } else {
        k_ch_rel<double><<<g, 128, 0, st>>>(ls.members, ls.prefix_rows_all, ls.nmem);
        k_ch_force_cell<double><<<g, 128, 0, st>>>(ls.members, ls.prefix_rows_all, ls.nmem);
        k_ch_extrap<double><<<g, 128, 0, st>>>(ls.members, ls.prefix_rows_all, ls.nmem);
        k_ch_corrector<double><<<g, 128, 0, st>>>(ls.members, ls.prefix_rows_all, ls.nmem);
    }
    return cudaGetLastError();
}

int channel_ctas(int ii, int jj) { return ((ii + 127) / 128) * jj; }


// ---------------------------------------------------------------------------
// The quad eddy covariances of a step (qg3.F90:683-721), at the point of the
// reference's diagnostics: psi of the inversion, rel (rel_from_zeta_and_psi
// with its boundary condition) and zeta with its boundary PV.  The zonal and
// meridional velocities (qg3p_diagnostics.F90:941-1107) are 0 on the nodes
// the reference never writes, rel / alpha, 0 or NaN on the walls by the
// velocity boundary condition; interface velocities (:1163-1194), thickness
// (:1197-1227), the dt-weighted products (:1360-1427) and the scaled
// buoyancy correlations (:1430-1537).  One thread per node, all layers.
// Launched before the step's CABARET kernel, so the model-time gate is the
// one the fused kernel uses for psi_av.  lf: a leapfrog sub-step, launched
// after its rel kernel on the level just inverted (psi, rel, zeta
// BLEAPFROG); its gate is the model time already advanced by the sub-step,
// as k_lf_average's.
template <typename T>
__global__ void k_quad(const Member* __restrict__ mems, const int* __restrict__ prefix, int nmem, int lf) {
    int local;
    const int mi = find_member(prefix, nmem, blockIdx.y, &local);
    const Member& Mb = mems[mi];
    if (Mb.quad == nullptr) return;
    if (lf ? !(Mb.psi_av != nullptr && Mb.sc->model_time > Mb.av_threshold) : !cab_average_gate(Mb)) return;
    const int ii = Mb.ii, jj = Mb.jj, L = Mb.L, pitch = Mb.pitch;
    const long long ls = Mb.lstride, qs = Mb.quad_stride;
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = local;
    if (i >= ii) return;
    const double dt = Mb.sc->dt;
    const T* zp = reinterpret_cast<const T*>(Mb.zeta);
    auto ps = [&](int a, int b, int l) { return Mb.psi[(long long)b * pitch + a + l * ls]; };
    const long long o = (long long)j * pitch + i;
    // A channel (periodic j) has no j walls: every row is interior and its
    // j neighbours wrap.
    const bool per = Mb.periodic != 0;
    const bool in_i = i > 0 && i < ii - 1, in_j = per || (j > 0 && j < jj - 1);
    const int jm = (per && j == 0) ? jj - 1 : j - 1, jp = (per && j == jj - 1) ? 0 : j + 1;
    const int bc = Mb.bc_type;  // u, v on a wall from rel: rel / alpha, 0, or NaN
    double P[PQ_MAXL], R[PQ_MAXL], Z[PQ_MAXL], U[PQ_MAXL], V[PQ_MAXL], Tn[PQ_MAXL];
#pragma unroll
    for (int l = 0; l < PQ_MAXL; ++l) {
        if (l >= L) break;
        P[l] = ps(i, j, l);
        const double r = rel_node(Mb, ps, (in_i && in_j) ? (double)zp[o + l * ls] : 0.0, i, j, l);
        R[l] = r;
        Z[l] = (in_i && in_j) ? (double)zp[o + l * ls] : zeta_bc_node(Mb, ps, r, i, j, l);
        auto wall = [&]() { return bc == 1 ? r / Mb.alpha : bc == 2 ? 0.0 : __longlong_as_double(0x7ff8000000000000LL); };
        U[l] = (in_i && in_j) ? 0.5 * (ps(i + 1, j, l) - ps(i - 1, j, l)) : (in_j ? wall() : 0.0);
        V[l] = (in_i && in_j) ? 0.5 * (ps(i, jp, l) - ps(i, jm, l)) : (in_i ? wall() : 0.0);
    }
#pragma unroll
    for (int l = 0; l < PQ_MAXL; ++l) {
        if (l >= L) break;
        if (L == 1)
            Tn[l] = 0.0;
        else if (l == 0)
            Tn[l] = -Mb.s2[0] * (P[0] - P[1]);
        else if (l == L - 1)
            Tn[l] = -Mb.s1[l] * (P[l] - P[l - 1]);
        else
            Tn[l] = -Mb.s1[l] * (P[l] - P[l - 1]) - Mb.s2[l] * (P[l] - P[l + 1]);
    }
    double* q = Mb.quad + o;
    auto add = [&](int f, int l, double v) { q[f * qs + l * ls] += v; };
#pragma unroll
    for (int l = 0; l < PQ_MAXL; ++l) {
        if (l >= L) break;
        add(0, l, dt * U[l] * U[l]);
        add(1, l, dt * V[l] * V[l]);
        add(4, l, dt * U[l] * V[l]);
        add(5, l, dt * U[l] * R[l]);
        add(6, l, dt * V[l] * R[l]);
        add(7, l, dt * R[l] * R[l]);
        add(8, l, dt * P[l] * R[l]);
        add(9, l, dt * U[l] * Z[l]);
        add(10, l, dt * V[l] * Z[l]);
        add(11, l, dt * Z[l] * Z[l]);
        add(12, l, dt * Z[l] * R[l]);
        add(13, l, dt * P[l] * P[l]);
        add(14, l, dt * P[l] * Z[l]);
        add(15, l, dt * U[l] * Tn[l]);
        add(16, l, dt * V[l] * Tn[l]);
        add(17, l, dt * Tn[l] * R[l]);
        add(18, l, dt * Tn[l] * Tn[l]);
        if (l < L - 1) {
            const double ui = 0.5 * (U[l] + U[l + 1]), vi = 0.5 * (V[l] + V[l + 1]);
            add(2, l, dt * ui * ui);
            add(3, l, dt * vi * vi);
            const double dp = P[l] - P[l + 1];
            const double scb = Mb.s2[l] * Mb.h[l] * dp;
            add(19, l, dt * (0.5 * (U[l + 1] + U[l]) * scb));
            add(20, l, dt * (0.5 * (V[l + 1] + V[l]) * scb));
            add(22, l, dt * (Mb.s2[l] * Mb.h[l] * (dp * dp) / (Mb.h[l] + Mb.h[l + 1])));
        }
        if (L > 1) {
            double sbb;
            if (l == 0) {
                const double a = P[1] - P[0];
                sbb = 0.25 * (Mb.s2[0] * (a * a));
            } else if (l == L - 1) {
                const double a = P[l - 1] - P[l];
                sbb = 0.25 * (Mb.s1[l] * (a * a));
            } else {
                const double a = P[l - 1] - P[l], b = P[l + 1] - P[l];
                sbb = 0.25 * (Mb.s1[l] * (a * a) + Mb.s2[l] * (b * b));
            }
            add(21, l, dt * sbb);
        }
    }
}

cudaError_t launch_quad(const LaunchSet& ls, int f32, int lf, cudaStream_t st) {
    const dim3 g((ls.maxI + 127) / 128, ls.maxJ * ls.nmem);
    if (f32)
        k_quad<float><<<g, 128, 0, st>>>(ls.members, ls.prefix_rows_all, ls.nmem, lf);
    else
        k_quad<double><<<g, 128, 0, st>>>(ls.members, ls.prefix_rows_all, ls.nmem, lf);
    return cudaGetLastError();
}

cudaError_t launch_cabaret_fused(const LaunchSet& ls, int predict_next, int f32, cudaStream_t st) {
    if (f32) return predict_next ? launch_cab<true, float>(ls, st) : launch_cab<false, float>(ls, st);
    return predict_next ? launch_cab<true, double>(ls, st) : launch_cab<false, double>(ls, st);
}

// ---------------------------------------------------------------------------
// rel on demand (rel_from_zeta_and_psi + apply_rel_bc) from the zeta that
// entered the inversion and the current psi.  One thread per node.
template <typename T>
__global__ void k_rel(const Member* __restrict__ mems, const int* __restrict__ prefix, int nmem) {
    int local;
    const int mi = find_member(prefix, nmem, blockIdx.x, &local);
    const Member& Mb = mems[mi];
    const int ii = Mb.ii, jj = Mb.jj, L = Mb.L, pitch = Mb.pitch;
    const long long ls = Mb.lstride;
    const int j = local;
    const T* zp = reinterpret_cast<const T*>(Mb.zeta);
    T* rel = reinterpret_cast<T*>(Mb.rel);
    auto ps = [&](int i, int jn, int l) { return Mb.psi[(long long)jn * pitch + i + l * ls]; };
    for (int i = threadIdx.x; i < ii; i += blockDim.x)
        for (int l = 0; l < L; ++l) {
            const long long o = (long long)j * pitch + i + l * ls;
            const bool interior = i > 0 && i < ii - 1 && (Mb.periodic || (j > 0 && j < jj - 1));
            rel[o] = (T)rel_node(Mb, ps, interior ? (double)zp[o] : 0.0, i, j, l);
        }
}

cudaError_t launch_rel(const LaunchSet& ls, int f32, cudaStream_t st) {
    if (f32)
        k_rel<float><<<ls.ctas_rows_all, 256, 0, st>>>(ls.members, ls.prefix_rows_all, ls.nmem);
    else
        k_rel<double><<<ls.ctas_rows_all, 256, 0, st>>>(ls.members, ls.prefix_rows_all, ls.nmem);
    return cudaGetLastError();
}

// End of the START_PERTURB initialisation (qg3.F90:389-391, 450-452): rel
// from zeta and the new psi, boundary zeta from update_zeta_bc, and
// zeta_old = zeta.  One thread per node, one CTA per row.
template <typename T>
__global__ void k_init_finish(const Member* __restrict__ mems, const int* __restrict__ prefix, int nmem) {
    int local;
    const int mi = find_member(prefix, nmem, blockIdx.x, &local);
    const Member& Mb = mems[mi];
    const int ii = Mb.ii, jj = Mb.jj, L = Mb.L, pitch = Mb.pitch;
    const long long ls = Mb.lstride;
    const int j = local;
    const T* zp = reinterpret_cast<const T*>(Mb.zeta);
    T* rel = reinterpret_cast<T*>(Mb.rel);
    T* zo = reinterpret_cast<T*>(Mb.zeta_old[Mb.cur]);
    auto ps = [&](int i, int jn, int l) { return Mb.psi[(long long)jn * pitch + i + l * ls]; };
    for (int i = threadIdx.x; i < ii; i += blockDim.x)
        for (int l = 0; l < L; ++l) {
            const long long o = (long long)j * pitch + i + l * ls;
            const bool interior = i > 0 && i < ii - 1 && (Mb.periodic || (j > 0 && j < jj - 1));
            const double r = rel_node(Mb, ps, (double)zp[o], i, j, l);
            rel[o] = (T)r;
            zo[o] = interior ? zp[o] : (T)zeta_bc_node(Mb, ps, r, i, j, l);
        }
}

cudaError_t launch_init_finish(const LaunchSet& ls, int f32, cudaStream_t st) {
    if (f32)
        k_init_finish<float><<<ls.ctas_rows_all, 128, 0, st>>>(ls.members, ls.prefix_rows_all, ls.nmem);
    else
        k_init_finish<double><<<ls.ctas_rows_all, 128, 0, st>>>(ls.members, ls.prefix_rows_all, ls.nmem);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// energy, qg3p_diagnostics.F90:778-863: one CTA per row j computes the row's
// trapezoid-weighted potential-energy sum and the kinetic-energy sums of the
// cells whose upper-right node is on the row; the last CTA adds the row
// partials in row order and scales them.
__global__ void __launch_bounds__(256) k_energy(const Member* __restrict__ mems, const int* __restrict__ prefix,
                                                 int nmem) {
    __shared__ double red[8][PQ_MAXL + 1];
    __shared__ int is_last;
    int local;
    const int mi = find_member(prefix, nmem, blockIdx.x, &local);
    const Member& Mb = mems[mi];
    const int ii = Mb.ii, jj = Mb.jj, L = Mb.L, pitch = Mb.pitch;
    const long long ls = Mb.lstride;
    const int j = local;
    const double* psi = Mb.psi;
    double acc[PQ_MAXL + 1];
    for (int q = 0; q <= L; ++q) acc[q] = 0.0;
    // A channel has no j boundary: full weights, and the kinetic-energy
    // corners of row 0 reach back to row jj - 1.
    const double wj = (!Mb.periodic && (j == 0 || j == jj - 1)) ? 0.5 : 1.0;
    const long long back = (j == 0) ? (long long)(jj - 1) * pitch : -(long long)pitch;  // row j-1, wrapped
    for (int i = threadIdx.x; i < ii; i += blockDim.x) {
        const double w = wj * ((i == 0 || i == ii - 1) ? 0.5 : 1.0);
        const long long o = (long long)j * pitch + i;
        for (int k = 0; k < L - 1; ++k) {
            const double fac = 0.5 * Mb.s2[k] * Mb.h[k] / Mb.htot;
            const double d = psi[o + k * ls] - psi[o + (k + 1) * ls];
            acc[L] += w * fac * (d * d);
        }
        if (i >= 1 && (j >= 1 || Mb.periodic)) {
            for (int k = 0; k < L; ++k) {
                const long long lo = k * ls;
                const double a = psi[o - 1 + lo] + psi[o + lo] - psi[o - 1 + back + lo] - psi[o + back + lo];
                const double b = psi[o + back + lo] + psi[o + lo] - psi[o - 1 + back + lo] - psi[o - 1 + lo];
                acc[k] += 0.25 * (a * a + b * b);
            }
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int q = 0; q <= L; ++q) {
        const double v = warp_sum(acc[q]);
        if (lane == 0) red[warp][q] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 0; q <= L; ++q) {
            double t = 0.0;
            for (int w = 0; w < 8; ++w) t += red[w][q];
            Mb.partials[(long long)local * (PQ_MAXL + 1) + q] = t;
        }
        __threadfence();
        const unsigned prev = atomicAdd(&Mb.counters[2], 1u);
        is_last = (prev == (unsigned)(jj - 1));
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    double tot[PQ_MAXL + 1];
    for (int q = 0; q <= L; ++q) tot[q] = block_sum_l2(Mb.partials + q, jj, PQ_MAXL + 1, &red[0][0]);
    if (threadIdx.x != 0) return;
    Scalars* sc = Mb.sc;
    const double cff = Mb.mean_scale;
    const double epot = cff * tot[L];
    sc->epot = epot;
    bool bad = (epot != epot);
    for (int k = 0; k < L; ++k) {
        const double ek = 0.5 * cff * (Mb.h[k] / Mb.htot) * tot[k];
        sc->ekin[k] = ek;
        bad = bad || (ek != ek);
    }
    if (bad) atomicOr(Mb.status, (int)ST_NAN_ENERGY);
    Mb.counters[2] = 0u;
}

cudaError_t launch_energy(const LaunchSet& ls, cudaStream_t st) {
    k_energy<<<ls.ctas_rows_all, 256, 0, st>>>(ls.members, ls.prefix_rows_all, ls.nmem);
    return cudaGetLastError();
}

}  // namespace pq

namespace pq {

// FP64 <-> FP32 copies of pitched fields (the mixed form's state I/O).
__global__ void k_convert(void* __restrict__ dst, const void* __restrict__ src, size_t count, int to_f32) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < count; t += stride) {
        if (to_f32)
            static_cast<float*>(dst)[t] = (float)static_cast<const double*>(src)[t];
        else
            static_cast<double*>(dst)[t] = (double)static_cast<const float*>(src)[t];
    }
}

cudaError_t launch_convert(void* dst, const void* src, size_t count, int to_f32, cudaStream_t st) {
    size_t blocks = (count + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    k_convert<<<(unsigned)blocks, 256, 0, st>>>(dst, src, count, to_f32);
    return cudaGetLastError();
}

}  // namespace pq
