// SPDX-License-Identifier: 0BSD
// ---------------------------------------------------------------------------
// The reference's five launch wrappers (include/lpbf_kernels.hpp) on the
// B200 kernels, plus the extended-physics step.
//
//   lpbf_launch_step            -> temporally blocked kernel with K = 1,
//                                  no reduction (phys 0); ext kernel (phys 1)
//   lpbf_launch_step_reduce     -> same, with the reduction folded in: one
//                                  Partial per CTA, the remaining entries of
//                                  the caller's array set to the neutral
//                                  element so the caller's finalize over
//                                  ((nx+15)/16)*((ny+15)/16) entries is exact
//   lpbf_launch_reduce          -> row-parallel block reduce
//   lpbf_launch_reduce_finalize -> one 8-CTA cluster; partial results are
//                                  combined through distributed shared memory
//                                  (replaces the reference's <<<1,1>>> loop)
//   lpbf_launch_extract_col     -> one thread per row
// ---------------------------------------------------------------------------
#include <algorithm>
#include <cstring>
#include <cooperative_groups.h>

#include "lpbf_host.hpp"
#include "lpbf_kernels.hpp"

namespace cg = cooperative_groups;

namespace lpbf_b200 {

// ---- extended physics (temperature-dependent IN718 properties) ------------
// Mills tables, include/params.hpp:67-73 (physical data, identical values).
constexpr double EXT_T_PTS[9]  = {298, 473, 673, 873, 1073, 1273, 1473, 1533, 1609};
constexpr double EXT_K_PTS[9]  = {8.9, 12.9, 15.8, 18.7, 21.9, 25.6, 28.6, 29.3, 29.6};
constexpr double EXT_CP_PTS[9] = {435, 479, 515, 558, 580, 628, 670, 685, 720};
constexpr double T_SOL = 1533.0, T_LIQ = 1609.0, LATENT = 210.0e3;
constexpr double INV_MUSHY = 1.0 / (T_LIQ - T_SOL);

// The clamped piecewise-linear tables of params.hpp:75-89 as ten straight
// lines y = a + b T, one per temperature segment: segment 0 (T <= 298) and 9
// (T > 1609) hold the clamped end values, segment j the chord between table
// points j-1 and j.  The reference evaluates the same chord as
// y[j-1] + (T - t[j-1]) / (t[j] - t[j-1]) (y[j] - y[j-1]); the line form
// agrees with it to a few ulp of y.  A cell's segment is the number of table
// temperatures below T, decided on a 32-bit key of T (ext_key): for T >= 0
// the key is twice the upper word of T's bit pattern plus one when the lower
// word is non-zero, and every table temperature (an integer of at most 11
// significant bits) has a zero lower word, so T > t_j exactly when
// key(T) > key(t_j); a negative T gets key 0, segment 0, like the
// reference's clamp, and a NaN the top segment.  The key's upper 16 bits
// (exponent and 5 mantissa bits) cut [256, 2048) K into 96 buckets of
// 8-32 K, none holding more than one table temperature (the closest two are
// 60 K apart): a bucket's base segment (table temperatures below it) plus
// one compare against the next table temperature gives the segment.
constexpr int EXT_BUCKET0 = 0x407 << 5;   // upper 16 key bits of 256.0
constexpr int EXT_BUCKETS = 96;           // up to 2048.0
struct ExtLines {
    double ak[10], bk[10], ac[10], bc[10];
    unsigned int tkey[10];             // keys of the table temperatures; [9] = no bound
    unsigned int sol_key, liq_key;     // of T_SOL and T_LIQ
    unsigned char bseg[EXT_BUCKETS];   // base segment of each bucket
};
static_assert(sizeof(ExtLines) % sizeof(double) == 0, "copied to shared memory as doubles");

inline unsigned int host_key(double v) {
    unsigned long long b;
    std::memcpy(&b, &v, sizeof(b));
    return (unsigned int)((b >> 32) << 1) | (unsigned int)((b & 0xffffffffull) != 0);
}

ExtLines make_ext_lines() {
    ExtLines L;
    L.ak[0] = EXT_K_PTS[0];  L.bk[0] = 0.0;
    L.ac[0] = EXT_CP_PTS[0]; L.bc[0] = 0.0;
    for (int j = 1; j < 9; ++j) {
        const double w = EXT_T_PTS[j] - EXT_T_PTS[j - 1];
        L.bk[j] = (EXT_K_PTS[j] - EXT_K_PTS[j - 1]) / w;
        L.ak[j] = EXT_K_PTS[j - 1] - L.bk[j] * EXT_T_PTS[j - 1];
        L.bc[j] = (EXT_CP_PTS[j] - EXT_CP_PTS[j - 1]) / w;
        L.ac[j] = EXT_CP_PTS[j - 1] - L.bc[j] * EXT_T_PTS[j - 1];
    }
    L.ak[9] = EXT_K_PTS[8];  L.bk[9] = 0.0;
    L.ac[9] = EXT_CP_PTS[8]; L.bc[9] = 0.0;
    for (int j = 0; j < 9; ++j) L.tkey[j] = host_key(EXT_T_PTS[j]);
    L.tkey[9] = 0xffffffffu;
    L.sol_key = host_key(T_SOL);
    L.liq_key = host_key(T_LIQ);
    for (int b = 0; b < EXT_BUCKETS; ++b) {
        // the bucket's lowest value: upper word (EXT_BUCKET0 + b) << 15
        const unsigned long long bits = (unsigned long long)(unsigned)(EXT_BUCKET0 + b) << 47;
        double lo;
        std::memcpy(&lo, &bits, sizeof(lo));
        int base = 0;
        while (base < 9 && EXT_T_PTS[base] < lo) ++base;
        L.bseg[b] = (unsigned char)base;
    }
    return L;
}

__global__ void reduce_rows_kernel(const double* T, int nx, int ny, double Tm,
                                   Partial* out);
constexpr int FIN_CTAS = 8;
constexpr int FIN_THREADS = 512;
__global__ void finalize_cluster_kernel(const Partial* parts, int nblocks, int nx, int ny,
                        Partial* out);

__global__ void finalize_small_kernel(const Partial* parts, int nblocks, int nx,
                                      int ny, Partial* out);

// Launch finalize_cluster_kernel as one cluster of FIN_CTAS CTAs, or, for up
// to FIN_THREADS Partials (the unfused reduce's 256), one CTA: a cluster's
// launch and two cluster barriers cost more than the reduction (4.9 us for
// 256 Partials).
inline cudaError_t launch_finalize(const Partial* parts, int nblocks, int nx, int ny,
                                   Partial* out, cudaStream_t stream) {
    if (nblocks <= FIN_THREADS)
        return launch_chained_raw(finalize_small_kernel, 1, nblocks <= 256 ? 256 : FIN_THREADS,
                                  0, stream, parts, nblocks, nx, ny, out);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(FIN_CTAS, 1, 1);
    cfg.blockDim = dim3(FIN_THREADS, 1, 1);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = FIN_CTAS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, finalize_cluster_kernel, parts, nblocks, nx, ny, out);
}

constexpr int EXT_WARPS = 8;       // warps per CTA
constexpr int EXT_V = 2;           // columns per lane
constexpr int EXT_OWN = 30 * EXT_V;   // columns a warp owns (its first and last lane are halo)
constexpr int EXT_H = 64;          // most rows per task
constexpr int EXT_R = 4;           // rows per block: updated together, the next block's loaded ahead

struct ExtParams {
    StepConst k;
    ExtLines L;
    double hx, hy;                 // inv_dx2 / 2, inv_dy2 / 2 (face averages folded in)
    double r_dsub, Ta4, esig;      // 1/dSub, Tamb^4, eps sigma (0 without radiation)
    double dt_rho;                 // dt / rho
    double r2_cut;                 // beyond this r^2 the source is below 2^-80 of its peak
    int band_lo, band_hi, bandx_lo, bandx_hi;   // cells the source can reach
    int nstrips, H, ntasks;
    int bc;
    double T_edge, Tm;
    Partial* ring;
    Partial* scratch;
    unsigned int* counter;
    Partial* ref_out;
    long long ref_nparts;
};

// 1/d for the positive, normal d = cp_eff(T) (435..3200): the hardware's
// approximate FP64 reciprocal refined by two Newton-Raphson steps,
// r <- r + r (1 - d r), each of which squares the relative error.
__device__ __forceinline__ double rcp_newton(double d) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    double e = fma(-d, r, 1.0);
    r = fma(r, e, r);
    e = fma(-d, r, 1.0);
    return fma(r, e, r);
}

// One factor of the laser's heat input (kernels.cu:141): the input is a row
// factor (with the amplitude) times a column factor, each zero beyond the
// truncation radius, as in the baseline kernel.  Out of line: the exp code
// exists once in the binary and holds no registers in the row loop.
static __device__ __noinline__ double ext_factor(int i, double d, double centre,
                                                 double inv_r0_sq, double r2_cut) {
    const double z = __dsub_rn(__dmul_rn((double)i, d), centre);
    const double z2 = __dmul_rn(z, z);
    return z2 < r2_cut ? exp(__dmul_rn(-2.0 * z2, inv_r0_sq)) : 0.0;
}

// The ordering key of T (see ExtLines).
__device__ __forceinline__ unsigned int ext_key(double T) {
    const unsigned int hi = (unsigned int)__double2hiint(T);
    const unsigned int lo = (unsigned int)__double2loint(T);
    const unsigned int k = (hi << 1) | (lo != 0u ? 1u : 0u);
    return (int)hi < 0 ? 0u : k;
}

// Segment of a key in the tables (bucket base plus one compare; see
// ExtLines), from the shared-memory copy of the tables.
__device__ __forceinline__ int ext_seg(unsigned int key, const ExtLines& L) {
    const int b = (int)(key >> 16) - EXT_BUCKET0;
    const int base = L.bseg[min(max(b, 0), EXT_BUCKETS - 1)];
    const int s = base + (key > L.tkey[base] ? 1 : 0);
    return b < 0 ? 0 : (b >= EXT_BUCKETS ? 9 : s);
}

// k_eff(T) = k_of(T) k_enh(T, kmult) (params.hpp:91-105); kp = k_of(T).
// L: the line tables in shared memory (indexed per lane); Lp: the same
// in the parameter space (uniform reads).
template <bool KM>
__device__ __forceinline__ double ext_keff(double T, unsigned int key, int s, const ExtLines& L,
                                           const ExtLines& Lp, double kmult, double& kp) {
    kp = fma(L.bk[s], T, L.ak[s]);
    if constexpr (!KM) {
        return kp;
    } else {
        const double f = (key <= Lp.sol_key) ? 0.0
                       : (key >= Lp.liq_key) ? 1.0 : (T - T_SOL) * INV_MUSHY;
        return kp * fma(kmult - 1.0, f, 1.0);
    }
}

// A cell as the row stream carries it: T, k_eff(T), k_of(T) (the substrate
// loss uses the conductivity without kmult) and its segment.
struct ExtCell { double T, k, kp; int seg; };

template <bool KM>
__device__ __forceinline__ ExtCell ext_cell(double T, const ExtLines& L, const ExtLines& Lp,
                                            double kmult) {
    ExtCell c;
    c.T = T;
    const unsigned int key = ext_key(T);
    c.seg = ext_seg(key, L);
    c.k = ext_keff<KM>(T, key, c.seg, L, Lp, kmult, c.kp);
    return c;
}

// Flux through the face between cells a and b, (k_a + k_b)(T_b - T_a) (twice
// the arithmetic-mean face conductivity times the difference; the 1/2 is in
// hx, hy).
__device__ __forceinline__ double ext_flux(const ExtCell& a, const ExtCell& b) {
    return __dmul_rn(__dadd_rn(a.k, b.k), __dsub_rn(b.T, a.T));
}

// The new temperature of cell c from div(k grad T) and the source:
// T + dt (div + (q_in - q_top - q_bot) / h) / (rho cp_eff(T)).  With one
// surrounding temperature (SAMET: Tamb == Tsub) convection and conduction
// share their difference.
template <bool SAMET, bool SRC>
__device__ __forceinline__ double ext_update(const ExtCell& c, double div, double q_in,
                                             const StepConst& k, const ExtParams& p,
                                             const ExtLines& L) {
    const double T = c.T;
    const double T2 = __dmul_rn(T, T);
    const double e4 = fma(T2, T2, -p.Ta4);
    const double da = __dsub_rn(T, k.Tamb);
    double q;
    if constexpr (SAMET)
        q = fma(p.esig, e4, __dmul_rn(da, fma(c.kp, p.r_dsub, k.hConv)));
    else
        q = fma(p.esig, e4, fma(__dmul_rn(c.kp, p.r_dsub), __dsub_rn(T, k.Tsub),
                                __dmul_rn(k.hConv, da)));
    const double rhs = SRC ? fma(q_in - q, k.inv_h, div) : fma(-q, k.inv_h, div);
    double cp = fma(L.bc[c.seg], T, L.ac[c.seg]);
    const unsigned int key = ext_key(T);
    if (key >= p.L.sol_key && key <= p.L.liq_key) cp += LATENT * INV_MUSHY;
    return fma(__dmul_rn(rhs, p.dt_rho), rcp_newton(cp), T);
}

// A warp's place in the field and its carried rows: the centre row's cells and
// the fluxes through the faces above them.
struct ExtStrip {
    int xa, xb, cv, ca, cb;        // the lane's columns; clamped load columns
    bool own, own_b;
    int y1;
    ExtCell a, b;
    double Fua, Fub;
    double cfa, cfb;               // column factors of the source
    double thr, tm;                // reduction: threshold, lane peak and its cell
    int py, px, mn, mx;
};

// What a cell must exceed to change the lane's peak or a molten row.  A melt
// threshold that is NaN (no cell is molten) leaves the peak's.
__device__ __forceinline__ double ext_threshold(const ExtStrip& s, double Tm) {
    return s.own ? (Tm < s.tm ? Tm : s.tm) : INFINITY;
}

// Row y (clamped to the field) of the lane's two columns.  VEC (rows on
// 16-byte boundaries, nx even): a pair lies wholly on or off the field; one
// off it takes the edge cell twice.
template <bool VEC>
__device__ __forceinline__ void ext_load(const double* Tin, int nx, int ny, int y,
                                         const ExtStrip& s, double& u, double& v) {
    const double* row = Tin + (size_t)min(max(y, 0), ny - 1) * nx;
    if constexpr (VEC) {
        const double2 t = *reinterpret_cast<const double2*>(row + s.cv);
        u = s.xa >= nx ? t.y : t.x;
        v = s.xa < 0 ? t.x : t.y;
    } else {
        u = row[s.ca];
        v = row[s.cb];
    }
}

// EXT_R rows from y on (those below y1) in one straight line: their lower
// neighbours' values in Q (replaced by the next block's), no branch between
// rows, so the rows' chains (a table lookup is three dependent shared loads,
// the reciprocal five dependent operations) overlap.  With a branch per row a
// lone warp took 1 us per row.  SRC: the block meets the source.
template <bool REDUCE, bool KM, bool SAMET, bool VEC, bool SRC>
__device__ __forceinline__ void ext_block(const double* Tin,
                                          double* Tout, const ExtParams& p,
                                          const ExtLines& L, int y, ExtStrip& s,
                                          double (&Q)[EXT_R][2], int lane) {
    const StepConst& k = p.k;
    const int nx = k.nx, ny = k.ny;
    ExtCell da[EXT_R], db[EXT_R];
#pragma unroll
    for (int i = 0; i < EXT_R; ++i) {
        da[i] = ext_cell<KM>(Q[i][0], L, p.L, k.kmult);
        db[i] = ext_cell<KM>(Q[i][1], L, p.L, k.kmult);
    }
    // the next block's rows (past the task's end: a clamped, unused row)
#pragma unroll
    for (int i = 0; i < EXT_R; ++i)
        ext_load<VEC>(Tin, nx, ny, y + EXT_R + 1 + i, s, Q[i][0], Q[i][1]);
    // row factors of the source, one row per lane
    double rfl = 0.0;
    if constexpr (SRC) {
        const double f = ext_factor(y + min(lane, EXT_R - 1), k.dy, k.y_l, k.inv_r0_sq, p.r2_cut);
        rfl = f > 0.0 ? k.q_scale * k.peak_S * f : 0.0;
    }
    double va[EXT_R], vb[EXT_R];
#pragma unroll
    for (int i = 0; i < EXT_R; ++i) {
        // x faces: a|b inside the lane, b|next lane's a, and the previous
        // lane's b|a as this lane's left face; y faces: down, carried up
        const double Fab = ext_flux(s.a, s.b);
        const double TR = __shfl_down_sync(0xffffffffu, s.a.T, 1);
        const double kR = __shfl_down_sync(0xffffffffu, s.a.k, 1);
        const double FbR = __dmul_rn(__dadd_rn(s.b.k, kR), __dsub_rn(TR, s.b.T));
        const double FLa = __shfl_up_sync(0xffffffffu, FbR, 1);
        const double Fda = ext_flux(s.a, da[i]), Fdb = ext_flux(s.b, db[i]);
        const double diva = fma(__dsub_rn(Fda, s.Fua), p.hy, __dmul_rn(__dsub_rn(Fab, FLa), p.hx));
        const double divb = fma(__dsub_rn(Fdb, s.Fub), p.hy, __dmul_rn(__dsub_rn(FbR, Fab), p.hx));
        double qa = 0.0, qb = 0.0;
        if constexpr (SRC) {
            const double rf = __shfl_sync(0xffffffffu, rfl, i);
            qa = s.cfa > 0.0 ? __dmul_rn(rf, s.cfa) : 0.0;
            qb = s.cfb > 0.0 ? __dmul_rn(rf, s.cfb) : 0.0;
        }
        va[i] = ext_update<SAMET, SRC>(s.a, diva, qa, k, p, L);
        vb[i] = ext_update<SAMET, SRC>(s.b, divb, qb, k, p, L);
        s.Fua = Fda; s.Fub = Fdb;
        s.a = da[i]; s.b = db[i];
    }
    if (p.bc == 1) {
#pragma unroll
        for (int i = 0; i < EXT_R; ++i) {
            const bool ey = y + i == 0 || y + i == ny - 1;
            if (ey || s.xa == 0 || s.xa == nx - 1) va[i] = p.T_edge;
            if (ey || s.xb == 0 || s.xb == nx - 1) vb[i] = p.T_edge;
        }
    }
    double* row = Tout + (size_t)y * nx + s.xa;
#pragma unroll
    for (int i = 0; i < EXT_R; ++i) {
        const bool in = y + i < s.y1;
        if constexpr (VEC) {
            asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %3, 0;\n\t"
                         "@q st.global.v2.f64 [%0], {%1, %2};\n\t}"
                         :: "l"(row + (size_t)i * nx), "d"(va[i]), "d"(vb[i]),
                            "r"((int)(in && s.own)));
        } else {
            if (in && s.own) row[(size_t)i * nx] = va[i];
            if (in && s.own_b) row[(size_t)i * nx + 1] = vb[i];
        }
    }
    if constexpr (REDUCE) {
        // tested against min(lane peak, Tm); only a block in which some lane
        // crosses it updates peaks and molten rows.  A lane meets its cells in
        // increasing index order (rows down, a before b): strict '>' keeps the
        // first maximum; NaN never wins
        bool hit = false;
#pragma unroll
        for (int i = 0; i < EXT_R; ++i) hit |= va[i] > s.thr || vb[i] > s.thr;
        if (__any_sync(0xffffffffu, hit)) {
            unsigned int rows = 0u;
#pragma unroll
            for (int i = 0; i < EXT_R; ++i) {
                const bool ka = s.own && y + i < s.y1, kb = s.own_b && y + i < s.y1;
                if (ka && va[i] > s.tm) { s.tm = va[i]; s.py = y + i; s.px = s.xa; }
                if (kb && vb[i] > s.tm) { s.tm = vb[i]; s.py = y + i; s.px = s.xb; }
                rows |= (ka && va[i] > p.Tm) || (kb && vb[i] > p.Tm) ? 1u << i : 0u;
            }
            rows = __reduce_or_sync(0xffffffffu, rows);
            if (rows) {
                s.mn = min(s.mn, y + __ffs(rows) - 1);
                s.mx = max(s.mx, y + 31 - __clz(rows));
            }
            s.thr = ext_threshold(s, p.Tm);
        }
    }
}

// One warp advances one (strip, chunk) task: 60 owned columns (lane l holds
// the two columns xs + 2l and xs + 2l + 1; the outer lanes are the neighbours
// either side) down H rows.  Each cell's T and
// k_eff are loaded and evaluated once, when its row enters; a face's flux
// (k_a + k_b)(T_b - T_a) is computed once, inside the lane, by the lane to
// its left (passed on by a shuffle) or by the cell above it (y faces,
// carried to the next row in registers).  Loads of the
// cells just outside the field are clamped to the edge cell, which makes the
// edge faces' flux exactly zero: the reference's mirror ghost (ghost =
// centre).  The cell arithmetic follows include/step_task.hpp:144-184 and
// src/gpu/kernels.cu:125-147: div(k grad T) on arithmetic-mean faces, the
// source, convection, radiation and substrate losses, and the update
// T + dt rhs / (rho cp_eff(T)) with 1/cp_eff by rcp_newton.  Partials as in
// the baseline kernel: per lane over its owned cells, then warps, CTAs and
// the last CTA.
template <bool REDUCE, bool KM, bool SAMET, bool VEC>
__global__ void __launch_bounds__(EXT_WARPS * 32, 2)
ext_step_kernel(const double* Tin, double* Tout,
                const __grid_constant__ ExtParams p) {
    const StepConst& k = p.k;
    __shared__ ExtLines L;
    __shared__ Partial red[EXT_WARPS];
    __shared__ unsigned int s_last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x < (int)(sizeof(ExtLines) / sizeof(double)))
        reinterpret_cast<double*>(&L)[threadIdx.x] =
            reinterpret_cast<const double*>(&p.L)[threadIdx.x];
    __syncthreads();
    pdl_trigger();
    pdl_wait();
    const int nx = k.nx, ny = k.ny;
    const long long N = (long long)nx * ny;
    ExtStrip s;
    s.tm = -1.0;
    s.py = -1; s.px = 0;                   // no peak cell yet
    s.mn = ny; s.mx = -1;
    for (int task = blockIdx.x * EXT_WARPS + wid; task < p.ntasks;
         task += gridDim.x * EXT_WARPS) {
        const int strip = task % p.nstrips, chunk = task / p.nstrips;
        const int xs = strip * EXT_OWN - EXT_V;
        s.xa = xs + EXT_V * lane;
        s.xb = s.xa + 1;
        s.ca = min(max(s.xa, 0), nx - 1);
        s.cb = min(max(s.xb, 0), nx - 1);
        s.cv = min(max(s.xa, 0), nx - 2);
        s.own = lane >= 1 && lane <= 30 && s.xa < nx;
        s.own_b = s.own && s.xb < nx;
        const int y0 = chunk * p.H;
        s.y1 = min(y0 + p.H, ny);
        s.thr = ext_threshold(s, p.Tm);
        const bool src_strip = k.q_scale != 0.0 && xs + 32 * EXT_V > p.bandx_lo &&
                               xs <= p.bandx_hi;
        double Q[EXT_R][2];
        {
            // rows y0 - 1 (up) and y0 (centre), clamped at the field's edges
            double t0, t1, u0, u1;
            ext_load<VEC>(Tin, nx, ny, y0 - 1, s, t0, t1);
            ext_load<VEC>(Tin, nx, ny, y0, s, u0, u1);
#pragma unroll
            for (int i = 0; i < EXT_R; ++i)
                ext_load<VEC>(Tin, nx, ny, y0 + 1 + i, s, Q[i][0], Q[i][1]);
            const ExtCell ua = ext_cell<KM>(t0, L, p.L, k.kmult);
            const ExtCell ub = ext_cell<KM>(t1, L, p.L, k.kmult);
            s.a = ext_cell<KM>(u0, L, p.L, k.kmult);
            s.b = ext_cell<KM>(u1, L, p.L, k.kmult);
            s.Fua = ext_flux(ua, s.a);
            s.Fub = ext_flux(ub, s.b);
        }
        s.cfa = s.cfb = 0.0;
        if (src_strip && s.y1 > p.band_lo && y0 <= p.band_hi) {
            s.cfa = ext_factor(s.xa, k.dx, k.x_l, k.inv_r0_sq, p.r2_cut);
            s.cfb = ext_factor(s.xb, k.dx, k.x_l, k.inv_r0_sq, p.r2_cut);
        }
#pragma unroll 1
        for (int y = y0; y < s.y1; y += EXT_R) {
            if (src_strip && y + EXT_R > p.band_lo && y <= p.band_hi)
                ext_block<REDUCE, KM, SAMET, VEC, true>(Tin, Tout, p, L, y, s, Q, lane);
            else
                ext_block<REDUCE, KM, SAMET, VEC, false>(Tin, Tout, p, L, y, s, Q, lane);
        }
    }
    if constexpr (REDUCE) {
        double tm = s.tm;
        long long ag = s.py < 0 ? N : (long long)s.py * nx + s.px;
        int mn = s.mn, mx = s.mx;
        partial_warp_reduce(tm, ag, mn, mx);
        if (lane == 0) red[wid] = Partial{tm, ag, mn, mx};
        __syncthreads();
        if (threadIdx.x == 0) {
            double a = -1.0; long long b = N; int c1 = ny, d1 = -1;
            for (int w = 0; w < EXT_WARPS; ++w)
                partial_take(a, b, c1, d1, red[w].tmax, red[w].arg, red[w].ymin, red[w].ymax);
            if (p.ref_out) p.ref_out[blockIdx.x] = Partial{a, b, c1, d1};
            else p.scratch[blockIdx.x] = Partial{a, b, c1, d1};
        }
        if (p.ref_out) {
            // the rest of the caller's entries: the neutral element
            const Partial neutral{-1.0, N, ny, -1};
            for (long long i = gridDim.x + blockIdx.x * (long long)blockDim.x + threadIdx.x;
                 i < p.ref_nparts; i += (long long)gridDim.x * blockDim.x)
                p.ref_out[i] = neutral;
            return;
        }
        __syncthreads();
        if (threadIdx.x == 0) s_last = (ticket(p.counter) == gridDim.x - 1) ? 1u : 0u;
        __syncthreads();
        if (!s_last) return;
        double a = -1.0; long long b = N; int c1 = ny, d1 = -1;
        for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) {
            const Partial* qq = &p.scratch[i];
            partial_take(a, b, c1, d1, __ldcg(&qq->tmax), __ldcg(&qq->arg), __ldcg(&qq->ymin),
                         __ldcg(&qq->ymax));
        }
        partial_warp_reduce(a, b, c1, d1);
        __syncthreads();
        if (lane == 0) red[wid] = Partial{a, b, c1, d1};
        __syncthreads();
        if (threadIdx.x == 0) {
            double a2 = -1.0; long long b2 = N; int c2 = ny, d2 = -1;
            for (int w = 0; w < EXT_WARPS; ++w)
                partial_take(a2, b2, c2, d2, red[w].tmax, red[w].arg, red[w].ymin, red[w].ymax);
            p.ring[0] = Partial{a2, b2, c2, d2};
            *p.counter = 0u;
        }
    }
}

template <bool REDUCE, bool KM, bool SAMET>
cudaError_t launch_ext_v(bool vec, int grid, const double* Tin, double* Tout, const ExtParams& p,
                         cudaStream_t stream) {
    constexpr int threads = EXT_WARPS * 32;
    return launch_chained(vec ? ext_step_kernel<REDUCE, KM, SAMET, true>
                              : ext_step_kernel<REDUCE, KM, SAMET, false>,
                          grid, threads, 0, stream, Tin, Tout, p);
}
template <bool REDUCE>
cudaError_t launch_ext_t(bool km, int grid, const double* Tin, double* Tout, const ExtParams& p,
                         cudaStream_t stream) {
    // even rows on 16-byte boundaries: 16-byte loads and stores
    const bool vec = p.k.nx % 2 == 0 && reinterpret_cast<uintptr_t>(Tin) % 16 == 0 &&
                     reinterpret_cast<uintptr_t>(Tout) % 16 == 0;
    if (p.k.Tamb == p.k.Tsub)
        return km ? launch_ext_v<REDUCE, true, true>(vec, grid, Tin, Tout, p, stream)
                  : launch_ext_v<REDUCE, false, true>(vec, grid, Tin, Tout, p, stream);
    return km ? launch_ext_v<REDUCE, true, false>(vec, grid, Tin, Tout, p, stream)
              : launch_ext_v<REDUCE, false, false>(vec, grid, Tin, Tout, p, stream);
}

cudaError_t launch_ext_step(const double* Tin, double* Tout, const StepConst& k, int bc,
                            double T_edge, double Tm, Partial* ring, Workspace* ws,
                            Partial* ref_out, long long ref_nparts, cudaStream_t stream) {
    static const ExtLines lines = make_ext_lines();
    ExtParams p;
    std::memset(&p, 0, sizeof(p));
    p.k = k; p.L = lines;
    p.hx = 0.5 * k.inv_dx2;
    p.hy = 0.5 * k.inv_dy2;
    p.r_dsub = 1.0 / k.dSub;
    p.Ta4 = k.Tamb * k.Tamb * k.Tamb * k.Tamb;
    p.esig = k.radiation ? k.eps * SIGMA_SB : 0.0;
    p.dt_rho = k.dt / k.rho;
    p.bc = bc; p.T_edge = T_edge; p.Tm = Tm;
    p.ring = ring; p.ref_out = ref_out; p.ref_nparts = ref_nparts;
    // the source's reach: rows and columns where r^2 < r2_cut (a superset)
    const Coef c = make_coef(k, bc, T_edge, Tm);
    const LaserSub las = make_laser(k, k.x_l, k.y_l, k.q_scale);
    p.r2_cut = c.r2_cut;
    laser_band(c, &las, 1, &p.band_lo, &p.band_hi, &p.bandx_lo, &p.bandx_hi);
    p.nstrips = (k.nx + EXT_OWN - 1) / EXT_OWN;
    // 8..64 rows per task, in whole blocks, with the fewest waves x rows over
    // the resident warps (two CTAs per SM), the taller on a tie
    const long long warps = 2ll * EXT_WARPS * sm_count();
    long long best = -1;
    p.H = 8;
    for (int h = 8; h <= EXT_H; h += EXT_R) {
        const long long tasks = (long long)((k.ny + h - 1) / h) * p.nstrips;
        const long long cost = ((tasks + warps - 1) / warps) * (h + 4);
        if (best < 0 || cost <= best) { best = cost; p.H = h; }
    }
    p.ntasks = p.nstrips * ((k.ny + p.H - 1) / p.H);
    int grid = (p.ntasks + EXT_WARPS - 1) / EXT_WARPS;
    // resident CTAs only: a warp goes on to its next task (in a later chunk, as
    // its peak's tie rule needs) without leaving its place
    if (p.nstrips <= warps) grid = std::min(grid, 2 * sm_count());
    const bool km = k.kmult > 1.0;
    const bool reduce = ring || ref_out;
    if (ref_out) {
        grid = (int)std::max<long long>(1, std::min<long long>(grid, ref_nparts));
        return launch_ext_t<true>(km, grid, Tin, Tout, p, stream);
    }
    if (reduce) {
        if (!ws) return cudaErrorInvalidValue;
        grid = std::min(grid, MAX_CTAS * KMAX);
        p.scratch = ws->parts;
        p.counter = &ws->counter;
        return launch_ext_t<true>(km, grid, Tin, Tout, p, stream);
    }
    return launch_ext_t<false>(km, grid, Tin, Tout, p, stream);
}

// ---- standalone reduce --------------------------------------------------------
// Block b takes rows b, b + nblocks, ... (the reference's API fixes the grid
// at nblocks Partials, 256 for large fields: under two CTAs per SM), so each
// CTA keeps many bytes in flight: 1024 threads, each loading RR_VEC
// independent 16-byte pairs of a row before examining them.  A thread meets
// its cells in increasing index order (pairs in order, then the next group
// of pairs, then the next row), so a strict '>' keeps its first maximal
// cell; the block's threads then combine by the same rule as every Partial.
constexpr int RR_THREADS = 1024;
constexpr int RR_VEC = 4;

__device__ __forceinline__ void rr_take(double v, long long i, double& tm, long long& ag,
                                        bool& molten, double Tm) {
    if (v > tm) { tm = v; ag = i; }
    molten |= (v > Tm);
}

// 48 registers: a CTA then fits beside the step's last CTA on its SM and waits
// there for the field (56, which the loads alone would take: step, reduce and
// finalize at 1024^2 19.2 us against 18.2; at 2048^2 28.0 against 27.4).
__global__ void __maxnreg__(48)
reduce_rows_kernel(const double* T, int nx, int ny, double Tm,
                   Partial* out) {
    const long long N = (long long)nx * ny;
    double tm = -1.0; long long ag = N; int mn = ny, mx = -1;
    pdl_trigger();
    pdl_wait();
    // 16-byte pairs when every row starts on a 16-byte boundary
    const bool pairs = (nx % 2 == 0) && (reinterpret_cast<uintptr_t>(T) % 16 == 0);
    // Rows shorter than the block's loads in flight: several rows at once (a
    // row of 512 pairs alone left half the threads idle and one load per
    // thread in flight: 8.5 us at 1024^2 for 8 MB that sit in L2).
    const int rpp = pairs ? RR_THREADS * RR_VEC / (nx / 2) : 0;      // rows per pass
    if (rpp > 1) {
        const int np = nx / 2, slots = rpp * np;
        for (long long y0 = blockIdx.x; y0 < ny; y0 += (long long)gridDim.x * rpp) {
            double2 v[RR_VEC];
            int xx[RR_VEC], yy[RR_VEC];
#pragma unroll
            for (int u = 0; u < RR_VEC; ++u) {
                const int q = threadIdx.x + u * RR_THREADS, rr = q / np;
                const long long y = y0 + (long long)rr * gridDim.x;
                v[u] = make_double2(-INFINITY, -INFINITY);
                xx[u] = 2 * (q - rr * np);
                yy[u] = (int)y;
                if (q < slots && y < ny) v[u] = *reinterpret_cast<const double2*>(T + y * nx + xx[u]);
            }
#pragma unroll
            for (int u = 0; u < RR_VEC; ++u) {
                bool molten = false;
                const long long i = (long long)yy[u] * nx + xx[u];
                rr_take(v[u].x, i, tm, ag, molten, Tm);
                rr_take(v[u].y, i + 1, tm, ag, molten, Tm);
                if (molten) { mn = min(mn, yy[u]); mx = max(mx, yy[u]); }
            }
        }
    }
    for (int y = rpp > 1 ? ny : blockIdx.x; y < ny; y += gridDim.x) {
        const double* row = T + (size_t)y * nx;
        const long long base = (long long)y * nx;
        bool molten = false;
        if (pairs) {
            const double2* r2 = reinterpret_cast<const double2*>(row);
            const int np = nx / 2;
            for (int p0 = threadIdx.x; p0 < np; p0 += RR_THREADS * RR_VEC) {
                double2 v[RR_VEC];
#pragma unroll
                for (int u = 0; u < RR_VEC; ++u) {
                    const int p = p0 + u * RR_THREADS;
                    v[u] = p < np ? r2[p] : make_double2(-INFINITY, -INFINITY);
                }
#pragma unroll
                for (int u = 0; u < RR_VEC; ++u) {
                    const long long i = base + 2ll * (p0 + u * RR_THREADS);
                    rr_take(v[u].x, i, tm, ag, molten, Tm);
                    rr_take(v[u].y, i + 1, tm, ag, molten, Tm);
                }
            }
        } else {
            for (int x0 = threadIdx.x; x0 < nx; x0 += RR_THREADS * RR_VEC) {
                double v[RR_VEC];
#pragma unroll
                for (int u = 0; u < RR_VEC; ++u) {
                    const int x = x0 + u * RR_THREADS;
                    v[u] = x < nx ? row[x] : -INFINITY;
                }
#pragma unroll
                for (int u = 0; u < RR_VEC; ++u)
                    rr_take(v[u], base + x0 + u * RR_THREADS, tm, ag, molten, Tm);
            }
        }
        if (molten) { mn = min(mn, y); mx = max(mx, y); }
    }
    partial_warp_reduce(tm, ag, mn, mx);
    __shared__ Partial red[RR_THREADS / 32];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = Partial{tm, ag, mn, mx};
    __syncthreads();
    if (threadIdx.x < 32) {
        Partial q = red[threadIdx.x];
        double a = q.tmax; long long b = q.arg; int c = q.ymin, d = q.ymax;
        partial_warp_reduce(a, b, c, d);
        if (threadIdx.x == 0) out[blockIdx.x] = Partial{a, b, c, d};
    }
}

// ---- finalize: one cluster of FIN_CTAS CTAs ----------------------------------

__global__ void finalize_cluster_kernel(const Partial* parts, int nblocks, int nx, int ny,
                        Partial* out) {
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ Partial red[FIN_THREADS / 32];
    __shared__ Partial cta_result;
    const long long N = (long long)nx * ny;
    double tm = -1.0; long long ag = N; int mn = ny, mx = -1;
    const int rank = (int)cluster.block_rank();
    pdl_trigger();
    pdl_wait();
    for (int i = rank * FIN_THREADS + threadIdx.x; i < nblocks; i += FIN_CTAS * FIN_THREADS) {
        const Partial q = parts[i];
        partial_take(tm, ag, mn, mx, q.tmax, q.arg, q.ymin, q.ymax);
    }
    partial_warp_reduce(tm, ag, mn, mx);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = Partial{tm, ag, mn, mx};
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = -1.0; long long b = N; int c = ny, d = -1;
        for (int w = 0; w < FIN_THREADS / 32; ++w)
            partial_take(a, b, c, d, red[w].tmax, red[w].arg, red[w].ymin, red[w].ymax);
        cta_result = Partial{a, b, c, d};
    }
    cluster.sync();
    if (rank == 0 && threadIdx.x == 0) {
        double a = -1.0; long long b = N; int c = ny, d = -1;
        for (int r = 0; r < FIN_CTAS; ++r) {
            const Partial* q = cluster.map_shared_rank(&cta_result, r);
            partial_take(a, b, c, d, q->tmax, q->arg, q->ymin, q->ymax);
        }
        out[0] = Partial{a, b, c, d};
    }
    cluster.sync();   // keep every CTA's shared memory alive until rank 0 has read it
}

__global__ void __launch_bounds__(FIN_THREADS)
finalize_small_kernel(const Partial* parts, int nblocks, int nx, int ny,
                      Partial* out) {
    __shared__ Partial red[FIN_THREADS / 32];
    const long long N = (long long)nx * ny;
    double tm = -1.0; long long ag = N; int mn = ny, mx = -1;
    pdl_trigger();
    pdl_wait();
    if ((int)threadIdx.x < nblocks) {
        const Partial q = parts[threadIdx.x];
        partial_take(tm, ag, mn, mx, q.tmax, q.arg, q.ymin, q.ymax);
    }
    partial_warp_reduce(tm, ag, mn, mx);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = Partial{tm, ag, mn, mx};
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = -1.0; long long b = N; int c = ny, d = -1;
        for (int w = 0; w < (int)blockDim.x / 32; ++w)
            partial_take(a, b, c, d, red[w].tmax, red[w].arg, red[w].ymin, red[w].ymax);
        out[0] = Partial{a, b, c, d};
    }
}

__global__ void extract_col_kernel(const double* T, int nx, int ny,
                                   const Partial* glob, double* col) {
    const int y = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_trigger();
    pdl_wait();
    if (y >= ny) return;
    const long long a = glob->arg;
    const int x = (int)(a % nx);
    col[y] = (a >= 0 && a < (long long)nx * ny) ? T[(size_t)y * nx + x] : 0.0;
}

}  // namespace lpbf_b200

using namespace lpbf_b200;

extern "C" {

void lpbf_launch_step(const double* Tin, double* Tout, const StepConst* k, int phys,
                      cudaStream_t stream) {
    if (phys == 0) {
        const Coef c = make_coef(*k, 0, 0.0, 0.0);
        const LaserSub las = make_laser(*k, k->x_l, k->y_l, k->q_scale);
        launch_advance(1, Tin, Tout, c, &las, nullptr, nullptr, nullptr, 0, 0, stream);
    } else {
        launch_ext_step(Tin, Tout, *k, 0, 0.0, 0.0, nullptr, nullptr, nullptr, 0, stream);
    }
}

void lpbf_launch_reduce(const double* T, int nx, int ny, double Tm, Partial* out,
                        int nblocks, cudaStream_t stream) {
    if (nblocks <= 0) return;
    launch_chained_raw(reduce_rows_kernel, nblocks, RR_THREADS, 0, stream, T, nx, ny, Tm, out);
}

void lpbf_launch_step_reduce(const double* Tin, double* Tout, const StepConst* k, int phys,
                             double Tm, Partial* out, cudaStream_t stream) {
    const long long nparts = (long long)((k->nx + 15) / 16) * ((k->ny + 15) / 16);
    if (phys == 0) {
        const Coef c = make_coef(*k, 0, 0.0, Tm);
        const LaserSub las = make_laser(*k, k->x_l, k->y_l, k->q_scale);
        launch_advance(1, Tin, Tout, c, &las, nullptr, nullptr, out, nparts, 0, stream);
    } else {
        launch_ext_step(Tin, Tout, *k, 0, 0.0, Tm, nullptr, nullptr, out, nparts, stream);
    }
}

void lpbf_launch_reduce_finalize(const Partial* parts, int nblocks, int nx, int ny,
                                 Partial* out, cudaStream_t stream) {
    launch_finalize(parts, nblocks, nx, ny, out, stream);
}

void lpbf_launch_extract_col(const double* T, int nx, int ny, const Partial* glob,
                             double* out_col, cudaStream_t stream) {
    const int bs = 128;
    launch_chained_raw(extract_col_kernel, (ny + bs - 1) / bs, bs, 0, stream, T, nx, ny, glob,
                       out_col);
}

}  // extern "C"
