// SPDX-License-Identifier: 0BSD
// ---------------------------------------------------------------------------
// Small and middling fields: one persistent launch for many time steps, the
// field resident in registers.
//
// A launch per few steps leaves a small field waiting: at 240 x 120 a launch
// of the temporally blocked kernel took 20 us and its cells' arithmetic under
// 0.1 us.  Here the field is cut into at most one tile per SM.  A CTA holds
// its tile and a halo of K cells per side, advances K steps on it, trades K
// boundary cells with its eight neighbours through global memory (L2) and
// goes on, up to RES_STEPS steps per launch.
//
// Layout.  A CTA's padded tile is 32 V columns by 16 NR rows: warp w holds
// rows w NR .. w NR + NR - 1, a lane V consecutive columns of each, all in
// registers.  Per step only the rows at the warps' seams pass through shared
// memory (double-buffered, one barrier per step); x neighbours come by
// shuffle; halo cells and rims move between registers and L2 directly.
// (With the tile in shared memory instead, loads, per-cell index tracking
// and store predicates took 140 instructions per row of two cells a lane,
// and a step of a 43 x 43 tile 2.2 us.)  V = 2 suits small fields (short
// steps), V = 4 larger ones (half the shuffles per cell).  What bounds it:
// for small tiles the exchange (store, release, poll, load: paid once per K
// steps) and the latency of one step inside the CTA; for large tiles the FP64
// pipe.  The host picks V, NR, K and the tiling by a model (resident_plan).
//
// Validity.  After step t of a block the outermost t rows and columns of the
// padded tile are stale (their neighbours lie outside); with kb <= K steps
// per block the owned cells are exact.  Cells off the field are computed too
// and never used: at a mirror edge the edge cell takes itself as neighbour.
//
// Exchange.  Block b (of nblocks, an odd number) ends with the tile's rim in
// buffer X_b, Tout for odd b and Tin for even b, and flag b posted; the CTA
// then waits for its neighbours' flags >= b and loads its halo from X_b.
// Two buffers suffice: a CTA overwrites X_b at the end of block b + 2, which
// it reaches only after every neighbour posted b + 1, that is, after each
// finished loading from X_b.  The last block writes the whole tile to Tout
// (nblocks is odd, so that is X_nblocks).  All CTAs are co-resident
// (cooperative launch) and every wait is bounded.
//
// Reduction.  Each lane leaves, per step, the first maximum of its owned
// cells in shared memory (a step's chain holds no warp reduction); a block's
// records are folded per CTA while the exchange is under way (integer warp
// reductions on an order-preserving key), and after the last block every CTA
// folds its share of the steps over all CTAs.  Molten rows are rare: shared
// atomics.
//
// Cell arithmetic is the temporally blocked kernel's (cell_core, cell_update,
// src_product): results equal it bit for bit.
// ---------------------------------------------------------------------------
#pragma once
#include "lpbf_advance.cuh"
#include "lpbf_host.hpp"

namespace lpbf_b200 {

constexpr int RES_THREADS = 512;
constexpr int RES_WARPS = RES_THREADS / 32;
constexpr int RES_STEPS = RES_MAX_STEPS;   // the laser records are kernel parameters
constexpr int RES_KMAX = 16;        // most steps between exchanges (one fold warp per step)
constexpr int RES_MAX_TILES = 160;  // most CTAs (tiles) of a launch
constexpr int RES_FLAG_STRIDE = 8;  // flags 32 bytes apart
static_assert(sizeof(Workspace::flags) >= RES_MAX_TILES * RES_FLAG_STRIDE * sizeof(unsigned), "flags");
static_assert(WS_PARTS >= RES_MAX_TILES * RES_STEPS, "records");
constexpr int RES_KEY_SHIFT = 8;    // local key of a cell: row << 8 | column (at most 128)
constexpr unsigned int RES_NO_KEY = 0x7fffffffu;      // a lane without a peak
constexpr unsigned long long RES_WAIT_NS = 4000000000ull;

struct ResParams {
    Coef c;
    const double* Tin;
    double* Tout;
    double* xbuf[2];               // [b & 1]: where block b leaves its rim
    Partial* ring;
    Partial* scratch;              // [step][cta]
    unsigned int* flags;           // RES_FLAG_STRIDE words per CTA, zero between launches
    unsigned int* counter;         // exit ticket, zero between launches
    unsigned int* barrier;         // arrivals of the final fold, zero between launches
    unsigned int* err;
    const unsigned int* wait_ns;   // Workspace::wait_ns
    int n_steps, nblocks, K;       // K: most steps of a block
    int gx, gy;                    // tiles per row and column of tiles
    int hx, hy;                    // halo columns and rows held per side
    LaserSub las[RES_STEPS];
};

// Bounds of tile i of n over a length: multiples of `unit` but for the end.
__host__ __device__ inline int res_bound(int i, int n, int len, int unit) {
    const int u = (len + unit - 1) / unit;
    const int b = (int)((long long)i * u / n) * unit;
    return b < len ? b : len;
}
// First step of block b.
__host__ __device__ inline int res_step(int b, int nblocks, int n) {
    return b * n / nblocks;       // n <= RES_STEPS
}
// Largest m over the warp and the smallest key (below 2^31) among the lanes
// that hold it, in every lane: partial_warp_peak with short indices.
__device__ __forceinline__ void res_warp_max(double& m, unsigned int& key) {
    unsigned long long k = order_key(m);
    const unsigned int z = k == NEG_ZERO_KEY ? 1u : 0u;
    k += z;
    const unsigned int hi = (unsigned int)(k >> 32), lo = (unsigned int)k;
    const unsigned int h = __reduce_max_sync(0xffffffffu, hi);
    const unsigned int l = __reduce_max_sync(0xffffffffu, hi == h ? lo : 0u);
    const unsigned int g =
        __reduce_min_sync(0xffffffffu, hi == h && lo == l ? key << 1 | z : 0xffffffffu);
    m = g & 1u ? -0.0 : order_unkey(((unsigned long long)h << 32) | l);
    key = g >> 1;
}

__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(unsigned int* p, unsigned int v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" :: "l"(p), "r"(v) : "memory");
}
// Wait until *p >= want, at most *limit ns (0: RES_WAIT_NS).
__device__ __forceinline__ bool res_wait(const unsigned int* p, unsigned int want,
                                         const unsigned int* limit) {
    if (ld_acquire(p) >= want) return true;
    const uint64_t t0 = globaltimer_ns();
    const unsigned int w = *limit;
    const uint64_t ns = w ? w : RES_WAIT_NS;
    while (ld_acquire(p) < want)
        if (globaltimer_ns() - t0 > ns) return false;
    return true;
}

// MODE 0: Tamb == Tsub, square cells; 1: Tamb == Tsub; 2: general.
template <int MODE, bool SRC>
__device__ __forceinline__ double res_cell(double T, double L, double R, double U, double D,
                                           double S, const HotCoef& h, const Coef& c) {
    if constexpr (MODE == 2) return cell_update(T, L, R, U, D, SRC ? S : 0.0, c);
    else if constexpr (SRC) return cell_core_src<MODE == 0>(T, L, R, U, D, S, h);
    else return cell_core<MODE == 0>(T, L, R, U, D, h);
}

// A lane's V cells of a row, to and from shared memory.
template <int V>
__device__ __forceinline__ void res_lds(double (&d)[V], const double* p) {
#pragma unroll
    for (int v = 0; v < V; v += 2) {
        const double2 a = *reinterpret_cast<const double2*>(p + v);
        d[v] = a.x;
        d[v + 1] = a.y;
    }
}
template <int V>
__device__ __forceinline__ void res_sts(double* p, const double (&d)[V]) {
#pragma unroll
    for (int v = 0; v < V; v += 2)
        *reinterpret_cast<double2*>(p + v) = make_double2(d[v], d[v + 1]);
}

// One step of a warp's NR rows, in place.  up, dn: the rows above and below
// (previous step).  rf: the rows' source factors, cf: the lane's columns'.
template <int V, int NR, int MODE, bool SRC>
__device__ __forceinline__ void res_step_rows(double (&T)[NR][V], const double (&up)[V],
                                              const double (&dn)[V], const double* rf,
                                              const double (&cf)[V], const HotCoef& h,
                                              const Coef& c, bool first_col, bool last_col) {
    double prev[V];
#pragma unroll
    for (int v = 0; v < V; ++v) prev[v] = up[v];
#pragma unroll
    for (int i = 0; i < NR; ++i) {
        double ce[V], nx[V];
#pragma unroll
        for (int v = 0; v < V; ++v) {
            ce[v] = T[i][v];
            nx[v] = i + 1 < NR ? T[i + 1 < NR ? i + 1 : i][v] : dn[v];
        }
        double Lo = __shfl_up_sync(0xffffffffu, ce[V - 1], 1);
        double Ro = __shfl_down_sync(0xffffffffu, ce[0], 1);
        // mirror edges: the field's first and last cell see themselves
        Lo = first_col ? ce[0] : Lo;
        Ro = last_col ? ce[V - 1] : Ro;
        double r = 0.0;
        if constexpr (SRC) r = rf[i];
#pragma unroll
        for (int v = 0; v < V; ++v) {
            double S = 0.0;
            if constexpr (SRC) S = src_product(r, cf[v]);
            T[i][v] = res_cell<MODE, SRC>(ce[v], v > 0 ? ce[v > 0 ? v - 1 : 0] : Lo,
                                          v + 1 < V ? ce[v + 1 < V ? v + 1 : v] : Ro, prev[v],
                                          nx[v], S, h, c);
        }
#pragma unroll
        for (int v = 0; v < V; ++v) prev[v] = ce[v];
    }
}

// Shared memory: seam rows, source factors, reduction records (peak, then key).
__host__ __device__ constexpr size_t res_smem_bytes(int V, int NR, int K) {
    return (2 * RES_WARPS * 2 * 32 * V + (size_t)K * (32 * V + RES_WARPS * NR)) * sizeof(double) +
           (size_t)K * RES_THREADS * (sizeof(double) + sizeof(unsigned int));
}

template <int V, int NR, int MODE, bool REDUCE>
__global__ void __launch_bounds__(RES_THREADS, 1)
resident_kernel(const __grid_constant__ ResParams p) {
    constexpr int COLS = 32 * V, ROWS = RES_WARPS * NR;
    extern __shared__ __align__(16) double res_smem[];
    __shared__ int s_mn[RES_KMAX], s_mx[RES_KMAX];       // molten rows of a block's steps
    __shared__ int s_flag;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const Coef& c = p.c;
    const int nx = c.nx, ny = c.ny;
    const HotCoef h = hot_coef(c);
    // the warps' top and bottom rows, double-buffered by step
    auto s_seam = reinterpret_cast<double (*)[RES_WARPS][2][COLS]>(res_smem);
    double* const colf = res_smem + 2 * RES_WARPS * 2 * COLS;       // [K][COLS]
    double* const rowf = colf + (size_t)p.K * COLS;      // [K][ROWS]
    double* const recm = rowf + (size_t)p.K * ROWS;      // [K][RES_THREADS]
    unsigned int* const reck = reinterpret_cast<unsigned int*>(recm + (size_t)p.K * RES_THREADS);
    if (tid < RES_KMAX) { s_mn[tid] = 0x7fffffff; s_mx[tid] = -1; }

    const int bx = blockIdx.x % p.gx, by = blockIdx.x / p.gx;
    const int tx0 = res_bound(bx, p.gx, nx, V), tx1 = res_bound(bx + 1, p.gx, nx, V);
    const int ty0 = res_bound(by, p.gy, ny, 1), ty1 = res_bound(by + 1, p.gy, ny, 1);
    const int px0 = tx0 - p.hx, py0 = ty0 - p.hy;        // the padded tile's corner
    const int x = px0 + V * lane;                        // this lane's first column
    const int y = py0 + NR * wid;                        // this warp's first row
    const bool own_x = x >= tx0 && x < tx1;              // tiles end on multiples of V (or nx)
    const bool first_col = x == 0 && c.bc == 0, last_col = x + V - 1 == nx - 1 && c.bc == 0;
    // edge work is left out of tiles that do not meet it (uniform over the CTA)
    const bool ragged = nx % V != 0 && px0 + COLS >= nx; // the field ends inside a lane
    const bool edge_y = py0 < 0 || py0 + ROWS >= ny;
    const bool edge_x = px0 <= 0 || px0 + COLS >= nx;

    double T[NR][V];
    // all the field's cells that block 1 needs
    {
        const int k1 = res_step(1, p.nblocks, p.n_steps);
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            const int yy = y + i;
            const bool row = yy >= max(ty0 - k1, 0) && yy < min(ty1 + k1, ny);
            const double* src = p.Tin + (size_t)yy * nx + x;
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const int xx = x + v;
                T[i][v] = row && xx >= max(tx0 - k1, 0) && xx < min(tx1 + k1, nx)
                              ? __ldcg(src + v) : c.Tamb;
            }
        }
    }
    // source factors of steps [s0, s0 + kb); whether any row, any column of
    // the padded tile meets the source
    bool any_row = false, any_col = false;
    auto factors = [&](int s0, int kb) {
        any_row = any_col = false;
        for (int i = tid; i < kb * (ROWS + COLS); i += RES_THREADS) {
            const int t = i / (ROWS + COLS), q = i % (ROWS + COLS);
            const LaserSub& l = p.las[s0 + t];
            const bool is_row = q < ROWS;
            const double d = is_row
                ? __dsub_rn(__dmul_rn((double)(py0 + q), c.dy), l.y_l)
                : __dsub_rn(__dmul_rn((double)(px0 + q - ROWS), c.dx), l.x_l);
            double f = src_factor(d, c.m2r, c.r2_cut);
            if (is_row) {
                f = f > 0.0 ? __dmul_rn(l.cs, f) : 0.0;          // src_row
                rowf[t * ROWS + q] = f;
                any_row |= f != 0.0;
            } else {
                colf[t * COLS + q - ROWS] = f;
                any_col |= f != 0.0;
            }
        }
    };

    // the columns past a field's end that lies inside a lane hold copies of
    // the last one: its mirror neighbour, and never a first maximum
    auto ghost_cols = [&]() {
#pragma unroll
        for (int i = 0; i < NR; ++i)
#pragma unroll
            for (int v = 0; v + 1 < V; ++v)
                T[i][v + 1] = x + v >= nx - 1 ? T[i][v] : T[i][v + 1];
    };

    bool failed = false;
    int s0 = 0, s1 = res_step(1, p.nblocks, p.n_steps);
    int buf = 0;
    factors(s0, s1);
    bool src = __syncthreads_or(any_row);
    src = __syncthreads_or(any_col) && src;
    for (int b = 1; b <= p.nblocks; ++b) {
        const int kb = s1 - s0;
        if (ragged) ghost_cols();
        // the seams of the block's first step
        res_sts<V>(&s_seam[buf][wid][0][V * lane], T[0]);
        if constexpr (NR > 1) res_sts<V>(&s_seam[buf][wid][1][V * lane], T[NR - 1]);
        __syncthreads();
        for (int t = 0; t < kb; ++t) {
            // rows this step must leave valid: one less per side and step
            const int grow = kb - 1 - t;
            double m = -1.0;
            unsigned int key = RES_NO_KEY;
            if (y + NR > max(ty0 - grow, 0) && y < min(ty1 + grow, ny)) {
                double up[V], dn[V], cf[V];
                res_lds<V>(up, &s_seam[buf][max(wid - 1, 0)][NR > 1 ? 1 : 0][V * lane]);
                res_lds<V>(dn, &s_seam[buf][min(wid + 1, RES_WARPS - 1)][0][V * lane]);
                if (edge_y && c.bc == 0) {
                    // mirror edges: the first and last row see themselves.  The
                    // row past the field's end may lie inside this warp: it is
                    // no use, so it can hold the copy
                    if (y == 0) {
#pragma unroll
                        for (int v = 0; v < V; ++v) up[v] = T[0][v];
                    }
                    if (y + NR == ny) {
#pragma unroll
                        for (int v = 0; v < V; ++v) dn[v] = T[NR - 1][v];
                    }
#pragma unroll
                    for (int i = 0; i + 1 < NR; ++i) {
                        if (y + i == ny - 1) {
#pragma unroll
                            for (int v = 0; v < V; ++v) T[i + 1][v] = T[i][v];
                        }
                        if (y + i + 1 == 0) {
#pragma unroll
                            for (int v = 0; v < V; ++v) T[i][v] = T[i + 1][v];
                        }
                    }
                }
                if (src) {
                    res_lds<V>(cf, colf + t * COLS + V * lane);
                    res_step_rows<V, NR, MODE, true>(T, up, dn, rowf + t * ROWS + NR * wid, cf, h,
                                                     c, first_col, last_col);
                } else {
                    res_step_rows<V, NR, MODE, false>(T, up, dn, nullptr, cf, h, c, first_col,
                                                      last_col);
                }
                if (c.bc == 1 && (edge_x || edge_y)) {
#pragma unroll
                    for (int i = 0; i < NR; ++i)
#pragma unroll
                        for (int v = 0; v < V; ++v)
                            if (y + i == 0 || y + i == ny - 1 || x + v == 0 || x + v == nx - 1)
                                T[i][v] = c.T_edge;
                }
                if (ragged) ghost_cols();
                res_sts<V>(&s_seam[buf ^ 1][wid][0][V * lane], T[0]);
                if constexpr (NR > 1) res_sts<V>(&s_seam[buf ^ 1][wid][1][V * lane], T[NR - 1]);
                if constexpr (REDUCE) {
                    // owned rows [oa, ob) of this warp
                    const int oa = max(ty0 - y, 0), ob = min(ty1 - y, NR);
                    bool hot = false, nan = false;
                    double rm[NR];
                    unsigned int rk[NR];
#pragma unroll
                    for (int i = 0; i < NR; ++i) {
                        // a row's first maximum (strict '>': the smaller
                        // column) pairwise, so that compares chain log V deep
                        double w[V];
                        unsigned int wk[V];
#pragma unroll
                        for (int v = 0; v < V; ++v) {
                            w[v] = T[i][v];
                            wk[v] = (unsigned)v;
                        }
#pragma unroll
                        for (int s = 1; s < V; s *= 2)
#pragma unroll
                            for (int v = 0; v + s < V; v += 2 * s) {
                                // a pair's left cell, NaN, has hidden the right
                                // one; only in place 0 does it show at the end
                                if (s > 1) nan |= isnan(w[v + s]);
                                const bool g = w[v + s] > w[v];
                                w[v] = g ? w[v + s] : w[v];
                                wk[v] = g ? wk[v + s] : wk[v];
                            }
                        rm[i] = own_x && i >= oa && i < ob ? w[0] : -INFINITY;
                        rk[i] = wk[0] + ((unsigned)i << RES_KEY_SHIFT);
                        hot |= !(rm[i] <= c.Tm);
                    }
                    if (__any_sync(0xffffffffu, hot || nan)) {
                        // a molten row, or one whose maximum met a NaN (NaN
                        // never wins: such a row is scanned again without it)
                        unsigned int rows = 0u;
#pragma unroll
                        for (int i = 0; i < NR; ++i) {
                            if (isnan(rm[i]) || (nan && own_x && i >= oa && i < ob)) {
                                rm[i] = -INFINITY;
#pragma unroll
                                for (int v = 0; v < V; ++v)
                                    if (T[i][v] > rm[i]) {
                                        rm[i] = T[i][v];
                                        rk[i] = (unsigned)v + ((unsigned)i << RES_KEY_SHIFT);
                                    }
                            }
                            rows |= rm[i] > c.Tm ? 1u << i : 0u;
                        }
                        rows = __reduce_or_sync(0xffffffffu, rows);
                        if (lane == 0 && rows) {
                            atomicMin(&s_mn[t], y + __ffs(rows) - 1);
                            atomicMax(&s_mx[t], y + 31 - __clz(rows));
                        }
                    }
#pragma unroll
                    for (int s = 1; s < NR; s *= 2)
#pragma unroll
                        for (int i = 0; i + s < NR; i += 2 * s) {
                            const bool g = rm[i + s] > rm[i];
                            rm[i] = g ? rm[i + s] : rm[i];
                            rk[i] = g ? rk[i + s] : rk[i];
                        }
                    if (rm[0] > -1.0) {
                        m = rm[0];
                        key = rk[0] + ((unsigned)(NR * wid) << RES_KEY_SHIFT) +
                              (unsigned)(V * lane);
                    }
                }
            }
            if constexpr (REDUCE) {
                recm[t * RES_THREADS + tid] = m;
                reck[t * RES_THREADS + tid] = key;
            }
            buf ^= 1;
            __syncthreads();
        }

        const bool last = b == p.nblocks;
        const int s2 = last ? s1 : res_step(b + 1, p.nblocks, p.n_steps);
        const int kn = s2 - s1;              // the next block's halo
        {
            // the rim, as wide as the next block's halo, or the whole tile.  A
            // NaN or infinite cell stays or turns NaN and is still there now:
            // one look per launch flags it.
            double* X = last ? p.Tout : p.xbuf[b & 1];
            const int w = last ? 1 << 30 : kn;
            bool bad = false;
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                const int yy = y + i;
                if (yy < ty0 || yy >= ty1) continue;
                const bool whole = yy - ty0 < w || ty1 - yy <= w;
                double* dst = X + (size_t)yy * nx + x;
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    const int xx = x + v;
                    if (own_x && xx < nx && (whole || xx - tx0 < w || tx1 - xx <= w)) {
                        __stcg(dst + v, T[i][v]);
                        if (REDUCE && last) bad |= !(fabs(T[i][v]) < INFINITY);
                    }
                }
            }
            if (bad) atomicOr(p.err, 2u);
        }
        if (!last) {
            if (tid == 0) s_flag = 1;
            __syncthreads();
            // the release is cumulative over the barrier: the CTA's rim first
            if (tid == 0) st_release(p.flags + blockIdx.x * RES_FLAG_STRIDE, (unsigned)b);
        }
        if constexpr (REDUCE) {
            // this CTA's Partial of each step of the block, one warp per step
            for (int t = wid; t < kb; t += RES_WARPS) {
                double m = -1.0;
                unsigned int key = RES_NO_KEY;
                // warps hold rows in order: strict '>' keeps the first maximum
#pragma unroll
                for (int j = 0; j < RES_WARPS; ++j) {
                    const double mj = recm[t * RES_THREADS + 32 * j + lane];
                    const unsigned int kj = reck[t * RES_THREADS + 32 * j + lane];
                    const bool g = mj > m;
                    m = g ? mj : m;
                    key = g ? kj : key;
                }
                res_warp_max(m, key);
                if (lane == 0) {
                    const bool none = key == RES_NO_KEY;
                    const int row = (int)(key >> RES_KEY_SHIFT) + py0;
                    const int col = (int)(key & ((1u << RES_KEY_SHIFT) - 1u)) + px0;
                    const int mx = s_mx[t];
                    Partial out;
                    out.tmax = m;
                    out.arg = none ? (long long)nx * ny : (long long)row * nx + col;
                    out.ymin = mx < 0 ? ny : s_mn[t];
                    out.ymax = mx;
                    p.scratch[(size_t)(s0 + t) * gridDim.x + blockIdx.x] = out;
                    s_mn[t] = 0x7fffffff;          // for the next block
                    s_mx[t] = -1;
                }
            }
        }
        if (last) break;
        factors(s1, kn);                     // while the neighbours' rims are on their way
        if (tid < 9 && tid != 4) {
            const int ox = bx + tid % 3 - 1, oy = by + tid / 3 - 1;
            if (ox >= 0 && ox < p.gx && oy >= 0 && oy < p.gy &&
                !res_wait(p.flags + (oy * p.gx + ox) * RES_FLAG_STRIDE, (unsigned)b, p.wait_ns))
                s_flag = 0;
        }
        src = __syncthreads_or(any_row);
        if (!s_flag) {
            // let the neighbours run on (their field is flagged incomplete
            // too) instead of each waiting out its own limit
            if (tid == 0) st_release(p.flags + blockIdx.x * RES_FLAG_STRIDE, 0x7fffffffu);
            failed = true;
            break;
        }
        {
            const double* X = p.xbuf[b & 1];
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                const int yy = y + i;
                if (yy < max(ty0 - kn, 0) || yy >= min(ty1 + kn, ny)) continue;
                const bool inner = yy >= ty0 && yy < ty1;
                const double* row = X + (size_t)yy * nx + x;
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    const int xx = x + v;
                    if (xx >= max(tx0 - kn, 0) && xx < min(tx1 + kn, nx) && !(inner && own_x))
                        T[i][v] = __ldcg(row + v);
                }
            }
        }
        src = __syncthreads_or(any_col) && src;
        s0 = s1;
        s1 = s2;
    }

    if (failed && tid == 0) atomicOr(p.err, 1u);
    if constexpr (REDUCE) {
        // every CTA's Partials are written: fold the steps over the CTAs
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            atomicAdd(p.barrier, 1u);
            s_flag = failed ? 0 : (res_wait(p.barrier, gridDim.x, p.wait_ns) ? 1 : 0);
            if (!s_flag) atomicOr(p.err, 1u);
        }
        __syncthreads();
        if (s_flag) {
            const long long N = (long long)nx * ny;
            for (int s = blockIdx.x + (int)gridDim.x * wid; s < p.n_steps;
                 s += (int)gridDim.x * RES_WARPS) {
                double tm = -1.0; long long ag = N; int mn = ny, mx = -1;
                const Partial* q = p.scratch + (size_t)s * gridDim.x;
                for (int i = lane; i < (int)gridDim.x; i += 32)
                    partial_take(tm, ag, mn, mx, __ldcg(&q[i].tmax), __ldcg(&q[i].arg),
                                 __ldcg(&q[i].ymin), __ldcg(&q[i].ymax));
                partial_warp_reduce(tm, ag, mn, mx);
                if (lane == 0) p.ring[s] = Partial{tm, ag, mn, mx};
            }
        }
    }
    // the last CTA to leave re-arms flags and counters for the next launch
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        s_flag = atomicAdd(p.counter, 1u) == gridDim.x - 1 ? 1 : 0;
    }
    __syncthreads();
    if (s_flag) {
        for (int i = tid; i < (int)gridDim.x; i += RES_THREADS) p.flags[i * RES_FLAG_STRIDE] = 0u;
        if (tid == 0) { *p.counter = 0u; *p.barrier = 0u; }
    }
}

}  // namespace lpbf_b200
