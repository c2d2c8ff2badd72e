// SPDX-License-Identifier: 0BSD
// ---------------------------------------------------------------------------
// FP32 compensated variant of the temporally blocked step.
//
// The field is held as two f32 arrays, hi and lo, with the temperature
// T = hi + lo (lo the rounding remainder of hi, |lo| <= ulp(hi)/2).  Per cell
// and step:
//   * neighbour differences are formed on the pairs,
//       (R - T) = (R.hi - T.hi) + (R.lo - T.lo),
//     the hi difference being exact for neighbours within a factor of two,
//     so the Laplacian keeps ~48 significant bits;
//   * the loss terms and the increment are f32; the Gaussian source is
//     evaluated in FP64 (as in the FP64 path) and rounded once;
//   * the increment is added with an error-free sum (Fast2Sum: the
//     increment is never larger than T), and the rounding error is carried
//     in lo (Kahan-compensated accumulation).
// Memory traffic per cell-update equals the FP64 path's (hi + lo = 8 bytes).
//
// Structure (warp tasks, lanes, TMA pipeline, wavefront, fast/general boxes,
// two-tier reduction) follows lpbf_advance.cuh; the per-step Partials are
// computed on T = (double)hi + (double)lo, which is exact.
//
// The same kernel with COMP = false is the plain FP32 field: one f32 array,
// each step's update rounded once (the FP64 step's fused form in f32, the
// source still evaluated in FP64), 8 bytes per cell-update; no lo array is
// loaded, staged, shuffled or stored.
// ---------------------------------------------------------------------------
#pragma once
#include <stddef.h>

#include <cstring>

#include "lpbf_advance.cuh"

namespace lpbf_b200 {

// floats per TMA stage: the hi box, then (compensated field) the lo box
template <bool COMP>
constexpr int fk_stage_floats() { return (COMP ? 2 : 1) * ADV_R * ADV_COLS; }
template <bool COMP>
constexpr size_t fk_smem_bytes() {
    return size_t(ADV_WARPS) * ADV_S * fk_stage_floats<COMP>() * sizeof(float)
           + size_t(ADV_WARPS) * ADV_S * sizeof(uint64_t);
}

// 16-byte store issued under a predicate (no branch), without a "memory"
// clobber: the kernel never reads the destination field back.
__device__ __forceinline__ void st_global_v4f_pred(float* p, const float* v, bool pred) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t"
                 "@q st.global.v4.f32 [%0], {%1, %2, %3, %4};\n\t}"
                 :: "l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"((int)pred));
}

// These kernels are bound by instruction issue, so the fast body holds and
// updates its four cells per lane as two pairs; only what needs a neighbour
// across a pair's seam stays scalar (the horizontal differences and sums,
// whose results land in pairs).
inline p2 p2_host(float v) {            // both halves v
    unsigned int b;
    std::memcpy(&b, &v, sizeof(b));
    return ((p2)b << 32) | b;
}

// FkCoef's constants as pairs, the loss coefficients negated (rounding is
// symmetric: the fast body adds -loss).
struct FkCoef2 {
    p2 ax, ay, ncls, ncrad, nTa4, clsTa, Ta_hi, Ta_lo, m4, m2;
};

// 16-byte store of two pairs issued under a predicate, as st_global_v4f_pred.
__device__ __forceinline__ void st_global_v2_pred(float* p, const p2* v, bool pred) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %3, 0;\n\t"
                 "@q st.global.v2.b64 [%0], {%1, %2};\n\t}"
                 :: "l"(p), "l"(v[0]), "l"(v[1]), "r"((int)pred));
}

struct FkCoef {
    float ax, ay, cls, crad;
    float Ta_hi, Ta_lo, Ta4;       // linear-loss reference T as a pair; Ta4 = f4(Tamb)
    float Tedge_hi, Tedge_lo;
    float clsTa;                   // c_ls * (linear-loss reference T), rounded once
};

struct FkParams {
    Coef c;                        // geometry, source and reduction constants
    FkCoef f;
    FkCoef2 f2;
    LaserSub las[KMAX];
    int band_lo, band_hi, bandx_lo, bandx_hi;
    int nstrips, nchunks, H, ntasks;
    int nA, nB, Hb, Ya, Yb;        // band-split chunks, as in AdvParams
    float* Thi_out;
    float* Tlo_out;
    Partial* ring;
    Partial* scratch;
    unsigned int* counter;
    unsigned int* tasks;
    unsigned int* err;
};

// T^4 of a pair, in f32 (the same expression for cells and for Tamb, so the
// radiation difference is exactly zero at equilibrium).
__device__ __host__ __forceinline__ float fk_pow4(float hi, float lo) {
    const float t = hi + lo;
    const float t2 = t * t;
    return t2 * t2;
}

// One compensated cell update.  (th, tl) centre; neighbour pairs; S_dt the
// dt-scaled FP64 source rounded to f32.  SQ (ax == ay): one Laplacian of the
// hi parts plus one of the lo parts, the source and loss in the same fused
// chain; otherwise the x and y terms apart.  T^4 - Ta^4 is one fused
// multiply-add.
template <bool SQ>
__device__ __forceinline__ void fk_cell(float th, float tl, float Lh, float Ll, float Rh,
                                        float Rl, float Uh, float Ul, float Dh, float Dl,
                                        float S, const FkCoef& f, float& oh, float& ol) {
    const float da = __fsub_rn(th, f.Ta_hi) + (tl - f.Ta_lo);
    const float t = th + tl;
    const float t2 = t * t;
    const float e4 = fmaf(t2, t2, -f.Ta4);
    const float loss = fmaf(f.crad, e4, __fmul_rn(f.cls, da));
    float d;
    if constexpr (SQ) {
        const float lh = (__fsub_rn(Rh, th) + __fsub_rn(Lh, th)) +
                         (__fsub_rn(Dh, th) + __fsub_rn(Uh, th));
        const float ll = fmaf(-4.0f, tl, (Rl + Ll) + (Dl + Ul));
        d = fmaf(f.ax, lh + ll, __fsub_rn(S, loss));
    } else {
        const float lx = ((__fsub_rn(Rh, th) + __fsub_rn(Lh, th)) + ((Rl - tl) + (Ll - tl)));
        const float ly = ((__fsub_rn(Dh, th) + __fsub_rn(Uh, th)) + ((Dl - tl) + (Ul - tl)));
        d = fmaf(f.ax, lx, fmaf(f.ay, ly, __fsub_rn(S, loss)));
    }
    // th + d with its rounding error (Fast2Sum, exact for |d| <= |th|: a
    // step's increment is far smaller than the temperature), the error
    // folded into lo, then renormalised
    const float s = __fadd_rn(th, d);
    const float err = __fsub_rn(d, __fsub_rn(s, th));
    const float lo = __fadd_rn(tl, err);
    oh = __fadd_rn(s, lo);
    ol = __fsub_rn(lo, __fsub_rn(oh, s));
}

// One plain f32 cell update: the FP64 step's form in f32.  T^4 - Ta^4 and
// c_ls T - c_ls Ta are each one fused multiply-add and the loss enters the
// increment's fused chain (SQ: one Laplacian (R + L) + (U + D) - 4T).  The
// Laplacian of a uniform field is exactly zero and its loss at Tamb far below
// half an ulp of T, so a uniform field at Tamb stays exactly uniform.
// The cell's source increment S is added to the net change before T.
template <bool SQ>
__device__ __forceinline__ float f32_cell(float t, float L, float R, float U, float D, float S,
                                          const FkCoef& f) {
    const float t2 = __fmul_rn(t, t);
    const float e4 = fmaf(t2, t2, -f.Ta4);
    const float loss = fmaf(f.crad, e4, fmaf(f.cls, t, -f.clsTa));
    float net;
    if constexpr (SQ) {
        const float lap = fmaf(-4.0f, t, __fadd_rn(__fadd_rn(R, L), __fadd_rn(U, D)));
        net = fmaf(f.ax, lap, -loss);
    } else {
        const float lx = fmaf(-2.0f, t, __fadd_rn(R, L));
        const float ly = fmaf(-2.0f, t, __fadd_rn(U, D));
        net = fmaf(f.ax, lx, fmaf(f.ay, ly, -loss));
    }
    return __fadd_rn(t, __fadd_rn(net, S));
}

// (a.hi, a.lo) > (b.hi, b.lo) for canonical pairs.
__device__ __forceinline__ bool fk_gt(float ah, float al, float bh, float bl) {
    return ah > bh || (ah == bh && al > bl);
}

template <int K, bool REDUCE, bool SQ, bool COMP>
struct FkStrip {
    static constexpr int V = ADV_V;
    static constexpr int STAGE = fk_stage_floats<COMP>();

    const FkParams& p;
    const CUtensorMap* map_hi;
    const CUtensorMap* map_lo;
    float* stages;
    uint64_t* bars;
    uint32_t gbox;
    const int lane;

    int x0, xs, xl, y0, y1, jy0, jend, nbox, issued;
    bool edge, failed, own_all;
    bool src_task;                     // rows the task depends on meet the source
    bool first_col, last_col;          // the lane holds the field's first / last column (mirror)
    double rowf;                       // this box's row factors of the source (as WarpStrip)
    double* colf;                      // the task's column factors, four per level

    p2 wh0[3][2], wl0[3][2];           // windows: a lane's four cells as two pairs
    p2 wh[K > 1 ? K - 1 : 1][3][2], wl[K > 1 ? K - 1 : 1][3][2];
    float thr_h[K], thr_l[K];
    bool hit[K];
    unsigned kmask;                    // last-level rows of this box in s_box
    double (*s_tmx)[32];
    long long (*s_arg)[32];
    int* s_ymn;
    int* s_ymx;
    float (*s_box)[32][2 * ADV_V];     // [3][32][hi0..3, lo0..3]

    __device__ __forceinline__ FkStrip(const FkParams& p_, const CUtensorMap* mh,
                                       const CUtensorMap* ml, float* st, uint64_t* b, int ln,
                                       double (*tm)[32], long long (*ar)[32], int* mn, int* mx,
                                       float (*bx)[32][2 * ADV_V])
        : p(p_), map_hi(mh), map_lo(ml), stages(st), bars(b), gbox(0), lane(ln), failed(false), kmask(0u),
          s_tmx(tm), s_arg(ar), s_ymn(mn), s_ymx(mx), s_box(bx) {
        if constexpr (REDUCE) {
            const long long N = (long long)p.c.nx * p.c.ny;
#pragma unroll
            for (int t = 0; t < K; ++t) {
                hit[t] = false;
                s_tmx[t][lane] = -1.0;
                s_arg[t][lane] = N;
                if (lane == 0) { s_ymn[t] = p.c.ny; s_ymx[t] = -1; }
            }
        }
        __syncwarp();
    }

    __device__ __forceinline__ void issue(int b) {
        const uint32_t g = gbox + b;
        const int st = g % ADV_S;
        float* dst = stages + st * STAGE;
        mbar_expect_tx(&bars[st], STAGE * sizeof(float));
        tma_load_2d(dst, map_hi, xs, jy0 + b * ADV_R, &bars[st]);
        if constexpr (COMP)
            tma_load_2d(dst + ADV_R * ADV_COLS, map_lo, xs, jy0 + b * ADV_R, &bars[st]);
        issued = b + 1;
    }

    __device__ __forceinline__ bool owned_lane() const {
        return xl >= x0 && xl < x0 + ADV_WOUT && xl < p.c.nx;
    }

    __device__ __noinline__ static void columns_to(double* out, int xl, const FkParams& p) {
#pragma unroll 1
        for (int t = 0; t < K; ++t) {
            const double4 f = src_columns(xl, p.las[t].x_l, p.c.dx, p.c.m2r, p.c.r2_cut);
            out[t * V] = f.x; out[t * V + 1] = f.y; out[t * V + 2] = f.z; out[t * V + 3] = f.w;
        }
    }

    __device__ __forceinline__ void run_task(int task) {
        double cols[K * V];
        colf = cols;
        rowf = 0.0;
        const int nx = p.c.nx, ny = p.c.ny;
        const int strip = task % p.nstrips, chunk = task / p.nstrips;
        x0 = strip * ADV_WOUT;
        xs = x0 - ADV_KH;
        xl = xs + 4 * lane;
        if (chunk < p.nA) {
            y0 = chunk * p.H;
            y1 = y0 + p.H;
        } else if (chunk < p.nA + p.nB) {
            y0 = p.Ya + (chunk - p.nA) * p.Hb;
            y1 = min(y0 + p.Hb, p.Yb);
        } else {
            y0 = p.Yb + (chunk - p.nA - p.nB) * p.H;
            y1 = min(y0 + p.H, ny);
        }
        jy0 = max(y0 - K, 0);
        jy0 -= jy0 % 3;
        jend = min(y1 + K, ny);
        nbox = (jend - jy0 + ADV_R - 1) / ADV_R;
        edge = (xs <= 0) || (xs + ADV_COLS > nx - 1);
        // one condition for the column factors and for the boxes that read them:
        // rows y0 - K .. y1 + K are all that an owned row depends on
        src_task = !(xs + ADV_COLS <= p.bandx_lo || xs > p.bandx_hi) &&
                   y0 - K <= p.band_hi && y1 + K >= p.band_lo;
        own_all = owned_lane();            // nx is a multiple of 4: whole lanes
        first_col = p.c.bc == 0 && xl == 0;
        last_col = p.c.bc == 0 && xl + V == nx;
        issued = 0;
        if (lane == 0) {
            const int pre = min(ADV_S, nbox);
            for (int b = 0; b < pre; ++b) issue(b);
        }
        const int jlast = y1 - 1 + K;
        if (src_task) columns_to(colf, xl, p);
        // per-box thresholds change only when an exact pass moves a peak
        if constexpr (REDUCE) set_thresholds();
        for (int b = 0, j = jy0; j <= jlast && !failed; ++b, j += ADV_R) {
            const float* st = nullptr;
            if (j < jend) {
                const uint32_t g = gbox + b;
                const int sidx = g % ADV_S;
                const bool ok = mbar_wait_bounded(&bars[sidx], (g / ADV_S) & 1);
                if (!__all_sync(0xffffffffu, ok)) {
                    if (lane == 0) atomicOr(p.err, 1u);
                    failed = true;
                    break;
                }
                st = stages + sidx * STAGE;
            }
            // mirror-edge strips too: row_update patches the edge cells'
            // outer neighbours itself (nx a multiple of 4: whole lanes)
            const bool src_box = src_task && j + 1 >= p.band_lo && j - K <= p.band_hi;
            const bool fast = (!edge || (p.c.bc == 0 && (p.c.nx & 3) == 0)) &&
                              j - K >= 1 && j + 1 <= ny - 2 && j < jend;
            rowf = 0.0;
            if (src_box) {
                const int t = min(lane / 3, K - 1);
                rowf = src_row(j + lane % 3 - (t + 1), p.las[t], p.c);
            }
            if (fast && !src_box) {
                fast_row<0, false>(j, st);
                fast_row<1, false>(j + 1, st);
                fast_row<2, false>(j + 2, st);
            } else if (fast) {
                fast_row<0, true>(j, st);
                fast_row<1, true>(j + 1, st);
                fast_row<2, true>(j + 2, st);
            } else {
                general_row<0>(j, st, jlast);
                general_row<1>(j + 1, st, jlast);
                general_row<2>(j + 2, st, jlast);
            }
            if constexpr (REDUCE) resolve_box(j);
            if (j < jend) {
                __syncwarp();
                if (lane == 0 && b + ADV_S < nbox) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    issue(b + ADV_S);
                }
            }
        }
        if (failed) {
            const int last = __shfl_sync(0xffffffffu, issued, 0);
            for (int b = max(0, last - ADV_S); b < last; ++b) {
                const uint32_t g = gbox + b;
                mbar_wait_bounded(&bars[g % ADV_S], (g / ADV_S) & 1);
            }
        }
        gbox += nbox;
    }

    template <int P>
    __device__ __forceinline__ void load_row0(const float* st) {
        const ulonglong2 h = *reinterpret_cast<const ulonglong2*>(st + P * ADV_COLS + 4 * lane);
        wh0[P][0] = h.x; wh0[P][1] = h.y;
        if constexpr (COMP) {
            const ulonglong2 l =
                *reinterpret_cast<const ulonglong2*>(st + (ADV_R + P) * ADV_COLS + 4 * lane);
            wl0[P][0] = l.x; wl0[P][1] = l.y;
        }
    }

    template <int T>
    __device__ __forceinline__ p2 (&winh())[3][2] {
        if constexpr (T == 0) return wh0; else return wh[T - 1];
    }
    template <int T>
    __device__ __forceinline__ p2 (&winl())[3][2] {
        if constexpr (T == 0) return wl0; else return wl[T - 1];
    }

    __device__ __forceinline__ static void unpack(const p2* w, float* d) {
        d[0] = p2_a(w[0]); d[1] = p2_b(w[0]); d[2] = p2_a(w[1]); d[3] = p2_b(w[1]);
    }

    // One row of level T from the three rows (up, centre, down) of level T-1
    // (plain field: the lo rows are not read and ol is not written).
    __device__ __forceinline__ void row_update(const float* uh, const float* ul, const float* ch,
                                               const float* cl, const float* dh, const float* dl,
                                               const float* S, float* oh, float* ol) {
        if constexpr (!COMP) {
            const float L0 = __shfl_up_sync(0xffffffffu, ch[V - 1], 1);
            const float R3 = __shfl_down_sync(0xffffffffu, ch[0], 1);
            float L[V] = {L0, ch[0], ch[1], ch[2]};
            float R[V] = {ch[1], ch[2], ch[3], R3};
            if (edge) {
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    if (xl + v == 0) L[v] = ch[v];
                    if (xl + v == p.c.nx - 1) R[v] = ch[v];
                }
            }
#pragma unroll
            for (int v = 0; v < V; ++v)
                oh[v] = f32_cell<SQ>(ch[v], L[v], R[v], uh[v], dh[v], S[v], p.f);
        } else {
            const float Lh0 = __shfl_up_sync(0xffffffffu, ch[V - 1], 1);
            const float Ll0 = __shfl_up_sync(0xffffffffu, cl[V - 1], 1);
            const float Rh3 = __shfl_down_sync(0xffffffffu, ch[0], 1);
            const float Rl3 = __shfl_down_sync(0xffffffffu, cl[0], 1);
            float Lh[V] = {Lh0, ch[0], ch[1], ch[2]}, Ll[V] = {Ll0, cl[0], cl[1], cl[2]};
            float Rh[V] = {ch[1], ch[2], ch[3], Rh3}, Rl[V] = {cl[1], cl[2], cl[3], Rl3};
            if (edge) {
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    if (xl + v == 0) { Lh[v] = ch[v]; Ll[v] = cl[v]; }
                    if (xl + v == p.c.nx - 1) { Rh[v] = ch[v]; Rl[v] = cl[v]; }
                }
            }
#pragma unroll
            for (int v = 0; v < V; ++v)
                fk_cell<SQ>(ch[v], cl[v], Lh[v], Ll[v], Rh[v], Rl[v], uh[v], ul[v], dh[v],
                            dl[v], S[v], p.f, oh[v], ol[v]);
        }
    }

    // One row of level T from the packed rows of level T-1 (interior and
    // mirror-edge lanes): the scalar cell functions' operations in their
    // order, two cells per instruction.  SRC: with the source increments S.
    template <bool SRC>
    __device__ __forceinline__ void fast_update(const p2* uh, const p2* ul, const p2* ch,
                                                const p2* cl, const p2* dh, const p2* dl,
                                                const p2* S, p2* oh, p2* ol) {
        const FkCoef2& f = p.f2;
        const float h0 = p2_a(ch[0]), h1 = p2_b(ch[0]), h2 = p2_a(ch[1]), h3 = p2_b(ch[1]);
        float Lo = __shfl_up_sync(0xffffffffu, h3, 1);
        float Ro = __shfl_down_sync(0xffffffffu, h0, 1);
        Lo = first_col ? h0 : Lo;
        Ro = last_col ? h3 : Ro;
        if constexpr (!COMP) {
            const p2 rl[2] = {p2_pack(__fadd_rn(h1, Lo), __fadd_rn(h2, h0)),
                              p2_pack(__fadd_rn(h3, h1), __fadd_rn(Ro, h2))};
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const p2 t = ch[q];
                const p2 t2 = p2_mul(t, t);
                const p2 e4 = p2_fma(t2, t2, f.nTa4);
                const p2 nloss = p2_fma(f.ncrad, e4, p2_fma(f.ncls, t, f.clsTa));
                p2 net;
                if constexpr (SQ) {
                    const p2 lap = p2_fma(f.m4, t, p2_add(rl[q], p2_add(uh[q], dh[q])));
                    net = p2_fma(f.ax, lap, nloss);
                } else {
                    const p2 lx = p2_fma(f.m2, t, rl[q]);
                    const p2 ly = p2_fma(f.m2, t, p2_add(uh[q], dh[q]));
                    net = p2_fma(f.ax, lx, p2_fma(f.ay, ly, nloss));
                }
                if constexpr (SRC) net = p2_add(net, S[q]);
                oh[q] = p2_add(t, net);
            }
        } else {
            const float l0 = p2_a(cl[0]), l1 = p2_b(cl[0]), l2 = p2_a(cl[1]), l3 = p2_b(cl[1]);
            float Ll = __shfl_up_sync(0xffffffffu, l3, 1);
            float Rl = __shfl_down_sync(0xffffffffu, l0, 1);
            Ll = first_col ? l0 : Ll;
            Rl = last_col ? l3 : Rl;
            // differences across the lane's faces: a cell's left difference is
            // its left neighbour's right one, negated
            const float a0 = __fsub_rn(h0, Lo), a1 = __fsub_rn(h1, h0), a2 = __fsub_rn(h2, h1),
                        a3 = __fsub_rn(h3, h2), a4 = __fsub_rn(Ro, h3);
            const p2 hx[2] = {p2_pack(__fsub_rn(a1, a0), __fsub_rn(a2, a1)),
                              p2_pack(__fsub_rn(a3, a2), __fsub_rn(a4, a3))};
            p2 lx[2];
            if constexpr (SQ) {
                lx[0] = p2_pack(__fadd_rn(l1, Ll), __fadd_rn(l2, l0));
                lx[1] = p2_pack(__fadd_rn(l3, l1), __fadd_rn(Rl, l2));
            } else {
                const float b0 = __fsub_rn(l0, Ll), b1 = __fsub_rn(l1, l0), b2 = __fsub_rn(l2, l1),
                            b3 = __fsub_rn(l3, l2), b4 = __fsub_rn(Rl, l3);
                lx[0] = p2_pack(__fsub_rn(b1, b0), __fsub_rn(b2, b1));
                lx[1] = p2_pack(__fsub_rn(b3, b2), __fsub_rn(b4, b3));
            }
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const p2 th = ch[q], tl = cl[q];
                const p2 da = p2_add(p2_sub(th, f.Ta_hi), p2_sub(tl, f.Ta_lo));
                const p2 t = p2_add(th, tl);
                const p2 t2 = p2_mul(t, t);
                const p2 e4 = p2_fma(t2, t2, f.nTa4);
                p2 nloss = p2_fma(f.ncrad, e4, p2_mul(f.ncls, da));
                if constexpr (SRC) nloss = p2_add(S[q], nloss);
                const p2 hy = p2_add(p2_sub(dh[q], th), p2_sub(uh[q], th));
                p2 d;
                if constexpr (SQ) {
                    const p2 lh = p2_add(hx[q], hy);
                    const p2 ll = p2_fma(f.m4, tl, p2_add(lx[q], p2_add(dl[q], ul[q])));
                    d = p2_fma(f.ax, p2_add(lh, ll), nloss);
                } else {
                    const p2 dx = p2_add(hx[q], lx[q]);
                    const p2 dy = p2_add(hy, p2_add(p2_sub(dl[q], tl), p2_sub(ul[q], tl)));
                    d = p2_fma(f.ax, dx, p2_fma(f.ay, dy, nloss));
                }
                const p2 sum = p2_add(th, d);
                const p2 err = p2_sub(d, p2_sub(sum, th));
                const p2 lo = p2_add(tl, err);
                oh[q] = p2_add(sum, lo);
                ol[q] = p2_sub(lo, p2_sub(oh[q], sum));
            }
        }
    }

    template <int P, bool SRC>
    __device__ __forceinline__ void fast_row(int jj, const float* st) {
        load_row0<P>(st);
        fast_level<P, 1, SRC>(jj);
    }

    template <int P, int T, bool SRC>
    __device__ __forceinline__ void fast_level(int jj) {
        if constexpr (T <= K) {
            constexpr int su = mod3(P - T - 1), sc = mod3(P - T), sd = mod3(P - T + 1);
            p2 (&ah)[3][2] = winh<T - 1>();
            p2 (&al)[3][2] = winl<T - 1>();
            p2 oh[2], ol[2], S[2];
            if constexpr (SRC) {
                __syncwarp();              // bounds the interleaving of levels (registers)
                const double rf = __shfl_sync(0xffffffffu, rowf, 3 * (T - 1) + P);
                const double* cf = colf + (T - 1) * V;
                S[0] = p2_pack((float)src_product(rf, cf[0]), (float)src_product(rf, cf[1]));
                S[1] = p2_pack((float)src_product(rf, cf[2]), (float)src_product(rf, cf[3]));
            }
            fast_update<SRC>(ah[su], al[su], ah[sc], al[sc], ah[sd], al[sd], S, oh, ol);
            const int r = jj - T;
            const bool own = own_all && r >= y0 && r < y1;
            if constexpr (T < K) {
                p2 (&bh)[3][2] = winh<T>();
                bh[sc][0] = oh[0]; bh[sc][1] = oh[1];
                if constexpr (COMP) {
                    p2 (&bl)[3][2] = winl<T>();
                    bl[sc][0] = ol[0]; bl[sc][1] = ol[1];
                }
            } else {
                const size_t off = (size_t)r * p.c.nx + xl;
                st_global_v2_pred(p.Thi_out + off, oh, own);
                if constexpr (COMP) st_global_v2_pred(p.Tlo_out + off, ol, own);
            }
            if constexpr (REDUCE) {
                // the largest of the four cells against the box threshold (NaN
                // never wins a maximum); pairs by the sign of their difference.
                // Its lo part is rounded up: where it all but cancels a step of
                // hi, a cell above the threshold must not come out equal to it
                // (one just below may pass: the exact pass decides)
                const float th = own ? thr_h[T - 1] : INFINITY;
                bool rh;
                if constexpr (COMP) {
                    const p2 tp = p2_pack(th, th), tq = p2_pack(thr_l[T - 1], thr_l[T - 1]);
                    const p2 e0 = p2_add(p2_sub(oh[0], tp), p2_sub_up(ol[0], tq));
                    const p2 e1 = p2_add(p2_sub(oh[1], tp), p2_sub_up(ol[1], tq));
                    rh = fmaxf(fmaxf(p2_a(e0), p2_b(e0)), fmaxf(p2_a(e1), p2_b(e1))) > 0.0f;
                } else {
                    rh = fmaxf(fmaxf(p2_a(oh[0]), p2_b(oh[0])),
                               fmaxf(p2_a(oh[1]), p2_b(oh[1]))) > th;
                }
                hit[T - 1] |= rh;
                if constexpr (T == K) {
                    if (rh) stage_row<P>(oh, ol);
                }
            }
            fast_level<P, T + 1, SRC>(jj);
        }
    }

    template <int P>
    __device__ __forceinline__ void general_row(int jj, const float* st, int jlast) {
        if (jj > jlast) return;
        if (jj < jend) load_row0<P>(st);
        general_level<P, 1>(jj);
    }

    template <int P, int T>
    __device__ __forceinline__ void general_level(int jj) {
        if constexpr (T <= K) {
            constexpr int su = mod3(P - T - 1), sc = mod3(P - T), sd = mod3(P - T + 1);
            const int ny = p.c.ny;
            const int r = jj - T;
            const int lo = max(y0 - K + T, 0);
            const int hi = min(y1 - 1 + K - T, ny - 1);
            if (r >= lo && r <= hi) {
                p2 (&ah)[3][2] = winh<T - 1>();
                p2 (&al)[3][2] = winl<T - 1>();
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (r == 0) {
                        ah[su][q] = ah[sc][q];
                        if constexpr (COMP) al[su][q] = al[sc][q];
                    }
                    if (r == ny - 1) {
                        ah[sd][q] = ah[sc][q];
                        if constexpr (COMP) al[sd][q] = al[sc][q];
                    }
                }
                float oh[V], ol[V];
                if (p.c.bc == 1 && (r == 0 || r == ny - 1)) {
#pragma unroll
                    for (int v = 0; v < V; ++v) { oh[v] = p.f.Tedge_hi; ol[v] = p.f.Tedge_lo; }
                } else {
                    const double rf = __shfl_sync(0xffffffffu, rowf, 3 * (T - 1) + P);
                    float S[V] = {0.f, 0.f, 0.f, 0.f};
                    if (rf != 0.0) {
#pragma unroll
                        for (int v = 0; v < V; ++v)
                            S[v] = (float)src_product(rf, colf[(T - 1) * V + v]);
                    }
                    float uh[V], ul[V], ch[V], cl[V], dh[V], dl[V];
                    unpack(ah[su], uh);
                    unpack(ah[sc], ch);
                    unpack(ah[sd], dh);
                    if constexpr (COMP) {
                        unpack(al[su], ul);
                        unpack(al[sc], cl);
                        unpack(al[sd], dl);
                    }
                    row_update(uh, ul, ch, cl, dh, dl, S, oh, ol);
                    if (edge && p.c.bc == 1) {
#pragma unroll
                        for (int v = 0; v < V; ++v)
                            if (xl + v == 0 || xl + v == p.c.nx - 1) {
                                oh[v] = p.f.Tedge_hi; ol[v] = p.f.Tedge_lo;
                            }
                    }
                }
                finish_level<P, T, sc>(r, oh, ol, r >= y0 && r < y1, !edge);
            }
            general_level<P, T + 1>(jj);
        }
    }

    // Keep the new row in level T's window slot SC (T < K) or store it
    // (T == K), and test it against the box threshold.
    template <int P, int T, int SC>
    __device__ __forceinline__ void finish_level(int r, const float* oh, const float* ol,
                                                 bool owned_row, bool full) {
        if constexpr (T < K) {
            p2 (&bh)[3][2] = winh<T>();
            bh[SC][0] = p2_pack(oh[0], oh[1]);
            bh[SC][1] = p2_pack(oh[2], oh[3]);
            if constexpr (COMP) {
                p2 (&bl)[3][2] = winl<T>();
                bl[SC][0] = p2_pack(ol[0], ol[1]);
                bl[SC][1] = p2_pack(ol[2], ol[3]);
            }
        } else {
            // nx is a multiple of 4 (checked on entry): an owned lane's four
            // cells are in the field and 16-byte aligned; the stores are
            // predicated, so no branch splits the box
            const size_t off = (size_t)r * p.c.nx + xl;
            const bool st = owned_row && owned_lane();
            st_global_v4f_pred(p.Thi_out + off, oh, st);
            if constexpr (COMP) st_global_v4f_pred(p.Tlo_out + off, ol, st);
        }
        if constexpr (REDUCE) {
            bool h = false;
            const bool ol_ok = owned_row && owned_lane();
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const bool ok = ol_ok && (full || xl + v < p.c.nx);
                if constexpr (COMP)
                    h = h | (ok && fk_gt(oh[v], ol[v], thr_h[T - 1], thr_l[T - 1]));
                else
                    h = h | (ok && oh[v] > thr_h[T - 1]);
            }
            hit[T - 1] |= h;
            if constexpr (T == K) {
                if (h) {
                    const p2 ph[2] = {p2_pack(oh[0], oh[1]), p2_pack(oh[2], oh[3])};
                    p2 pl[2] = {0ull, 0ull};
                    if constexpr (COMP) {
                        pl[0] = p2_pack(ol[0], ol[1]);
                        pl[1] = p2_pack(ol[2], ol[3]);
                    }
                    stage_row<P>(ph, pl);
                }
            }
        }
    }

    // ---- two-tier reduction on T = hi + lo ------------------------------
    __device__ __forceinline__ void set_thresholds() {
        const bool ol = owned_lane();
#pragma unroll
        for (int t = 0; t < K; ++t) {
            double a = s_tmx[t][lane];
            a = (a < p.c.Tm) ? a : p.c.Tm;
            if constexpr (COMP) {
                // the largest pair not above a: compare strictly against it
                const float h = (float)a;
                const float l = (float)(a - (double)h);
                thr_h[t] = ol ? h : INFINITY;
                thr_l[t] = ol ? l : 0.0f;
            } else {
                // the largest float not above a: a float cell exceeds it
                // exactly when it exceeds a
                thr_h[t] = ol ? __double2float_rd(a) : INFINITY;
            }
        }
    }

    template <int T>
    __device__ __forceinline__ void stage_level() {
        if constexpr (T >= 1 && T < K) {
#pragma unroll
            for (int P = 0; P < 3; ++P) {
                const int sl = ((P - T) % 3 + 3) % 3;
                p2* d = reinterpret_cast<p2*>(s_box[P][lane]);
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    d[q] = (sl == 0) ? winh<T>()[0][q] : (sl == 1) ? winh<T>()[1][q] : winh<T>()[2][q];
                    if constexpr (COMP)
                        d[2 + q] = (sl == 0) ? winl<T>()[0][q]
                                 : (sl == 1) ? winl<T>()[1][q] : winl<T>()[2][q];
                }
            }
        }
    }

    // A last-level row that crossed its threshold (box row P), for the exact
    // pass: the last level has no register window, and reading the stored
    // row back costs an L2 round trip per box.
    template <int P>
    __device__ __forceinline__ void stage_row(const p2* h, const p2* l) {
        p2* d = reinterpret_cast<p2*>(s_box[P][lane]);
        d[0] = h[0];
        d[1] = h[1];
        if constexpr (COMP) {
            d[2] = l[0];
            d[3] = l[1];
        }
        kmask |= 1u << P;
    }

    // Exact update of level t from the lane's rows in s_box (those of `rows`):
    // its first maximal owned cell in flat-index order and the molten rows.
    __device__ __forceinline__ void exact_level(int t, int j, unsigned rows) {
        const int nx = p.c.nx;
        unsigned molten = 0u;
        double m = -INFINITY;
        int a = -1;
#pragma unroll
        for (int P = 0; P < 3; ++P) {
            const int r = j + P - t;
            const bool cand = ((rows >> P) & 1u) && r >= y0 && r < y1 && own_all;
            const float4 h = *reinterpret_cast<const float4*>(&s_box[P][lane][0]);
            const float hv[V] = {h.x, h.y, h.z, h.w};
            double c[V];
            if constexpr (COMP) {
                const float4 l = *reinterpret_cast<const float4*>(&s_box[P][lane][V]);
                const float lv[V] = {l.x, l.y, l.z, l.w};
#pragma unroll
                for (int v = 0; v < V; ++v) c[v] = (double)hv[v] + (double)lv[v];
            } else {
#pragma unroll
                for (int v = 0; v < V; ++v) c[v] = (double)hv[v];
            }
#pragma unroll
            for (int v = 0; v < V; ++v) {
                molten |= cand && c[v] > p.c.Tm ? 1u << P : 0u;
                c[v] = cand && c[v] > -INFINITY ? c[v] : -INFINITY;      // NaN never wins
            }
            // pairs, then their winners (strict '>': the smaller index)
            const bool h01 = c[1] > c[0], h23 = c[3] > c[2];
            const double m01 = h01 ? c[1] : c[0], m23 = h23 ? c[3] : c[2];
            const bool hh = m23 > m01;
            const double mr = hh ? m23 : m01;
            const int ar = P * V + (hh ? (h23 ? 3 : 2) : (h01 ? 1 : 0));
            a = mr > m ? ar : a;
            m = mr > m ? mr : m;
        }
        molten = __reduce_or_sync(0xffffffffu, molten);
        if (molten && lane == 0) {
            s_ymn[t - 1] = min(s_ymn[t - 1], j - t + __ffs(molten) - 1);
            s_ymx[t - 1] = max(s_ymx[t - 1], j - t + 31 - __clz(molten));
        }
        if (m > s_tmx[t - 1][lane]) {
            s_tmx[t - 1][lane] = m;
            s_arg[t - 1][lane] = (long long)(j + a / V - t) * nx + xl + a % V;
        }
    }

    __device__ __forceinline__ void resolve_box(int j) {
        unsigned bits = 0;
#pragma unroll
        for (int t = 0; t < K; ++t) { bits |= hit[t] ? (1u << t) : 0u; hit[t] = false; }
        bits = __reduce_or_sync(0xffffffffu, bits);
        if (bits == 0u) return;
        // the last level first: its rows sit in s_box, where the others are
        // staged from their windows in turn (a lane reads only its own)
#pragma unroll 1
        for (int t = K; t >= 1; --t) {
            if (!((bits >> (t - 1)) & 1u)) continue;
            switch (t < K ? t : 0) {
                case 1: stage_level<1>(); break;
                case 2: stage_level<2>(); break;
                case 3: stage_level<3>(); break;
                default: break;
            }
            exact_level(t, j, t < K ? 7u : kmask);
        }
        kmask = 0u;
        __syncwarp();
        set_thresholds();
    }
};

// Resident CTAs per SM the register budget is sized for: the plain field's
// 24 KB of stages admit more than three.
template <int K, bool COMP>
struct FkOcc { static constexpr int min_ctas = !COMP && K <= 3 ? 4 : 3; };

template <int K, bool REDUCE, bool SQ, bool COMP>
__global__ void __launch_bounds__(ADV_WARPS * 32, FkOcc<K, COMP>::min_ctas)
advance_f32k_kernel(const __grid_constant__ CUtensorMap map_hi,
                    const __grid_constant__ CUtensorMap map_lo,
                    const __grid_constant__ FkParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ Partial red[ADV_WARPS][K];
    __shared__ unsigned int s_last;
    __shared__ double s_tmx[ADV_WARPS][K][32];
    __shared__ long long s_arg[ADV_WARPS][K][32];
    __shared__ int s_ymn[ADV_WARPS][K], s_ymx[ADV_WARPS][K];
    __shared__ __align__(16) float s_box[ADV_WARPS][3][32][2 * ADV_V];

    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    constexpr int STAGE = fk_stage_floats<COMP>();
    float* stages = reinterpret_cast<float*>(smem) + wid * (ADV_S * STAGE);
    uint64_t* bars = reinterpret_cast<uint64_t*>(
        smem + size_t(ADV_WARPS) * ADV_S * STAGE * sizeof(float)) + wid * ADV_S;
    if (lane == 0) {
        for (int s = 0; s < ADV_S; ++s) mbar_init(&bars[s], 1);
        fence_mbar_init();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();

    FkStrip<K, REDUCE, SQ, COMP> ws(p, &map_hi, &map_lo, stages, bars, lane, s_tmx[wid], s_arg[wid],
                          s_ymn[wid], s_ymx[wid], s_box[wid]);
    pdl_trigger();
    pdl_wait();
    for (;;) {
        unsigned int t = 0;
        if (lane == 0) t = atomicAdd(p.tasks, 1u);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= (unsigned int)p.ntasks) break;
        ws.run_task((int)t);
        if (ws.failed) break;
    }

    const long long N = (long long)p.c.nx * p.c.ny;
    if constexpr (REDUCE) {
        __syncwarp();
        for (int t = 0; t < K; ++t) {
            double tm = s_tmx[wid][t][lane];
            long long ag = s_arg[wid][t][lane];
            const int mn = s_ymn[wid][t], mx = s_ymx[wid][t];
            partial_warp_peak(tm, ag);
            if (lane == 0) red[wid][t] = Partial{tm, ag, mn, mx};
        }
        __syncthreads();
        if (threadIdx.x < K) {
            const int t = threadIdx.x;
            double tm = -1.0; long long ag = N; int mn = p.c.ny, mx = -1;
            for (int w = 0; w < ADV_WARPS; ++w)
                partial_take(tm, ag, mn, mx, red[w][t].tmax, red[w][t].arg,
                             red[w][t].ymin, red[w][t].ymax);
            p.scratch[(size_t)blockIdx.x * K + t] = Partial{tm, ag, mn, mx};
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) s_last = (ticket(p.counter) == gridDim.x - 1) ? 1u : 0u;
    __syncthreads();
    if (!s_last) return;
    if constexpr (REDUCE) {
        // all of a thread's record loads before any combine, as the FP64 kernel
        constexpr int FIN_U = 5;
        double tm[K]; long long ag[K]; int mn[K], mx[K];
#pragma unroll
        for (int t = 0; t < K; ++t) { tm[t] = -1.0; ag[t] = N; mn[t] = p.c.ny; mx[t] = -1; }
        for (int i0 = threadIdx.x; i0 < (int)gridDim.x; i0 += blockDim.x * FIN_U) {
#pragma unroll
            for (int t = 0; t < K; ++t) {
                Partial q[FIN_U];
#pragma unroll
                for (int u = 0; u < FIN_U; ++u) {
                    const int i = i0 + u * (int)blockDim.x;
                    q[u] = Partial{-1.0, N, p.c.ny, -1};
                    if (i < (int)gridDim.x) {
                        const Partial* r = &p.scratch[(size_t)i * K + t];
                        q[u] = Partial{__ldcg(&r->tmax), __ldcg(&r->arg), __ldcg(&r->ymin),
                                       __ldcg(&r->ymax)};
                    }
                }
#pragma unroll
                for (int u = 0; u < FIN_U; ++u)
                    partial_take(tm[t], ag[t], mn[t], mx[t], q[u].tmax, q[u].arg, q[u].ymin,
                                 q[u].ymax);
            }
        }
        __syncthreads();
#pragma unroll
        for (int t = 0; t < K; ++t) {
            partial_warp_all(tm[t], ag[t], mn[t], mx[t]);
            if (lane == 0) red[wid][t] = Partial{tm[t], ag[t], mn[t], mx[t]};
        }
        __syncthreads();
        if (threadIdx.x < K) {
            const int t = threadIdx.x;
            double a = -1.0; long long b = N; int c1 = p.c.ny, d1 = -1;
            for (int w = 0; w < ADV_WARPS; ++w)
                partial_take(a, b, c1, d1, red[w][t].tmax, red[w][t].arg, red[w][t].ymin,
                             red[w][t].ymax);
            p.ring[t] = Partial{a, b, c1, d1};
        }
    }
    if (threadIdx.x == 0) { *p.counter = 0u; *p.tasks = 0u; }
}

}  // namespace lpbf_b200
