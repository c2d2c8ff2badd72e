// SPDX-License-Identifier: 0BSD
// ---------------------------------------------------------------------------
// Device building blocks shared by every kernel of liblpbf_b200:
//   * Coef / LaserSub: the per-launch constants, pre-scaled by dt on the host;
//   * cell_update: the baseline explicit-Euler update of one cell;
//   * PTX wrappers for mbarriers and TMA (cp.async.bulk.tensor) loads;
//   * the Partial combine rule (max T, ties -> smallest flat index, min/max
//     molten row) used by every reduction.
//
// The update evaluates the reference's step (include/step_task.hpp:95-129,
// src/gpu/kernels.cu:106-124)
//     T' = T + dt * ( alpha*(lap_x + lap_y) + S - loss(T) )
// with every dt-scaled coefficient folded on the host:
//     T' = T + ( ax*(R + L - 2T) + ay*(U + D - 2T) + S_dt - loss_dt(T) ).
// At equilibrium (uniform field at the ambient temperature) every term is
// zero or, in the fused Tamb == Tsub form of the step kernel, a last rounding
// far below half an ulp of T, so untouched far-field cells stay bit-exactly
// at T_amb, as in the reference; all other differences are rounding of the
// increment, far below 1e-12 of T.
// ---------------------------------------------------------------------------
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "lpbf_step_const.hpp"

namespace lpbf_b200 {

constexpr int KMAX = 8;            // most time steps one launch can carry
constexpr double SIGMA_SB = 5.670374419e-8;
// Gaussian truncation: a cell whose Gaussian factor exp(-2 r^2 / r0^2) is
// below 2^-80 (exponent below -80 ln 2, r > 5.27 r0) gets S = 0 without
// evaluating exp.  The heat left out is under 2^-80 of the step's peak
// increment per cell (below 1e-22 K per step for a 200 W, 50 um spot), many
// orders of magnitude under the 1e-12 relative agreement with the
// reference's untruncated step; it keeps the exp-evaluating region a few
// spot radii wide instead of the ~19 radii at which exp underflows to zero.
constexpr double EXP_CUT = 55.451774444795625;   // 80 ln 2

struct LaserSub {
    double x_l, y_l;
    double cs;                     // dt * q_scale * peak_S / (rho_cp * h)
};

struct Coef {
    int    nx, ny;
    double dx, dy;
    double ax, ay;                 // dt*alpha/dx^2, dt*alpha/dy^2
    double c_conv, c_sub, c_ls;    // dt*hConv/(h rho cp), dt*(K/dSub)/(h rho cp), their sum
    double c_rad;                  // dt*eps*sigma/(h rho cp), 0 without radiation
    double Tamb, Tsub, Tamb4;      // Tamb4 = (Tamb*Tamb)*(Tamb*Tamb)
    double m2r;                    // -2 / r0^2
    double r2_cut;                 // r^2 beyond which S is taken as 0 (truncation)
    double Tm;                     // melt threshold of the reduction
    double T_edge;                 // fixed edge temperature (bc == 1)
    int    bc;                     // 0 mirror (ghost = centre), 1 fixed edges
    int    same_T;                 // Tamb == Tsub: one conduction term
};

// Host: fold a reference StepConst into launch constants.
inline Coef make_coef(const StepConst& k, int bc, double T_edge, double Tm) {
    Coef c{};
    c.nx = k.nx; c.ny = k.ny;
    c.dx = k.dx; c.dy = k.dy;
    c.ax = k.dt * k.alpha * k.inv_dx2;
    c.ay = k.dt * k.alpha * k.inv_dy2;
    const double s = k.dt * k.inv_h / k.rho_cp;
    c.c_conv = s * k.hConv;
    c.c_sub  = s * (k.K / k.dSub);
    c.c_ls   = c.c_conv + c.c_sub;
    c.c_rad  = k.radiation ? s * (k.eps * SIGMA_SB) : 0.0;
    c.Tamb = k.Tamb; c.Tsub = k.Tsub;
    const double ta2 = k.Tamb * k.Tamb;
    c.Tamb4 = ta2 * ta2;
    c.m2r = -2.0 * k.inv_r0_sq;
    c.r2_cut = (0.5 * EXP_CUT) / k.inv_r0_sq;
    c.Tm = Tm; c.T_edge = T_edge; c.bc = bc;
    c.same_T = (k.Tamb == k.Tsub) ? 1 : 0;
    return c;
}

inline LaserSub make_laser(const StepConst& k, double x_l, double y_l, double q_scale) {
    LaserSub l;
    l.x_l = x_l; l.y_l = y_l;
    l.cs = k.dt * (q_scale * k.peak_S) / (k.rho_cp * k.h);
    return l;
}

// dt-scaled loss of one cell.  The multiplies are spelled out so that the
// radiation difference is exactly zero at T = Tamb (Tamb4 is formed the same
// way on the host).
__device__ __forceinline__ double loss_dt(double T, const Coef& c) {
    const double da = __dsub_rn(T, c.Tamb);
    const double t2 = __dmul_rn(T, T);
    const double e4 = __dsub_rn(__dmul_rn(t2, t2), c.Tamb4);
    double lin;
    if (c.same_T) lin = __dmul_rn(c.c_ls, da);
    else          lin = fma(c.c_sub, __dsub_rn(T, c.Tsub), __dmul_rn(c.c_conv, da));
    return fma(c.c_rad, e4, lin);
}

// Baseline update of one cell (general Tamb != Tsub form); S_dt dt-scaled.
__device__ __forceinline__ double cell_update(double T, double L, double R,
                                              double U, double D, double S_dt,
                                              const Coef& c) {
    const double lx = fma(-2.0, T, R + L);
    const double ly = fma(-2.0, T, U + D);
    const double inc = fma(c.ax, lx, __dmul_rn(c.ay, ly));
    return __dadd_rn(T, __dsub_rn(__dadd_rn(inc, S_dt), loss_dt(T, c)));
}

// ---- Partial combine: larger T wins, equal T -> smaller index ------------
__device__ __forceinline__ void partial_take(double& tm, long long& ag, int& mn, int& mx,
                                             double t2, long long a2, int mn2, int mx2) {
    if (t2 > tm || (t2 == tm && a2 < ag)) { tm = t2; ag = a2; }
    mn = min(mn, mn2);
    mx = max(mx, mx2);
}
__device__ __forceinline__ void partial_warp_reduce(double& tm, long long& ag, int& mn, int& mx) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const double t2 = __shfl_xor_sync(0xffffffffu, tm, off);
        const long long a2 = __shfl_xor_sync(0xffffffffu, ag, off);
        const int mn2 = __shfl_xor_sync(0xffffffffu, mn, off);
        const int mx2 = __shfl_xor_sync(0xffffffffu, mx, off);
        partial_take(tm, ag, mn, mx, t2, a2, mn2, mx2);
    }
}

// Order-preserving unsigned key of a double (not NaN) and back.
__device__ __forceinline__ unsigned long long order_key(double v) {
    const long long b = __double_as_longlong(v);
    return (unsigned long long)b ^ ((unsigned long long)(b >> 63) | 0x8000000000000000ull);
}
__device__ __forceinline__ double order_unkey(unsigned long long k) {
    const unsigned long long b =
        (k & 0x8000000000000000ull) ? k ^ 0x8000000000000000ull : ~k;
    return __longlong_as_double((long long)b);
}
// -0.0's key, one below +0.0's, although the two compare equal.
constexpr unsigned long long NEG_ZERO_KEY = 0x7fffffffffffffffull;
// Largest tm over the warp and the smallest index among the lanes that hold
// it, in every lane: four integer warp reductions on the halves of the two
// words (five rounds of shuffles take thirty).  Peaks are never NaN and
// indices never negative.  A -0.0 takes +0.0's key and leaves a mark in the
// index's lowest bit, so that the winner's own zero comes back (with a vote
// and a shuffle for it instead, 90 steps of a 2048^2 field took 1.5 % longer).
__device__ __forceinline__ void partial_warp_peak(double& tm, long long& ag) {
    unsigned long long k = order_key(tm);
    const unsigned int z = k == NEG_ZERO_KEY ? 1u : 0u;
    k += z;
    const unsigned long long a = ((unsigned long long)ag << 1) | z;
    const unsigned int hi = (unsigned int)(k >> 32), lo = (unsigned int)k;
    const unsigned int h = __reduce_max_sync(0xffffffffu, hi);
    const unsigned int l = __reduce_max_sync(0xffffffffu, hi == h ? lo : 0u);
    const bool top = hi == h && lo == l;
    const unsigned int ah = (unsigned int)(a >> 32), al = (unsigned int)a;
    const unsigned int gh = __reduce_min_sync(0xffffffffu, top ? ah : 0xffffffffu);
    const unsigned int gl = __reduce_min_sync(0xffffffffu, top && ah == gh ? al : 0xffffffffu);
    tm = gl & 1u ? -0.0 : order_unkey(((unsigned long long)h << 32) | l);
    ag = (long long)((((unsigned long long)gh << 32) | gl) >> 1);
}

// The whole warp's Partial, in every lane.
__device__ __forceinline__ void partial_warp_all(double& tm, long long& ag, int& mn, int& mx) {
    partial_warp_peak(tm, ag);
    mn = __reduce_min_sync(0xffffffffu, mn);
    mx = __reduce_max_sync(0xffffffffu, mx);
}
// Take a ticket after this thread's earlier writes, and (the release is
// cumulative) those of threads it has synchronized with; whoever draws the
// last one sees the writes behind the others.
__device__ __forceinline__ unsigned int ticket(unsigned int* p) {
    unsigned int v;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// ---- PTX: shared-memory addresses, mbarriers, TMA ----------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(bar)), "r"(count)
                 : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                 :: "r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Wait for an mbarrier phase with a time limit (1 s).  Returns false when the
// limit ran out; the caller then records an error and stops issuing work.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = globaltimer_ns();
    while (!mbar_try_wait(bar, parity)) {
        if (globaltimer_ns() - t0 > 1000000000ull) return false;
    }
    return true;
}
// Programmatic dependent launch.  Kernels of a run are launched with
// launch_chained (lpbf_host.hpp): the next launch's blocks may take the places
// of finished blocks before this kernel ends.  pdl_trigger allows that;
// pdl_wait, before a kernel's first access to global memory, waits until every
// earlier kernel of the stream has completed and its writes are visible.
// What such a kernel wrote is read by plain loads, which stay behind the wait:
// __ldg and const __restrict__ promise memory that nobody writes while this
// kernel runs, and it runs while its producer still does.
__device__ __forceinline__ void pdl_trigger() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
// 2D tiled TMA load of box (x, y) into this CTA's shared memory.  x must be
// even for f64 (16-byte rule); y may be negative or past the end (zero fill).
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y,
                                            uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];"
        :: "r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y),
           "r"(smem_u32(bar))
        : "memory");
}

// Untiled bulk copy of `bytes` (a multiple of 16) from global memory into
// this CTA's shared memory; both addresses 16-byte aligned.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes,
                                          uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        :: "r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes),
           "r"(smem_u32(bar))
        : "memory");
}

// ---- packed pairs of f32 -----------------------------------------------------
// sm_100a executes two f32 operations per instruction on a 64-bit register
// pair, each rounded as its scalar form.
typedef unsigned long long p2;
__device__ __forceinline__ p2 p2_pack(float a, float b) {
    p2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float p2_a(p2 v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return a;
}
__device__ __forceinline__ float p2_b(p2 v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return b;
}
__device__ __forceinline__ p2 p2_add(p2 a, p2 b) {
    p2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ p2 p2_mul(p2 a, p2 b) {
    p2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ p2 p2_fma(p2 a, p2 b, p2 c) {
    p2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ p2 p2_sub(p2 a, p2 b) {
    p2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// Rounded towards +infinity.
__device__ __forceinline__ p2 p2_sub_up(p2 a, p2 b) {
    p2 r;
    asm("sub.rp.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

}  // namespace lpbf_b200
