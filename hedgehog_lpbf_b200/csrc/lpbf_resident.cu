// SPDX-License-Identifier: 0BSD
// ---------------------------------------------------------------------------
// Tiling, eligibility and launch of the resident kernel (lpbf_resident.cuh).
// ---------------------------------------------------------------------------
#include <algorithm>
#include <cstring>

#include "lpbf_host.hpp"
#include "lpbf_resident.cuh"

namespace lpbf_b200 {

namespace {

template <int V, int NR, int MODE, bool REDUCE>
cudaError_t launch_t(const ResParams& p, cudaStream_t stream) {
    const size_t smem = res_smem_bytes(V, NR, p.K);
    static bool done[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    if (!done[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(
            resident_kernel<V, NR, MODE, REDUCE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
            (int)res_smem_bytes(V, NR, RES_KMAX));
        if (e != cudaSuccess) return e;
        done[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.gx * p.gy), 1, 1);
    cfg.blockDim = dim3(RES_THREADS, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return take_error(cudaLaunchKernelEx(&cfg, resident_kernel<V, NR, MODE, REDUCE>, p));
}

template <int V, int NR>
cudaError_t launch_m(const ResParams& p, cudaStream_t stream) {
    const Coef& c = p.c;
    const int mode = !c.same_T ? 2 : (c.ax == c.ay ? 0 : 1);
    switch (mode * 2 + (p.ring ? 1 : 0)) {
        case 0: return launch_t<V, NR, 0, false>(p, stream);
        case 1: return launch_t<V, NR, 0, true>(p, stream);
        case 2: return launch_t<V, NR, 1, false>(p, stream);
        case 3: return launch_t<V, NR, 1, true>(p, stream);
        case 4: return launch_t<V, NR, 2, false>(p, stream);
        default: return launch_t<V, NR, 2, true>(p, stream);
    }
}

// The padded tiles there are: V columns per lane, NR rows per warp.
struct Shape { int V, NR; };
constexpr Shape RES_SHAPES[] = {{2, 1}, {2, 2}, {2, 4}, {4, 2}, {2, 8}, {4, 4}, {4, 8}};

// Narrowest tile of n over a length in units.
int narrowest(int n, int len, int unit) {
    int w = len;
    for (int i = 0; i < n; ++i)
        w = std::min(w, res_bound(i + 1, n, len, unit) - res_bound(i, n, len, unit));
    return w;
}

// The padded tile, tiling and exchange depth with the least modelled time per
// step.
bool search_plan(int nx, int ny, int n_steps, ResPlan* out) {
    const int sms = std::min(sm_count(), RES_MAX_TILES);
    if (n_steps < 1 || nx < 2 || ny < 2 || (long long)nx * ny > (long long)sms * 128 * 128)
        return false;
    double best = 0.0;
    bool found = false;
    for (const Shape& sh : RES_SHAPES) {
        const int cols = 32 * sh.V, rows = RES_WARPS * sh.NR;
        for (int K = 1; K <= std::min(RES_KMAX, n_steps); ++K) {
            ResPlan pl;
            pl.V = sh.V; pl.NR = sh.NR; pl.K = K;
            // one tile across needs no halo on that axis
            pl.hx = nx <= cols ? 0 : (K + sh.V - 1) / sh.V * sh.V;
            pl.hy = ny <= rows ? 0 : K;
            const int tw = cols - 2 * pl.hx, th = rows - 2 * pl.hy;   // most a tile owns
            if (tw < 1 || th < 1) break;
            pl.gx = (nx + tw - 1) / tw;
            pl.gy = (ny + th - 1) / th;
            if ((long long)pl.gx * pl.gy > sms) break;
            // every halo must lie in the adjacent tile
            if ((pl.gx > 1 && narrowest(pl.gx, nx, sh.V) < K) ||
                (pl.gy > 1 && narrowest(pl.gy, ny, 1) < K))
                continue;
            // us: a step (fixed latency and per row of a warp), plus one
            // exchange per K steps; fitted to a sweep of all shapes and K
            const double step = sh.V == 2 ? 0.24 + 0.24 * sh.NR : 0.55 + 0.40 * sh.NR;
            const double exch = 2.1 + 0.14 * sh.V * sh.NR;
            const double t = step + exch / K;
            if (!found || t < best) { best = t; *out = pl; found = true; }
        }
    }
    if (found) out->steps = std::min(RES_STEPS, WS_PARTS / (out->gx * out->gy));
    return found;
}

}  // namespace

// The search's answer depends on its arguments and the SM count only, and
// takes longer than a short launch: each thread keeps its last one.
bool resident_plan(int nx, int ny, int n_steps, ResPlan* out) {
    struct Last { int nx, ny, n, sms; bool ok; ResPlan pl; };
    static thread_local Last last = {0, 0, 0, 0, false, {}};
    const int n = std::min(n_steps, RES_STEPS), sms = sm_count();
    if (last.nx != nx || last.ny != ny || last.n != n || last.sms != sms) {
        last.ok = search_plan(nx, ny, n, &last.pl);
        last.nx = nx; last.ny = ny; last.n = n; last.sms = sms;
    }
    *out = last.pl;
    return last.ok;
}

cudaError_t launch_resident(const ResPlan& pl, const double* Tin, double* Tout, double* Tin_rw,
                            const Coef& c, const LaserSub* las, int n_steps, Partial* ring,
                            Workspace* ws, cudaStream_t stream) {
    ResParams p;
    std::memset(&p, 0, sizeof(p));
    p.c = c;
    p.Tin = Tin;
    p.Tout = Tout;
    p.xbuf[0] = Tin_rw;
    p.xbuf[1] = Tout;
    p.ring = ring;
    p.scratch = ws->parts;
    p.flags = ws->flags;
    p.counter = &ws->counter;
    p.barrier = &ws->barrier;
    p.err = &ws->err;
    p.wait_ns = &ws->wait_ns;
    p.n_steps = n_steps;
    p.K = pl.K;
    p.nblocks = (n_steps + pl.K - 1) / pl.K | 1;      // odd: the result is in Tout
    p.gx = pl.gx; p.gy = pl.gy;
    p.hx = pl.hx; p.hy = pl.hy;
    for (int s = 0; s < n_steps; ++s) p.las[s] = las[s];
    switch (pl.V * 16 + pl.NR) {
        case 2 * 16 + 1: return launch_m<2, 1>(p, stream);
        case 2 * 16 + 2: return launch_m<2, 2>(p, stream);
        case 2 * 16 + 4: return launch_m<2, 4>(p, stream);
        case 2 * 16 + 8: return launch_m<2, 8>(p, stream);
        case 4 * 16 + 2: return launch_m<4, 2>(p, stream);
        case 4 * 16 + 4: return launch_m<4, 4>(p, stream);
        case 4 * 16 + 8: return launch_m<4, 8>(p, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace lpbf_b200
