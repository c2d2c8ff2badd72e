# SPDX-License-Identifier: 0BSD
"""Boxes beside the source rows read no source factor that was not filled.

A task keeps its column factors in local memory.  A kernel that writes +inf
into every thread's local memory runs before each advance: a factor read
without having been filled would then give 0 * inf = NaN.  Row chunks end
right below the source rows (where the band split puts a seam) at every depth
and task height; fields and Partials must not depend on what the local memory
held."""
import numpy as np
import pytest

from hedgehog_lpbf_b200 import params as P
from hedgehog_lpbf_b200 import plan as PL

pytestmark = pytest.mark.gpu
NX, NY = 484, 300

FILL = r"""
extern "C" __global__ void fill_local(double v, int n, double* out) {
    volatile double f[64];
    for (int i = 0; i < n; ++i) f[i & 63] = v;
    if (f[n & 63] == 0.123) out[0] = v;
}
"""


@pytest.fixture(scope="module")
def fill(gpu):
    import torch
    kern = torch.cuda._compile_kernel(FILL, "fill_local")
    out = torch.zeros(1, dtype=torch.float64, device="cuda:0")
    sms = torch.cuda.get_device_properties(0).multi_processor_count

    def run(value):
        # every warp's place on every SM (512 threads, 4 CTAs per SM), twice
        kern(grid=(8 * sms, 1, 1), block=(512, 1, 1), args=[float(value), 64, out])
    return run


def _setup(n):
    mat, pr = P.benchmark_material_process()
    dom = P.Domain(Lx=(NX - 1) * 5e-6, Ly=(NY - 1) * 5e-6, nx=NX, ny=NY)
    k = P.make_const(mat, pr, dom, P.dt_fraction(mat, dom))
    plan = np.zeros(n, dtype=PL.TICK_DTYPE)
    plan["q_scale"] = 1.0
    plan["x_l"] = 0.5 * dom.Lx
    plan["y_l"] = 0.4 * dom.Ly + np.arange(n) * 1e-6
    return mat, k, plan


@pytest.mark.parametrize("form", ["Solver", "SolverF32", "SolverF32K"])
@pytest.mark.parametrize("depth", [1, 2, 3, 4])
def test_local_memory_does_not_matter(gpu, fill, form, depth):
    from hedgehog_lpbf_b200 import solver as S
    mat, k, plan = _setup(depth)
    for rows in (0, 16):
        got = []
        for value in (0.0, np.inf):
            s = getattr(S, form)(k, Tm=mat.Tm, depth=depth, rows=rows, T0=900.0, device="cuda:0")
            ring = s.new_ring(depth)
            fill(value)
            s.advance(plan, ring)
            T = s.field if form == "Solver" else s.field64()
            got.append((T.cpu().numpy(), S.ring_to_numpy(ring).tobytes()))
        assert np.isfinite(got[1][0]).all(), (rows, int((~np.isfinite(got[1][0])).sum()))
        assert np.array_equal(got[0][0], got[1][0]) and got[0][1] == got[1][1], rows


@pytest.mark.parametrize("depth", [1, 2, 3, 4])
def test_local_memory_does_not_matter_in_a_batch(gpu, fill, depth):
    from hedgehog_lpbf_b200.batch import Batch, Scenario, batch_opts
    mat, k, plan = _setup(depth)
    for rows in ((0, 0, 0, 0), (16, 16, 16, 16)):
        got = []
        for value in (0.0, np.inf):
            scs = [Scenario(k=k, plan=plan, bc=0, T_edge=300.0, Tm=mat.Tm,
                            T0=np.full((NY, NX), 900.0)) for _ in range(3)]
            b = Batch(scs, depth, opts=batch_opts(depth=depth, rows=rows), device="cuda:0")
            fill(value)
            b.run(0, depth)
            got.append([(b.field(i).cpu().numpy(), b.ring(i)[:depth].tobytes()) for i in range(3)])
            b.close()
        for (T, r), (Tp, rp) in zip(*got):
            assert np.isfinite(Tp).all()
            assert np.array_equal(T, Tp) and r == rp
