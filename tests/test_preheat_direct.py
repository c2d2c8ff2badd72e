# SPDX-License-Identifier: 0BSD
"""Fields with Tamb != Tsub on direct loads (odd widths), which have a form of
the strip of their own: the laser on each mirror edge, on strip and chunk seams,
off the field and switched off, every depth and task height, with and
without Partials.  Against the oracle (1e-12 relative, the parity bar) and bit for
bit over depths and heights."""
import numpy as np
import pytest

from hedgehog_lpbf_b200 import params as P
from hedgehog_lpbf_b200 import plan as PL
from oracle import oracle as O

pytestmark = pytest.mark.gpu
N = 9


@pytest.mark.parametrize("nx,ny", [(3, 5), (119, 40), (121, 64), (245, 201), (483, 130)])
@pytest.mark.parametrize("bc,dy", [(0, 5e-6), (1, 5e-6), (0, 6e-6)])
@pytest.mark.parametrize("fx,fy", [(0.0, 0.5), (1.0, 1.0), (0.5, 0.0), (0.4, 0.4), (-0.4, 0.5)])
def test_every_depth_and_height(gpu, nx, ny, bc, dy, fx, fy):
    from hedgehog_lpbf_b200.solver import Solver, ring_to_numpy
    mat, pr = P.benchmark_material_process()
    pr.Tsub = 360.0
    dom = P.Domain(Lx=(nx - 1) * 5e-6, Ly=(ny - 1) * dy, nx=nx, ny=ny)
    k = P.make_const(mat, pr, dom, P.dt_fraction(mat, dom, 0.15))
    plan = np.zeros(N, dtype=PL.TICK_DTYPE)
    plan["x_l"] = fx * dom.Lx + np.arange(N) * 3e-6
    plan["y_l"] = fy * dom.Ly + np.arange(N) * 1e-6
    plan["q_scale"] = np.arange(N) % 4 != 3
    T0 = np.random.default_rng(nx * ny).uniform(290.0, 2100.0, nx * ny)
    ref, ring_ref = O.run(T0, k, PL.laser_array(plan), bc=bc, T_D=300.0, Tm=mat.Tm)
    first = None
    for depth in (1, 2, 3, 4):
        for rows in (0, 16, 64):
            s = Solver(k, bc=bc, T_edge=300.0, Tm=mat.Tm, depth=depth, rows=rows, T0=T0,
                       device="cuda:0")
            ring = s.new_ring(N)
            T = s.advance(plan, ring).cpu().numpy().ravel()
            r = ring_to_numpy(ring)
            if first is None:
                first = (T, r.tobytes())
                assert np.max(np.abs(T - ref) / np.maximum(np.abs(ref), 1.0)) <= 1e-12
                assert np.array_equal(r["ymin"], ring_ref["ymin"])
                assert np.array_equal(r["ymax"], ring_ref["ymax"])
                assert np.max(np.abs(r["tmax"] - ring_ref["tmax"]) / ring_ref["tmax"]) <= 1e-12
            assert np.array_equal(T, first[0]) and r.tobytes() == first[1], (depth, rows)
            s2 = Solver(k, bc=bc, T_edge=300.0, Tm=mat.Tm, depth=depth, rows=rows, T0=T0,
                        device="cuda:0")
            assert np.array_equal(s2.advance(plan).cpu().numpy().ravel(), T)    # no ring


@pytest.mark.parametrize("nx", [121, 245])
@pytest.mark.parametrize("depth", [1, 2, 3, 4])
def test_row_windows(gpu, nx, depth):
    """Row strips of the field: the rows of one launch equal the whole field's."""
    import ctypes
    import torch
    from hedgehog_lpbf_b200 import _lib
    from hedgehog_lpbf_b200.solver import Solver
    ny = 150
    mat, pr = P.benchmark_material_process()
    pr.Tsub = 360.0
    dom = P.Domain(Lx=(nx - 1) * 5e-6, Ly=(ny - 1) * 5e-6, nx=nx, ny=ny)
    k = P.make_const(mat, pr, dom, P.dt_fraction(mat, dom, 0.15))
    plan = np.zeros(depth, dtype=PL.TICK_DTYPE)
    plan["x_l"], plan["y_l"], plan["q_scale"] = 0.4 * dom.Lx, 0.45 * dom.Ly, 1.0
    T0 = np.random.default_rng(nx).uniform(290.0, 2100.0, (ny, nx))
    s = Solver(k, Tm=mat.Tm, depth=depth, T0=T0, device="cuda:0")
    src = s.field.clone()
    want = s.advance(plan).clone()
    for r0, r1, lo, hi in ((0, 70, 0, 60), (40, 110, 50, 100), (90, 150, 100, 150)):
        buf = src[r0:r1].clone()
        out = torch.full_like(buf, -7.0)
        kb = P.StepConst.from_buffer_copy(bytes(k))
        kb.ny = r1 - r0
        rows = _lib.Rows(row0=r0, global_ny=ny, lo=lo - r0, hi=hi - r0)
        opts = _lib.Opts(phys=0, bc=0, T_edge=300.0, Tm=mat.Tm, depth=depth, rows=0)
        _lib.check(s.lib.lpbf_b200_advance_rows(
            buf.data_ptr(), out.data_ptr(), ctypes.byref(kb), plan.ctypes.data, depth,
            ctypes.byref(opts), ctypes.byref(rows), None, s.work.data_ptr(), s.work.numel(),
            torch.cuda.current_stream().cuda_stream), "advance_rows")
        assert torch.equal(out[lo - r0:hi - r0], want[lo:hi]), (r0, lo)
        assert (out[:lo - r0] == -7.0).all() and (out[hi - r0:] == -7.0).all()
