# SPDX-License-Identifier: 0BSD
"""Source boxes at the places where their route changes: the laser on each
mirror edge and corner, on strip seams (120 columns) and chunk seams, and off
the field, for the FP64 and both FP32 fields; every depth and task height
against the oracle.

Tolerances: FP64 1e-12 relative (the parity bar).  FP32 plain: one rounding
per step of values below 4096 K is at most 1.3e-4 K; 12 steps and the source's
own rounding stay below 4e-3 K.  Compensated: 1e-3 K."""
import numpy as np
import pytest

from hedgehog_lpbf_b200 import params as P
from hedgehog_lpbf_b200 import plan as PL
from oracle import oracle as O

pytestmark = pytest.mark.gpu
NX, NY, N = 484, 200, 12


def _setup():
    mat, pr = P.benchmark_material_process()
    dom = P.Domain(Lx=(NX - 1) * 5e-6, Ly=(NY - 1) * 5e-6, nx=NX, ny=NY)
    k = P.make_const(mat, pr, dom, P.dt_fraction(mat, dom))
    plan = np.zeros(N, dtype=PL.TICK_DTYPE)
    plan["q_scale"] = 1.0
    return mat, dom, k, plan


@pytest.mark.parametrize("fx,fy", [(0.0, 0.5), (1.0, 0.5), (0.0, 0.0), (1.0, 1.0), (0.5, 0.0),
                                   (119.5 / 483, 64.0 / 199), (240.0 / 483, 0.4), (-0.1, 0.5)])
def test_source_on_edges_and_seams(gpu, fx, fy):
    from hedgehog_lpbf_b200.solver import Solver, SolverF32, SolverF32K, ring_to_numpy
    mat, dom, k, plan = _setup()
    plan["x_l"] = fx * dom.Lx + np.arange(N) * 3e-6
    plan["y_l"] = fy * dom.Ly + np.arange(N) * 1e-6
    T0 = np.full(NX * NY, 300.0)
    T0[: NX * 70] = 900.0
    ref, ring_ref = O.run(T0, k, PL.laser_array(plan), Tm=mat.Tm)
    for cls, tol, depths in ((Solver, None, (1, 2, 3, 4)), (SolverF32, 4e-3, (1, 2, 3, 4)),
                             (SolverF32K, 1e-3, (1, 2, 3, 4))):
        first = None
        for d in depths:
            for rows in (0, 16, 64):
                s = cls(k, Tm=mat.Tm, depth=d, rows=rows, T0=T0, device="cuda:0")
                ring = s.new_ring(N)
                s.advance(plan, ring)
                T = (s.field if cls is Solver else s.field64()).cpu().numpy().ravel()
                r = ring_to_numpy(ring)
                if first is None:
                    first = (T, r.tobytes())
                    if tol is None:
                        assert np.max(np.abs(T - ref) / np.maximum(np.abs(ref), 1.0)) <= 1e-12
                        assert np.array_equal(r["ymin"], ring_ref["ymin"])
                        assert np.array_equal(r["ymax"], ring_ref["ymax"])
                    else:
                        assert np.max(np.abs(T - ref)) <= tol
                        assert np.max(np.abs(r["tmax"] - ring_ref["tmax"])) <= tol
                assert np.array_equal(T, first[0]), (cls.__name__, d, rows)
                assert r.tobytes() == first[1], (cls.__name__, d, rows)
