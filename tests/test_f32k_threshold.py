# SPDX-License-Identifier: 0BSD
"""Compensated FP32: a later cell that exceeds the lane's peak by the least a
pair can (2^-25 of an ulp of hi, across a step of hi) is the peak.  Coefficients
are zero, so the pairs keep their values; both cells belong to one lane and to
interior rows of one task.  Bodies and depths agree bit for bit."""
import numpy as np
import pytest

from hedgehog_lpbf_b200 import params as P
from hedgehog_lpbf_b200 import plan as PL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [1, 2, 3, 4])
@pytest.mark.parametrize("dy", [5e-6, 6e-6])
def test_smallest_step_above_the_peak(gpu, depth, dy):
    from hedgehog_lpbf_b200.solver import SolverF32K, ring_to_numpy
    nx, ny, n = 484, 200, 4
    mat, pr = P.benchmark_material_process()
    dom = P.Domain(Lx=(nx - 1) * 5e-6, Ly=(ny - 1) * dy, nx=nx, ny=ny)
    k = P.make_const(mat, pr, dom, 5e-7)
    k.alpha = k.K = k.hConv = 0.0
    k.radiation = False
    plan = np.zeros(n, dtype=PL.TICK_DTYPE)          # beam off
    hi = np.float32(1500.0)                          # even mantissa, ulp 2^-13
    ulp = 2.0 ** -13
    a = float(hi) + 0.5 * ulp                        # (hi, +ulp/2): a tie, to even
    b = a + ulp * 2.0 ** -25                         # (hi + ulp, -(ulp/2 - 2^-25 ulp))
    assert np.float32(a) == hi and np.float32(b) == np.float32(float(hi) + ulp) and b > a
    T0 = np.full((ny, nx), 300.0)
    T0[95, 200], T0[110, 201] = a, b
    s = SolverF32K(k, Tm=1e4, depth=depth, rows=64, T0=T0, device="cuda:0")
    ring = s.new_ring(n)
    s.advance(plan, ring)
    T = s.field64().cpu().numpy()
    assert np.array_equal(T, T0)
    for r in ring_to_numpy(ring):
        assert r["tmax"] == b and r["arg"] == 110 * nx + 201, r
