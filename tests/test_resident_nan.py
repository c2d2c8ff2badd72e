# SPDX-License-Identifier: 0BSD
"""NaN never wins and never hides a finite peak beside it, at every position
of the NaN within a lane's cells, on resident fields of either lane width
(two cells at 200 x 150, four at the larger sizes), against the oracle and,
bit for bit, the launch path."""
import numpy as np
import pytest

from hedgehog_lpbf_b200 import params as P
from hedgehog_lpbf_b200 import plan as PL
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(200, 150), (768, 768), (1021, 763), (1024, 1024),
                                   (1344, 1216)])
@pytest.mark.parametrize("col", [100, 101, 102, 103])
@pytest.mark.parametrize("side", [-1, 1])
def test_peak_beside_a_nan(gpu, nx, ny, col, side):
    from hedgehog_lpbf_b200.solver import Solver, ring_to_numpy
    n = 2
    mat, pr = P.benchmark_material_process()
    dom = P.Domain(Lx=(nx - 1) * 5e-6, Ly=(ny - 1) * 5e-6, nx=nx, ny=ny)
    k = P.make_const(mat, pr, dom, P.dt_fraction(mat, dom, 0.05))
    plan = np.zeros(n, dtype=PL.TICK_DTYPE)          # beam off
    T0 = np.full((ny, nx), 300.0)
    y = 75
    T0[y, col] = np.nan
    # after one step the NaN covers (y +- 1, col); the peak stands beside it
    # (a lone hot cell keeps four fifths of its excess per step)
    T0[y + 1, col + side] = 2900.0
    T0[y - 1, col + 2 * side] = 2500.0               # the peak after two steps
    ref, want = O.run(T0, k, PL.laser_array(plan), Tm=mat.Tm)
    out = []
    for depth in (0, 1):
        s = Solver(k, Tm=mat.Tm, depth=depth, T0=T0, device="cuda:0")
        ring = s.new_ring(n)
        T = s.advance(plan, ring).cpu().numpy()
        assert s.read_error() & 2
        out.append((T, ring_to_numpy(ring)))
    (Ta, ra), (Tb, rb) = out
    assert np.array_equal(ra["arg"], want["arg"]), (ra, want)
    assert np.array_equal(ra["ymin"], want["ymin"]) and np.array_equal(ra["ymax"], want["ymax"])
    assert np.max(np.abs(ra["tmax"] - want["tmax"]) / want["tmax"]) <= 1e-12
    assert np.array_equal(Ta, Tb, equal_nan=True) and ra.tobytes() == rb.tobytes()
