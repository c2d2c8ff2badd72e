# SPDX-License-Identifier: 0BSD
"""Extended physics at the edges of its tiling (60-column strips, 4-row
blocks, paired and single loads) and with the laser on edges and corners,
against the oracle: field within 1e-12 relative (the parity bar), Partials'
rows exact, peaks within 1e-12, Tsub equal to and other than Tamb."""
import numpy as np
import pytest

from hedgehog_lpbf_b200 import params as P
from hedgehog_lpbf_b200 import plan as PL
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [2, 3, 58, 60, 61, 62, 64, 119, 122])
@pytest.mark.parametrize("bc", [0, 1])
def test_strip_and_block_edges(gpu, nx, bc):
    from hedgehog_lpbf_b200.solver import Solver, ring_to_numpy
    n = 5
    for ny in (2, 3, 5, 8, 13, 66):
        mat, pr = P.benchmark_material_process()
        pr.Tsub = 300.0 if (nx + ny) % 2 else 340.0
        dom = P.Domain(Lx=(nx - 1) * 5e-6, Ly=(ny - 1) * 5e-6, nx=nx, ny=ny)
        k = P.make_const(mat, pr, dom, P.dt_fraction(mat, dom, 0.05))
        k.kmult = 2.0 if ny % 3 == 0 else 1.0
        las = np.array([[0.0, 0.0, 1.0], [dom.Lx, dom.Ly, 1.0], [0.5 * dom.Lx, 0.0, 1.0],
                        [dom.Lx, 0.3 * dom.Ly, 0.5], [0.4 * dom.Lx, 0.6 * dom.Ly, 0.0]])
        plan = np.zeros(n, dtype=PL.TICK_DTYPE)
        plan["x_l"], plan["y_l"], plan["q_scale"] = las.T
        T0 = np.random.default_rng(nx * 100 + ny).uniform(280.0, 2300.0, nx * ny)
        ref, rr = O.run(T0, k, las, phys=1, bc=bc, T_D=300.0, Tm=mat.Tm)
        s = Solver(k, phys=1, bc=bc, T_edge=300.0, Tm=mat.Tm, T0=T0, device="cuda:0")
        ring = s.new_ring(n)
        T = s.advance(plan, ring).cpu().numpy().ravel()
        assert np.max(np.abs(T - ref) / np.maximum(np.abs(ref), 1.0)) <= 1e-12, (nx, ny)
        r = ring_to_numpy(ring)
        assert np.array_equal(r["ymin"], rr["ymin"]) and np.array_equal(r["ymax"], rr["ymax"])
        assert np.max(np.abs(r["tmax"] - rr["tmax"]) / rr["tmax"]) <= 1e-12
