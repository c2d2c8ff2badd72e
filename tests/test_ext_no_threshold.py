# SPDX-License-Identifier: 0BSD
"""Extended physics with melt thresholds no cell can exceed (NaN, +inf): peaks
are reported all the same, no row is molten; against the oracle."""
import numpy as np
import pytest

from hedgehog_lpbf_b200 import params as P
from hedgehog_lpbf_b200 import plan as PL
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Tm", [np.nan, np.inf])
@pytest.mark.parametrize("nx", [122, 125])
def test_peaks_without_a_melt_threshold(gpu, Tm, nx):
    from hedgehog_lpbf_b200.solver import Solver, ring_to_numpy
    ny, n = 90, 4
    mat, pr = P.benchmark_material_process()
    dom = P.Domain(Lx=(nx - 1) * 5e-6, Ly=(ny - 1) * 5e-6, nx=nx, ny=ny)
    k = P.make_const(mat, pr, dom, P.dt_fraction(mat, dom, 0.05))
    plan = PL.raster_for_steps(dom, k.dt, n, V=1.0, hatch=100e-6, n_tracks=2)
    T0 = np.random.default_rng(nx).uniform(280.0, 2300.0, nx * ny)
    ref, want = O.run(T0, k, PL.laser_array(plan), phys=1, Tm=Tm)
    s = Solver(k, phys=1, Tm=Tm, T0=T0, device="cuda:0")
    ring = s.new_ring(n)
    s.advance(plan, ring)
    got = ring_to_numpy(ring)
    assert np.max(np.abs(got["tmax"] - want["tmax"]) / want["tmax"]) <= 1e-12
    assert np.array_equal(got["arg"], want["arg"])
    assert (got["ymin"] == ny).all() and (got["ymax"] == -1).all()
