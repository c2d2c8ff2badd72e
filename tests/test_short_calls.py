# SPDX-License-Identifier: 0BSD
"""Calls of one to three steps around the sizes where they change from the
resident kernel to the launch path: one launch either way, fields and Partials
bit for bit those of single-step launches."""
import numpy as np
import pytest

from hedgehog_lpbf_b200 import params as P
from hedgehog_lpbf_b200 import plan as PL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1000, 1000), (1025, 1023), (1024, 1024), (1344, 1216),
                                   (2000, 1000), (1900, 1000)])
@pytest.mark.parametrize("n", [1, 2, 3])
def test_one_launch_and_the_same_bits(gpu, nx, ny, n):
    from hedgehog_lpbf_b200.solver import Solver, ring_to_numpy
    mat, pr = P.benchmark_material_process()
    dom = P.Domain(Lx=(nx - 1) * 5e-6, Ly=(ny - 1) * 5e-6, nx=nx, ny=ny)
    k = P.make_const(mat, pr, dom, P.dt_fraction(mat, dom))
    plan = PL.raster_for_steps(dom, k.dt, n, V=1.0, hatch=100e-6, n_tracks=2)
    T0 = np.random.default_rng(nx + n).uniform(300.0, 2100.0, nx * ny)
    out = []
    for depth in (0, 1):
        s = Solver(k, Tm=mat.Tm, depth=depth, T0=T0, device="cuda:0")
        ring = s.new_ring(n)
        T = s.advance(plan, ring)
        out.append((T.cpu().numpy(), ring_to_numpy(ring).tobytes(), s.read_error()))
        assert depth or (s.launches(n) == 1 and s.cur == 1)
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]
    assert out[0][2] == out[1][2] == 0
