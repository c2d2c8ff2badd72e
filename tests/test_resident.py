# SPDX-License-Identifier: 0BSD
"""The resident kernel (fields advanced many steps per launch from shared
memory) against the temporally blocked launch path: fields and Partials bit
for bit, at the edges of its tiling (one tile, odd sides, long and narrow
fields, step counts around its exchange and launch lengths), and against the
oracle's non-finite and tie rules."""
import numpy as np
import pytest

from hedgehog_lpbf_b200 import params as P
from hedgehog_lpbf_b200 import plan as PL

pytestmark = pytest.mark.gpu


def _run(k, plan, T0, Tm, bc, depth, ring=True, T_edge=300.0):
    from hedgehog_lpbf_b200.solver import Solver, ring_to_numpy
    s = Solver(k, bc=bc, T_edge=T_edge, Tm=Tm, depth=depth, T0=T0, device="cuda:0")
    r = s.new_ring(len(plan)) if ring else None
    s.advance(plan, r)
    err = s.read_error()
    return s.field.cpu().numpy(), ring_to_numpy(r) if ring else None, err, s.launches(len(plan))


def _case(nx, ny, n, dy=5e-6, Tsub=300.0, angle=0.3):
    mat, pr = P.benchmark_material_process()
    pr.Tsub = Tsub
    dom = P.Domain(Lx=(nx - 1) * 5e-6, Ly=(ny - 1) * dy, nx=nx, ny=ny)
    k = P.make_const(mat, pr, dom, P.dt_fraction(mat, dom, 0.15))
    # tracks that leave the domain: the source meets every edge
    plan = PL.raster(dom, k.dt, n, V=40.0, hatch=60e-6, track_len=1.3 * dom.Lx + 1e-5,
                     n_tracks=3, angle=angle, jump_time=3 * k.dt)
    return mat, k, plan


# one tile; odd and even sides; narrow in x and in y; more tiles than rows of
# one SM; the largest tiles; rectangular cells; Tsub != Tamb
SHAPES = [(8, 8), (2, 40), (33, 2), (97, 61), (240, 120), (512, 512), (1021, 763), (1400, 37),
          (30, 3000), (1344, 1216)]


@pytest.mark.parametrize("nx,ny", SHAPES)
@pytest.mark.parametrize("bc", [0, 1])
def test_equals_launch_path(gpu, nx, ny, bc):
    rng = np.random.default_rng(nx + ny)
    T0 = 300.0 + rng.uniform(0.0, 1800.0, nx * ny)
    big = nx * ny > 300000
    for n in ([19] if big else [1, 2, 7, 33, 300]):
        for kw in ({}, {"dy": 6e-6}, {"Tsub": 353.0}):
            if big and kw and bc:
                continue
            mat, k, plan = _case(nx, ny, n, **kw)
            a, ra, ea, la = _run(k, plan, T0, mat.Tm, bc, 0)
            b, rb, eb, _ = _run(k, plan, T0, mat.Tm, bc, 1)
            assert la == (n + 255) // 256
            assert np.array_equal(a, b), (n, kw, np.max(np.abs(a - b)))
            assert ra.tobytes() == rb.tobytes(), (n, kw)
            assert ea == eb == 0


def test_ties_plateaus_and_no_ring(gpu):
    """Uniform and plateau fields with the beam off (every cell or several
    tiles tie for the peak), and a run without a ring."""
    nx, ny, n = 400, 300, 21
    mat, k, plan = _case(nx, ny, n)
    plan["q_scale"] = 0.0
    for T0 in (np.full((ny, nx), 300.0), np.full((ny, nx), 2000.0)):
        T0 = T0.copy()
        T0[40:60, 30:50] = T0[40:60, 330:350] = T0[240:260, 30:50] = 2500.0
        for start in (T0, np.full((ny, nx), T0[0, 0])):
            a, ra, _, _ = _run(k, plan, start, mat.Tm, 0, 0)
            b, rb, _, _ = _run(k, plan, start, mat.Tm, 0, 2)
            assert np.array_equal(a, b) and ra.tobytes() == rb.tobytes()
            c, _, _, _ = _run(k, plan, start, mat.Tm, 0, 0, ring=False)
            assert np.array_equal(a, c)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_cells_are_flagged(gpu, bad):
    nx, ny = 200, 150
    mat, k, plan = _case(nx, ny, 3)
    T0 = np.full((ny, nx), 300.0)
    T0[70, 90] = bad
    a, ra, err, _ = _run(k, plan, T0, mat.Tm, 0, 0)
    b, rb, eb, _ = _run(k, plan, T0, mat.Tm, 0, 1)
    assert err & 2 and eb & 2
    assert np.array_equal(a, b, equal_nan=True)
    assert ra.tobytes() == rb.tobytes()


def test_two_streams(gpu):
    """Two solvers on two streams at once: each its own field and workspace."""
    import torch
    from hedgehog_lpbf_b200.solver import Solver
    mat, k, plan = _case(320, 200, 120)
    want, _, _, _ = _run(k, plan, np.full((200, 320), 300.0), mat.Tm, 0, 0)
    ss = [Solver(k, Tm=mat.Tm, T0=300.0, device="cuda:0") for _ in range(2)]
    rings = [s.new_ring(120) for s in ss]
    streams = [torch.cuda.Stream() for _ in ss]
    torch.cuda.synchronize()
    for s, r, st in zip(ss, rings, streams):
        s.advance(plan, r, stream=st)
    torch.cuda.synchronize()
    for s in ss:
        assert s.read_error() == 0
        assert np.array_equal(s.field.cpu().numpy(), want)


def test_capture_and_replay(gpu):
    """Two launches (300 steps) captured in a CUDA graph and replayed twice."""
    import torch
    from hedgehog_lpbf_b200.solver import Solver, ring_to_numpy
    mat, k, plan = _case(240, 120, 300)
    want, rw, _, n = _run(k, plan, np.full((120, 240), 300.0), mat.Tm, 0, 0)
    assert n == 2
    s = Solver(k, Tm=mat.Tm, T0=300.0, device="cuda:0")
    ring = s.new_ring(300)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):
        s.advance(plan, ring, stream=side)
    assert s.cur == 0                      # an even number of launches
    for _ in range(2):
        s.set_field(300.0)
        ring.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(s.field.cpu().numpy(), want)
        assert ring_to_numpy(ring).tobytes() == rw.tobytes()
    assert s.read_error() == 0
