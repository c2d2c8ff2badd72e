# SPDX-License-Identifier: 0BSD
"""A wait between the resident kernel's tiles that runs out: the call ends,
the error word says so (bit 0), and the workspace is ready for the next call.
The limit is a word of the workspace (0: 4 s); one nanosecond lets some wait of
the many exchanges run out while its neighbour is merely a little behind."""
import numpy as np
import pytest

from hedgehog_lpbf_b200 import params as P
from hedgehog_lpbf_b200 import plan as PL

pytestmark = pytest.mark.gpu

COUNTER, TASKS, BARRIER, WAIT_NS = 0, 2, 3, 4        # words of the workspace's header
HEADER, PARTS = 256, 40960 * 24                      # bytes before the progress flags


@pytest.mark.parametrize("with_ring", [True, False])
@pytest.mark.parametrize("nx,ny", [(240, 120), (1021, 763)])
def test_wait_runs_out(gpu, nx, ny, with_ring):
    import torch
    from hedgehog_lpbf_b200 import _lib
    from hedgehog_lpbf_b200.solver import Solver, ring_to_numpy
    n = 300                                          # two launches
    mat, pr = P.benchmark_material_process()
    dom = P.Domain(Lx=(nx - 1) * 5e-6, Ly=(ny - 1) * 5e-6, nx=nx, ny=ny)
    k = P.make_const(mat, pr, dom, P.dt_fraction(mat, dom))
    plan = PL.raster_for_steps(dom, k.dt, n, V=1.0, hatch=100e-6, n_tracks=2)

    ref = Solver(k, Tm=mat.Tm, depth=3, T0=300.0, device="cuda:0")
    rr = ref.new_ring(n)
    want = ref.advance(plan, rr).cpu().numpy()

    s = Solver(k, Tm=mat.Tm, T0=300.0, device="cuda:0")
    assert s.launches(n) == 2
    words = s.work.view(torch.int32)
    ring = s.new_ring(n)
    words[WAIT_NS] = 1
    for _ in range(20):
        s.advance(plan, ring if with_ring else None)
        err = s.read_error()
        if err:
            break
    assert err & 1
    # re-armed by the call itself
    assert [int(words[w]) for w in (COUNTER, TASKS, BARRIER)] == [0, 0, 0]
    assert not s.work[HEADER + PARTS:].any()
    # a normal run on the same workspace, before and after its initialisation
    words[WAIT_NS] = 0
    for fresh in (False, True):
        if fresh:
            _lib.check(s.lib.lpbf_b200_workspace_init(
                s.work.data_ptr(), s.work.numel(), torch.cuda.current_stream().cuda_stream),
                "workspace_init")
        s.set_field(300.0)
        ring.zero_()
        got = s.advance(plan, ring).cpu().numpy()
        assert np.array_equal(got, want)
        assert ring_to_numpy(ring).tobytes() == ring_to_numpy(rr).tobytes()
        assert s.read_error() == (0 if fresh else err)
