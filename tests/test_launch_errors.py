# SPDX-License-Identifier: 0BSD
"""A launch that the runtime refuses is reported by the call's own status and
leaves no pending error behind for the next call of this library or of the
program's other CUDA code.  The refusal here is a stream whose capture was
invalidated by a synchronize: nothing reaches the device."""
import ctypes

import numpy as np
import pytest

from hedgehog_lpbf_b200 import params as P
from hedgehog_lpbf_b200 import plan as PL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("phys,depth", [(0, 0), (0, 1), (1, 0)])
def test_refused_launch_leaves_no_pending_error(gpu, phys, depth):
    import torch
    from hedgehog_lpbf_b200 import _lib
    from hedgehog_lpbf_b200.solver import Solver
    rt = ctypes.CDLL("libcudart.so.12")
    mat, pr = P.benchmark_material_process()
    dom = P.square_domain(64)
    k = P.make_const(mat, pr, dom, P.dt_fraction(mat, dom, 0.05))
    s = Solver(k, phys=phys, Tm=mat.Tm, depth=depth, T0=300.0, device="cuda:0")
    plan = np.zeros(1, dtype=PL.TICK_DTYPE)
    s.advance(plan)                                  # the kernel is loaded
    torch.cuda.synchronize()

    stream = ctypes.c_void_p()
    assert rt.cudaStreamCreate(ctypes.byref(stream)) == 0
    assert rt.cudaStreamBeginCapture(stream, 2) == 0           # relaxed mode
    assert rt.cudaStreamSynchronize(stream) != 0               # invalidates the capture
    rt.cudaGetLastError()
    in_b = ctypes.c_int(0)
    st = _lib.lib().lpbf_b200_advance(
        s.bufs[0].data_ptr(), s.bufs[1].data_ptr(), ctypes.byref(k), plan.ctypes.data, 1,
        ctypes.byref(s.opts), None, s.work.data_ptr(), s.work.numel(), stream, ctypes.byref(in_b))
    pending = rt.cudaGetLastError()
    graph = ctypes.c_void_p()
    rt.cudaStreamEndCapture(stream, ctypes.byref(graph))
    rt.cudaGetLastError()
    assert rt.cudaStreamDestroy(stream) == 0
    assert st == -4 and pending == 0, (st, pending)
