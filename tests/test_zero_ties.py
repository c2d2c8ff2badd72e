# SPDX-License-Identifier: 0BSD
"""-0.0 and +0.0 tie for the peak: the smaller flat index wins and its own
zero is the peak, as in the reference's rule (src/gpu/kernels.cu:205-262,
where they compare equal).  Fixed edges at -0.0 around a field at 0 K, on
every path that reduces a field; against the rule applied to the returned
field."""
import numpy as np
import pytest

from hedgehog_lpbf_b200 import params as P
from hedgehog_lpbf_b200 import plan as PL

pytestmark = pytest.mark.gpu


def _const(nx, ny, frac=0.2):
    mat, pr = P.benchmark_material_process()
    pr.Tamb = pr.Tsub = 0.0
    dom = P.Domain(Lx=(nx - 1) * 5e-6, Ly=(ny - 1) * 5e-6, nx=nx, ny=ny)
    return mat, P.make_const(mat, pr, dom, P.dt_fraction(mat, dom, frac))


def _check(T, r):
    flat = T.ravel()
    a = int(np.argmax(flat))                         # the first of equal maxima
    assert a == 0 and np.signbit(flat[0]) and not np.signbit(T[1:-1, 1:-1]).any()
    assert r["arg"] == a, r
    assert r["tmax"] == 0.0 and np.signbit(r["tmax"])


@pytest.mark.parametrize("nx,ny", [(64, 48), (400, 300), (1024, 1024)])
@pytest.mark.parametrize("depth", [0, 1, 3])
def test_single_field(gpu, nx, ny, depth):
    from hedgehog_lpbf_b200.solver import Solver, ring_to_numpy
    n = 3
    mat, k = _const(nx, ny)
    plan = np.zeros(n, dtype=PL.TICK_DTYPE)
    s = Solver(k, bc=1, T_edge=-0.0, Tm=mat.Tm, depth=depth, T0=0.0, device="cuda:0")
    ring = s.new_ring(n)
    T = s.advance(plan, ring).cpu().numpy()
    for r in ring_to_numpy(ring):
        _check(T, r)


@pytest.mark.parametrize("nx,ny", [(200, 150), (1024, 1024)])
@pytest.mark.parametrize("depth", [0, 1, 3])
def test_zeros_of_both_signs_in_one_row(gpu, nx, ny, depth):
    """A lone -0.0 among subnormals keeps its sign (its increment underflows to
    -0.0) and stands before a +0.0 of the same row, in another lane."""
    from hedgehog_lpbf_b200.solver import Solver, ring_to_numpy
    mat, k = _const(nx, ny, 0.05)
    plan = np.zeros(1, dtype=PL.TICK_DTYPE)
    T0 = np.full((ny, nx), -5e-324)
    T0[70, 90], T0[70, 101] = -0.0, 0.0
    s = Solver(k, Tm=mat.Tm, depth=depth, T0=T0, device="cuda:0")
    ring = s.new_ring(1)
    T = s.advance(plan, ring).cpu().numpy()
    assert np.signbit(T[70, 90]) and T[70, 90] == 0.0 and not np.signbit(T[70, 101])
    r = ring_to_numpy(ring)[0]
    assert r["arg"] == int(np.argmax(T.ravel())) == 70 * nx + 90, r
    assert r["tmax"] == 0.0 and np.signbit(r["tmax"]), r


def test_batch(gpu):
    from hedgehog_lpbf_b200.batch import Batch, Scenario
    n = 3
    plan = np.zeros(n, dtype=PL.TICK_DTYPE)
    scs = []
    for nx, ny in ((64, 48), (400, 300), (1024, 1024)):
        mat, k = _const(nx, ny)
        scs.append(Scenario(k=k, plan=plan, bc=1, T_edge=-0.0, Tm=mat.Tm, T0=np.zeros((ny, nx))))
    b = Batch(scs, n, device="cuda:0")
    b.run(0, n)
    for i in range(len(scs)):
        for r in b.ring(i)[:n]:
            _check(b.field(i).cpu().numpy(), r)
    b.close()


@pytest.mark.parametrize("form", ["SolverF32", "SolverF32K"])
@pytest.mark.parametrize("depth", [1, 3])
def test_f32_fields(gpu, form, depth):
    from hedgehog_lpbf_b200 import solver as S
    n = 3
    mat, k = _const(400, 300)
    plan = np.zeros(n, dtype=PL.TICK_DTYPE)
    s = getattr(S, form)(k, bc=1, T_edge=-0.0, Tm=mat.Tm, depth=depth, T0=0.0, device="cuda:0")
    ring = s.new_ring(n)
    s.advance(plan, ring)
    for r in S.ring_to_numpy(ring):
        assert r["arg"] == 0 and r["tmax"] == 0.0, r
