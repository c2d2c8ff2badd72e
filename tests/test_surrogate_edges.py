# SPDX-License-Identifier: 0BSD
"""Gradients of the super-stepper at the edges of the narrow layers' tiles
(128-pixel column tiles, 8-row units, 64-pixel tiles of the input gradient)
against the FP64 restatement.  Per layer: within 3 % in norm (bf16 operands:
the bar of the gradient tests); the loss within 1 %.  The output layer's bias
gradient is one sum of residuals that may nearly cancel, so its bar is 3 % of
the sum of their magnitudes."""
import numpy as np
import pytest

from oracle import surrogate_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W", [(1, 1, 1), (1, 9, 130), (2, 17, 65), (1, 8, 128), (3, 5, 257),
                                   (1, 33, 63)])
def test_gradients_at_tile_edges(gpu, B, H, W):
    import torch
    from hedgehog_lpbf_b200 import surrogate as S
    rng = np.random.default_rng(B * 1000 + H * 10 + W)
    ps = [(torch.tensor(w).to(torch.bfloat16).double().numpy(), rng.normal(0, 0.1, b.shape))
          for w, b in S.init_params(3)]
    x = torch.tensor(rng.normal(0, 1, (B, H, W, 4)), dtype=torch.float32).to(torch.bfloat16)
    y = rng.normal(0, 1, (B, H, W)).astype(np.float32)
    net = S.Net(ps, device="cuda:0")
    loss = float(net.gradients(x.cuda().contiguous(), torch.tensor(y).cuda()).item())
    got = S.unflatten(net.grads_vector())
    want_loss, want = R.loss_and_grads(ps, x.double().numpy(), y.astype(np.float64))
    terms = np.sum(np.abs(2.0 / y.size * (R.forward(ps, x.double().numpy())[0] - y)))
    assert net.error_word() == 0
    assert abs(loss - want_loss) <= 1e-2 * want_loss
    for i, ((gw, gb), (rw, rb)) in enumerate(zip(got, want)):
        for g, r in ((gw, rw), (gb, rb)):
            g, r = np.asarray(g).ravel(), np.asarray(r).ravel()
            size = terms if i == 4 and r.size == 1 else np.linalg.norm(r)
            assert np.linalg.norm(g - r) <= 3e-2 * size + 1e-7


def test_features_in_and_around_the_source_box(gpu):
    """Every cell inside the source's reach, at its rim and off it (odd and
    even widths, beams off the field and switched off): the bf16 features of
    the plain sums."""
    import torch
    from hedgehog_lpbf_b200 import params as P
    from hedgehog_lpbf_b200 import plan as PL
    from hedgehog_lpbf_b200 import surrogate as S
    mat, pr = P.benchmark_material_process(r0=20e-6)
    for nx, ny in ((1, 1), (2, 3), (129, 70), (514, 130)):
        dom = P.Domain(Lx=max(nx - 1, 1) * 5e-6, Ly=max(ny - 1, 1) * 5e-6, nx=nx, ny=ny)
        k = P.make_const(mat, pr, P.Domain(Lx=dom.Lx, Ly=dom.Ly, nx=max(nx, 2), ny=max(ny, 2)),
                         5e-7)
        k.nx, k.ny = nx, ny
        k.dx = k.dy = 5e-6
        plan = np.zeros(S.STEPS, dtype=PL.TICK_DTYPE)
        plan["x_l"] = np.linspace(-0.3, 0.7, S.STEPS) * nx * 5e-6
        plan["y_l"] = np.linspace(0.2, 1.2, S.STEPS) * ny * 5e-6
        plan["q_scale"] = (np.arange(S.STEPS) % 4 != 3)
        T = torch.rand((ny, nx), dtype=torch.float64, device="cuda") * 1500.0 + 300.0
        got = S.features(T, k, plan).double().cpu().numpy()
        X, Y = np.arange(nx) * k.dx, (np.arange(ny) * k.dy)[:, None]
        src = np.zeros((ny, nx))
        for t in plan:
            src += (k.dt * t["q_scale"] * k.peak_S / (k.rho_cp * k.h)
                    * np.exp(-2 * k.inv_r0_sq * ((X - t["x_l"]) ** 2 + (Y - t["y_l"]) ** 2)))
        m = plan[S.STEPS // 2]
        want = np.stack([(T.cpu().numpy() - k.Tamb) / 1000.0, src / 1000.0,
                         np.clip((X - m["x_l"]) / 1e-4, -8, 8) + 0 * Y,
                         np.clip((Y - m["y_l"]) / 1e-4, -8, 8) + 0 * X], -1)
        # bf16: half a step of 2^-8 relative (and of a result a rounding away)
        assert np.max(np.abs(got - want) - 2.0 ** -8 * np.abs(want)) <= 1e-9
