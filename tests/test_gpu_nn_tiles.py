"""The network's forward and gradient kernels (rtg_nn.cu) against the oracle at
the edges of their tiles: one row, one row less and more than a 64-row tile, and
one less, as many and one more tile than there are CTAs.

Tolerances as in the comparisons with the oracle at one size: FP32 sums of at most
128 terms, 1e-5 of the largest output and of the loss, 1e-4 of the gradient."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 63, 65, 64 * 152 - 64, 64 * 152, 64 * 152 + 1])
def test_forward_and_gradient_match_oracle(rows):
    import torch
    from oracle import nn_oracle as NO
    from rtg import learned as LN
    rng = np.random.default_rng(rows)
    F = rng.standard_normal((rows, NO.N_IN)).astype(np.float32)
    F[:, :2] = np.abs(F[:, :2])        # optical thickness and albedo: the gate is positive
    M = rng.standard_normal((rows, NO.N_MOM)).astype(np.float32)
    B, t = rng.standard_normal((rows, 3, 5)), rng.standard_normal((rows, 5))
    G, q = B @ B.transpose(0, 2, 1), np.einsum("rij,rj->ri", B, t)
    S = np.zeros((rows, 12), dtype=np.float32)
    S[:, :10] = np.stack([G[:, 0, 0], G[:, 0, 1], G[:, 0, 2], G[:, 1, 1], G[:, 1, 2], G[:, 2, 2],
                          q[:, 0], q[:, 1], q[:, 2], (t * t).sum(1)], axis=1) / rows
    p = np.concatenate([rng.standard_normal(int(np.prod(shp))) * (0.3 if i == 0 else 0.1)
                        for i, (_, shp) in enumerate(NO.SHAPES)]).astype(np.float32)
    dev = "cuda"
    P, Ft = torch.as_tensor(p, device=dev), torch.as_tensor(F, device=dev)
    O = LN.forward(P, Ft).cpu().numpy()
    ref, _ = NO.forward(NO.device_params(p), F.astype(np.float64))
    assert np.abs(O - ref).max() <= 1e-5 * max(1.0, np.abs(ref).max())
    tr = LN.Trainer(dev)
    Mt, St = torch.as_tensor(M, device=dev), torch.as_tensor(S, device=dev)
    loss, grad = (a.clone() for a in tr.loss_grad(P, Ft, Mt, St))
    lo, go = NO.loss_grad(NO.device_params(p), F.astype(np.float64), M.astype(np.float64),
                          S.astype(np.float64)[:, :10])
    assert abs(float(loss[0]) - lo) <= 1e-5 * abs(lo)
    g = grad.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(g - go) <= 1e-4 * np.linalg.norm(go)
    again = tr.loss_grad(P, Ft, Mt, St)
    assert torch.equal(loss, again[0]) and torch.equal(grad, again[1])
