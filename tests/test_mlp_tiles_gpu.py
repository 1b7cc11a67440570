"""The MLP training kernels at the edges of their tiles: sample counts around
one tile (32), one tile per block (148 tiles) and several, with and without
row indices, against a float64 evaluation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTS = [1, 31, 32, 33, 127, 129, 148 * 32, 148 * 32 + 1, 3 * 148 * 32 - 5]


@pytest.mark.parametrize("indexed", [False, True], ids=["rows", "indexed"])
@pytest.mark.parametrize("n", COUNTS)
def test_grad_and_forward_at_tile_edges(gpu, n, indexed):
    import torch
    from flowcraft_b200.closure_train import MlpTrainer, he_init
    from oracle.mlp_oracle import forward, loss_grad
    rng = np.random.default_rng(n)
    total = n + 50 if indexed else n
    x = rng.normal(size=(total, 5)).astype(np.float32)
    y = rng.normal(size=total).astype(np.float32)
    idx = rng.permutation(total)[:n] if indexed else np.arange(n)
    p = he_init(3)
    p[160:192] = rng.normal(0, 0.1, 32)
    p[1216:1248] = rng.normal(0, 0.1, 32)
    tr = MlpTrainer(p)
    tx, ty = torch.tensor(x, device="cuda"), torch.tensor(y, device="cuda")
    loss, g = tr.grad(tx, ty, torch.tensor(idx, device="cuda") if indexed else None)
    l_ref, g_ref = loss_grad(p.astype(np.float64), x[idx].astype(np.float64), y[idx].astype(np.float64))
    want, (z1, _, z2, _) = forward(p.astype(np.float64), x.astype(np.float64))
    # float rounding of the outputs moves the error e = out - y by about 1e-6
    # of |out|, and with it the loss and every gradient; sums add a small
    # multiple of u; a unit whose z lies within rounding of zero may switch,
    # which moves the gradient by that sample's share
    scale = 1.0 + np.abs(want[idx]).max() / np.sqrt(l_ref)
    near = (np.abs(z1[idx]) < 2e-6).sum() + (np.abs(z2[idx]) < 2e-6).sum()
    assert abs(loss.item() - l_ref) < 4e-6 * scale * l_ref
    assert np.abs(g.cpu().numpy() - g_ref).max() < 2e-5 * scale * np.abs(g_ref).max() + 50.0 * near / n
    first = g.clone()
    tr.grad(tx, ty, torch.tensor(idx, device="cuda") if indexed else None)
    assert torch.equal(first, tr.g)  # deterministic
    out = tr.predict(tx).cpu().numpy()
    assert np.abs(out - want).max() < 1e-5 * max(1.0, np.abs(want).max())
