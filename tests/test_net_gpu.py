"""The fused training step (forward, loss, backward, weight gradients per
tile of 128 rows) against the FP64 evaluation of the quantised network, at
the edges of its tiling: one row, one full tile, more tiles than CTAs, padded
rows, no weights.  Tolerance as for the network's other gradient test: every
product's operands are bf16 (2^-9 relative), twice along the backward chain,
so a few per cent of a block's largest entry bounds its sums."""
import numpy as np
import pytest

from tests.test_mlp_gpu import oracle_forward, oracle_grad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("n,n_pad", [(1, 128), (128, 128), (129, 256), (149 * 128 - 5, 149 * 128),
                                     (300 * 128 - 200, 300 * 128)])
@pytest.mark.parametrize("weighted", [True, False])
def test_training_step_at_tile_edges(cuda, order, n, n_pad, weighted):
    import torch
    from devil_ray_b200 import learned as LG
    model = LG.GuessMLP(cuda, seed=order, order=order)
    lay = model.layout
    g = torch.Generator().manual_seed(n + order)
    model.params += ((torch.rand(lay.n_params, generator=g) - 0.5) * 0.02).to(cuda)
    model.prepare()
    X = torch.zeros((n_pad, lay.n_in_pad))
    X[:n, :lay.n_in] = torch.rand((n, lay.n_in), generator=g) * 2 - 1
    X = X.to(cuda).bfloat16()
    label = torch.rand((n, 3), generator=g).to(cuda)
    w = (torch.rand(n, generator=g) > 0.3).float().to(cuda) if weighted else None
    grad, loss = model.grad(X, label, n, w)
    again, _ = model.grad(X, label, n, w)
    y = model.forward(X, n)
    torch.cuda.synchronize()
    model.check_err()
    assert torch.equal(grad, again)            # slots are added in order
    p, Xn = model.params.cpu().numpy(), X.float().cpu().numpy()[:n]
    wn = np.ones(n) if w is None else w.cpu().numpy().astype(np.float64)
    want, want_loss = oracle_grad(p, Xn, label.cpu().numpy().astype(np.float64), wn, n, order)
    *_, want_y = oracle_forward(p, Xn, order)
    assert np.abs(y.cpu().numpy() - want_y).max() < 2e-3 * max(1.0, np.abs(want_y).max())
    got = grad.cpu().numpy()
    at = {"W1": (lay.W1, lay.B1), "b1": (lay.B1, lay.W2), "W2": (lay.W2, lay.B2),
          "b2": (lay.B2, lay.W3), "W3": (lay.W3, lay.B3), "b3": (lay.B3, lay.n_params)}
    for k, (a, b) in at.items():
        ref = want[k].reshape(-1)
        off = np.abs(got[a:b] - ref).max() / max(np.abs(ref).max(), 1e-12)
        assert off < 3e-2 or (wn.sum() == 0 and np.all(got[a:b] == 0)), f"{k}: {off:.2e}"
    assert abs(float(loss.item()) - want_loss) <= 1e-3 * max(1.0, want_loss)
