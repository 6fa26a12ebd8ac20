"""The fused training and inference kernels where a CTA takes several tiles of
128 rows and where the last tile is ragged: gradients of batches on both sides
of one tile per CTA (152 CTAs) against the float64 restatement with the same
bfloat16 roundings, equal gradients from equal calls, and predictions of row
counts around a tile and around a full round of tiles.  Tolerances are those
of the one-tile cases: fp32 sums of at most 2^15 rows stay far inside them."""
import numpy as np
import pytest

from oracle import mlp

pytestmark = pytest.mark.gpu


def _rows(torch, n, seed):
    g = torch.Generator().manual_seed(seed)
    feat = torch.randn(n, 5, generator=g)
    lab = 0.3 * torch.randn(n, generator=g) + feat[:, 0] * 0.2
    return feat.cuda(), lab.cuda()


@pytest.mark.parametrize("batch", [256, 152 * 128, 152 * 128 + 256, 1 << 15])
def test_gradients(fvs, torch_cuda, batch):
    feat, lab = _rows(torch_cuda, batch, batch)
    net = fvs.LearnedGuess(seed=3)
    g, loss = net.gradients(feat, lab, batch)
    g2, loss2 = net.gradients(feat, lab, batch)
    np.testing.assert_array_equal(g, g2)
    assert loss == loss2
    p = net.master().astype(np.float64)
    rloss, rg = mlp.loss_and_grad(p, feat.cpu().numpy(), lab.cpu().numpy().astype(np.float64),
                                  bf16_operands=True)
    assert abs(loss - rloss) <= 1e-4 * rloss
    for lo, hi in [(mlp.OFF_W1, mlp.OFF_B1), (mlp.OFF_B1, mlp.OFF_W2), (mlp.OFF_W2, mlp.OFF_B2),
                   (mlp.OFF_B2, mlp.OFF_W3), (mlp.OFF_W3, mlp.OFF_B3),
                   (mlp.OFF_B3, mlp.N_PARAMS)]:
        assert np.linalg.norm(g[lo:hi] - rg[lo:hi]) < 5e-3 * np.linalg.norm(rg[lo:hi])


@pytest.mark.parametrize("n", [1, 127, 128, 129, 3 * 152 * 128 + 5])
def test_predictions(fvs, torch_cuda, n):
    torch = torch_cuda
    feat, _ = _rows(torch, n, n)
    net = fvs.LearnedGuess(seed=4)
    y = torch.full((n + 1,), 7.0, dtype=torch.float32, device="cuda")
    net.predict(feat, y[:n])
    torch.cuda.synchronize()
    ref = mlp.forward(net.master().astype(np.float64), feat.cpu().numpy(), bf16_operands=True)
    err = np.abs(y[:n].cpu().numpy() - ref)
    assert err.max() < 2e-3 * max(1.0, np.abs(ref).max())
    assert float(y[n]) == 7.0  # nothing past the last row
