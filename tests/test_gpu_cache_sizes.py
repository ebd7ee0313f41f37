"""Radiance-cache kernels at the sizes where their tiling changes: one row,
around a 128-row tile, around one pass of tiles over all pipelines (5 per SM in
inference, 2 per SM in training, 148 SMs), and rows that are not numbers."""
import numpy as np
import pytest
import torch

from oracle import mlp

pytestmark = pytest.mark.gpu

SM = 148


def _batch(n, seed):
    rng = np.random.default_rng(seed)
    x = mlp.bf16(rng.uniform(-1, 1, (n, 64)).astype(np.float32))
    t = np.zeros((n, 4), np.float32)
    t[:, :3] = rng.uniform(0.05, 2.0, (n, 3))
    return x, t, torch.from_numpy(mlp.bf16_bits(x).view(np.int16).copy()).cuda(), torch.from_numpy(t).cuda()


@pytest.mark.parametrize('n', [1, 127, 128, 129, 5 * 128 + 1, 5 * SM * 128, 5 * SM * 128 + 1])
def test_forward_sizes(vb, gpu_ctx, n):
    cache = vb.RadianceCache(gpu_ctx, seed=13)
    x, _, xd, _ = _batch(n, 5)
    out = torch.full((n + 1, 4), 7.0, device='cuda')
    cache.infer(xd.data_ptr(), n, out.data_ptr())
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert np.all(got[n] == 7.0)  # nothing written past the end
    _, y = mlp.forward(cache.weights(), x)
    # A different FP32 accumulation order can move a hidden activation by one
    # BF16 unit (2^-8), diluted over 64 inputs.
    assert np.abs(got[:n, :3] - y).max() <= 2e-2 * np.abs(y).max()
    assert np.mean(np.abs(got[:n, :3] - y) <= 1e-3 * (1 + np.abs(y))) >= 0.99
    cache.close()


def test_forward_nan_rows_are_isolated(vb, gpu_ctx):
    cache = vb.RadianceCache(gpu_ctx, seed=13)
    n = 300
    _, _, xd, _ = _batch(n, 6)
    ref = torch.zeros((n, 4), device='cuda')
    cache.infer(xd.data_ptr(), n, ref.data_ptr())
    bad = xd.clone()
    rows = [0, 127, 128, 299]
    for r in rows:
        bad[r, 5] = 0x7fc0  # BF16 NaN
    out = torch.zeros((n, 4), device='cuda')
    torch.cuda.synchronize()
    cache.infer(bad.data_ptr(), n, out.data_ptr())
    torch.cuda.synchronize()
    ok = torch.ones(n, dtype=torch.bool)
    ok[rows] = False
    assert torch.equal(out.cpu()[ok], ref.cpu()[ok])
    # ReLU takes NaN to zero, so every hidden activation of such a row is zero.
    assert torch.all(out.cpu()[rows] == 0.0)
    cache.close()


@pytest.mark.parametrize('n', [1, 127, 128, 129, SM * 128, SM * 128 + 1, 2 * SM * 128 + 1, 3 * SM * 128 + 1])
def test_gradient_sizes(vb, gpu_ctx, n):
    cache = vb.RadianceCache(gpu_ctx, seed=17)
    w = cache.weights()
    x, t, xd, td = _batch(n, 7)
    for _ in range(2):  # a second call starts from a cleared gradient
        cache.train(xd.data_ptr(), td.data_ptr(), n, update=False)
    g, loss = cache.gradient()
    loss_ref, g_ref, _ = mlp.loss_and_grad(w, x, t)
    assert abs(loss - loss_ref) <= 5e-3 * loss_ref
    # One BF16 unit is 2^-8; with few samples single roundings show.
    for a, b in zip(mlp.split(g), mlp.split(g_ref)):
        assert np.linalg.norm(a - b) <= 2e-2 * np.linalg.norm(b)
    np.testing.assert_array_equal(cache.weights(), w)
    cache.close()
