"""The training kernels at the edges of their chunks (32 samples) and of the
rows that the update sums at a time (256 chunks), against the FP64 oracle.
Tolerance as in test_mlp_gpu.py: |g - g_ref| <= 2e-4 * max|g_ref| + 1e-6 per
parameter, loss to 1e-5 relative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 15, 17, 32, 64, 8160, 8192, 8193, 16385])
def test_gradient_at_chunk_edges(song, n):
    from oracle import mlp_oracle as M
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 5)).astype(np.float32)
    y = (x[:, 0] - 0.5 * x[:, 3] > 0).astype(np.float32)
    w = rng.uniform(0.5, 2.0, n).astype(np.float32)
    p = song.mlp_init(seed=n)
    g, loss = song.mlp_grad(x, y, p, w)
    l_ref, g_ref = M.loss_and_grad(x, y, p, w)
    assert abs(loss - l_ref) <= 1e-5 * max(1.0, abs(l_ref))
    assert np.abs(g - g_ref).max() <= 2e-4 * np.abs(g_ref).max() + 1e-6


def test_training_in_several_row_groups(song):
    """Batches of more than 256 chunks, the last one partial: one step of the
    training equals Adam's first step on the gradient call's result."""
    import torch
    n = 9001
    rng = np.random.default_rng(3)
    x = rng.standard_normal((n, 5)).astype(np.float32)
    y = (x[:, 1] > 0.2).astype(np.float32)
    p0 = song.mlp_init(seed=3)
    g, loss = song.mlp_grad(x, y, p0)
    dx, dy, dp = (torch.from_numpy(a.copy()).cuda() for a in (x, y, p0))
    dl = torch.zeros(1, dtype=torch.float32, device="cuda")
    song.mlp_train_device(dx.data_ptr(), dy.data_ptr(), 0, n, 0, 1, n, 1e-2, dp.data_ptr(), dl.data_ptr(), 0)
    step = 1e-2 * g.astype(np.float64) / (np.abs(g.astype(np.float64)) + 1e-8)
    got = p0.astype(np.float64) - dp.cpu().numpy().astype(np.float64)
    # the step is lr times g / (|g| + eps): FP32 rounding of p (|p| < 2: 2^-23)
    # and of the moments' ratio (2^-20 of lr)
    assert np.abs(got - step).max() <= 2.0 ** -22 + 1e-2 * 2.0 ** -18
    assert float(dl.cpu()[0]) == loss
