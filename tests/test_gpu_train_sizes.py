"""The training kernels at the edges of their clusters: one gradient sum (one cluster of blocks), an
odd number of them, and more clusters than fit the GPU at once -- gradients against the FP64 oracle."""
import numpy as np
import pytest

from fvmic2d_gb300 import gpu, workloads as W
from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [128, 384, 16384 + 128])
def test_gradient_by_batch_size(n):
    """Each block of parameters within 2e-4 of its norm, the bound one batch's gradients are held to,
    plus what FP32 sums may lose to cancellation: chains of 128 samples and up to 129 clusters,
    257 x 2^-24 of the summed magnitudes (2 mean |err|, activations of order one)."""
    rng = np.random.default_rng(n)
    G = gpu.MicProblem(W.convection_member(4, 4, 2, 2, 1e4, 10.0, 1), capacity=64)
    p = np.zeros(M.N_PARAMS, dtype=np.float32)
    p[:M.N_TRAIN] = rng.normal(0, 0.3, M.N_TRAIN)
    p[M.OFF_NORM], p[M.OFF_NORM + 1] = 5.0, 1.5
    X = rng.uniform(-1, 1, (n, 4)).astype(np.float32)
    t = rng.normal(5.0, 1.5, n).astype(np.float32)
    g, loss = G.creep_grad(p, X, t)
    G.close()
    p64, X64, t64 = p.astype(np.float64), X.astype(np.float64), t.astype(np.float64)
    loss_o, g_o = M.loss_and_grad(p64, X64, t64, w2_bf16=True)
    assert abs(loss - loss_o) <= 1e-4 * loss_o
    err = M.forward(p64, X64, w2_bf16=True)[0] - (t64 - 5.0) / 1.5
    lost = 257 * 2.0 ** -24 * 2.0 * np.mean(np.abs(err))
    for a, b in [(M.OFF_W1, M.OFF_B1), (M.OFF_B1, M.OFF_W2), (M.OFF_W2, M.OFF_B2), (M.OFF_B2, M.OFF_W3),
                 (M.OFF_W3, M.OFF_B3), (M.OFF_B3, M.OFF_NORM)]:
        assert np.linalg.norm(g[a:b] - g_o[a:b]) <= 2e-4 * np.linalg.norm(g_o[a:b]) + np.sqrt(b - a) * lost
