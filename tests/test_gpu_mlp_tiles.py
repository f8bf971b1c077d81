"""GPU: the network's kernels around their tile of 32 samples and the 148
blocks that share them, against the float64 CPU restatement (mlp_cpu.py)."""
import numpy as np
import pytest

import mlp_cpu
from sbb import selector as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 31, 32, 33, 1000, 32 * 148, 32 * 148 + 1, 10007])
def test_gradient_and_forward_at_tile_edges(cuda, N):
    """Bounds: FP32 sums of 64 products a layer and over blocks of at most
    32 * ceil(N / 4736) samples, each rounding below 2^-24 of the running sum;
    1e-5 of the gradient's norm leaves a factor of ten."""
    rng = np.random.default_rng(N)
    X = (rng.normal(size=(N, S.N_FEATURES)) * 2 + 1).astype(np.float32)
    times = np.exp(rng.normal(size=(N, S.N_CLASSES)))
    P = S.init_params(np.concatenate([X, X + 1]), 1)
    T, W = S.targets(times), S.sample_weights(times)
    for w in (W, None):
        L, G = S.grad(P, X, T, w)
        Lc, Gc = mlp_cpu.loss_grad(P, X, T, w)
        assert abs(L - Lc) <= 1e-5 * abs(Lc)
        assert np.linalg.norm(G - Gc) <= 1e-5 * np.linalg.norm(Gc)
        assert np.all(G[:S.OFF["W1"]] == 0)
    y, _ = mlp_cpu.forward(P, X)
    assert np.allclose(S.predict(P, X), y, rtol=1e-5, atol=1e-5)
