"""Tensor-core scoring at the edges of its tiles, CTAs and tile groups."""

import numpy as np
import pytest

from oracle import mlp as M

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if torch.cuda.is_available():
    from xkgpu.prune import PairPruner, init_params

ROUND = 128 * 152  # one tile on every SM of a full GPU


@pytest.mark.parametrize("n", [1, 127, 128, 129, ROUND - 1, ROUND + 1, 5 * ROUND, 5 * ROUND + 1, 11 * ROUND + 5])
def test_scores_at_tile_edges(n):
    th = (init_params(2) + np.random.default_rng(2).normal(0.0, 0.02, M.N_PARAMS)).astype(np.float32)
    X = np.random.default_rng(n).normal(0.0, 1.0, (n, 8)).astype(np.float32)
    pr = PairPruner(th)
    feat = torch.as_tensor(X.ravel(), device="cuda")
    got = pr.logits(feat, n)
    assert not pr.tcgen05_failed() and got.numel() >= n
    # a row's score does not depend on its tile: the last rows alone give the same bits
    k = min(n, 200)
    tail = pr.logits(feat[8 * (n - k):].clone(), k)
    assert torch.equal(got[n - k:n], tail[:k])
    exp, _ = M.forward(th, X)
    scale = max(1.0, float(np.max(np.abs(exp))))
    # a float sum in another order may round an activation to the neighbouring bfloat16 value
    d = np.abs(got[:n].cpu().numpy() - exp)
    assert np.mean(d > 1e-5 * scale) <= 0.01 or n < 200
    assert np.max(d) <= 2.0**-6 * scale
