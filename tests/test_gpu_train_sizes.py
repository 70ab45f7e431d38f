"""The training kernels at the edges of their tiles (128 samples) and chunks (whole tiles of 32, 456 chunks)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from oracle import mlp as M  # noqa: E402
from test_gpu_prune import _random_batch, _theta  # noqa: E402
from xkgpu import prune as P  # noqa: E402


@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 1000, 456 * 32, 456 * 32 + 1, 152 * 3 * 128 + 5])
def test_gradient_against_the_oracle(n):
    th = _theta(2)
    X = _random_batch(n, n)
    rng = np.random.default_rng(n)
    y = (rng.random(n) < 0.25).astype(np.float32)
    w = np.where(y > 0, 3.0, 1.0).astype(np.float32)
    pr = P.PairPruner(th)
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    loss, grad, logit = pr.gradient(dev(X.ravel()), dev(y), dev(w), n)
    again = pr.gradient(dev(X.ravel()), dev(y), dev(w), n)
    assert all(torch.equal(a, b) for a, b in zip((loss, grad, logit), again))
    loss_ref, grad_ref = M.loss_and_grad(th, X, y, w)
    # as the existing check: float sums, and the odd activation at a bfloat16 tie (2^-8 of one of n samples)
    assert abs(float(loss) - loss_ref) <= 1e-4 * max(loss_ref, 1e-3)
    tol = 1e-3 + 2.0**-6 / n
    assert np.max(np.abs(grad.cpu().numpy() - grad_ref)) <= tol * np.max(np.abs(grad_ref))
    p = grad.cpu().numpy()
    b4 = float(np.sum(w * (1.0 / (1.0 + np.exp(-logit.cpu().numpy().astype(np.float64))) - y)) / n)
    assert abs(p[-1] - b4) <= 1e-5 * max(abs(b4), 1e-3)
