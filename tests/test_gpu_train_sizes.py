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


def test_gradient_sums_of_many_samples():
    """No gradient is a longer chain of float additions than 1,024 samples and the chunks of a group.

    Every sample adds the same value, c up to a power of two (a zero network: sigmoid 1/2, label 0, weight c).  It
    loses almost half a last place in every addition to a sum between 4,096 c and 8,192 c: chains that go on that far
    are off by 1.3e-4.  Bound: a chain of k additions is off by at most k 2^-24 of its sum.
    """
    n = 1 << 22
    th = np.zeros(P.NPARAM, np.float32)
    th[-129:-65] = 1.0  # the last activations: 1
    pr = P.PairPruner(th)
    c = np.float32(1.0 + 2.0**-12 - 2.0**-23)
    X = torch.zeros(8 * n, device="cuda")
    y = torch.zeros(n, device="cuda")
    w = torch.full((n,), float(c), device="cuda")
    _, grad, _ = pr.gradient(X, y, w, n)
    g = grad.cpu().numpy()
    want = 0.5 * float(c)  # the mean of c / 2
    chunks = n // 1024
    tol = (1024 + chunks // 8 + 8) * 2.0**-24
    assert abs(g[-1] - want) <= tol * want  # b4
    assert np.max(np.abs(g[-65:-1] - want)) <= tol * want
