"""The correctly rounded double divide and square root of the kernels, bit for bit against the operators, on the
operands whose results lie next to a rounding tie (random ones never do).

The headers' functions are compiled into a small library of the test's own.
"""

from __future__ import annotations

import ctypes as C
import math
import random
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from xkgpu import build as B  # noqa: E402

SOURCE = """
#include "xk_common.cuh"
xk_status xk_set_cuda_error(cudaError_t, const char*, int) { return XK_ERR_CUDA; }
__global__ void k_div(long long n, const double* x, const double* d, double* q, double* want) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  q[i] = div64(x[i], d[i]);
  want[i] = x[i] / d[i];
}
__global__ void k_sqrt(long long n, const double* x, double* q, double* want) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  q[i] = sqrt64(x[i]);
  want[i] = sqrt(x[i]);
}
__global__ void k_div_unit(long long n, const double* x, const double* d, double* q, double* want) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  bool sure;
  const double y = div_next_to_one64(x[i], d[i], units_from_one64(d[i]), sure);
  q[i] = !next_to_one64(d[i]) ? -1.0 : sure ? y : x[i] / d[i];
  want[i] = x[i] / d[i];
}
extern "C" int t_div_unit(long long n, const double* x, const double* d, double* q, double* want) {
  k_div_unit<<<(unsigned)((n + 255) / 256), 256>>>(n, x, d, q, want);
  return (int)cudaDeviceSynchronize();
}
extern "C" int t_div(long long n, const double* x, const double* d, double* q, double* want) {
  k_div<<<(unsigned)((n + 255) / 256), 256>>>(n, x, d, q, want);
  return (int)cudaDeviceSynchronize();
}
extern "C" int t_sqrt(long long n, const double* x, double* q, double* want) {
  k_sqrt<<<(unsigned)((n + 255) / 256), 256>>>(n, x, q, want);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("device_math")
    (d / "t.cu").write_text(SOURCE)
    subprocess.run([B.nvcc(), *B.ARCH, *B.FLAGS, "-I", str(B.SRC), "-I", str(B.INCLUDE), "-shared", "-o",
                    str(d / "t.so"), str(d / "t.cu")], check=True, capture_output=True)
    return C.CDLL(str(d / "t.so"))


def _run(fn, *arrays):
    dev = [torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda") for a in arrays]
    got, want = torch.zeros_like(dev[0]), torch.zeros_like(dev[0])
    args = [C.c_void_p(t.data_ptr()) for t in (*dev, got, want)]
    torch.cuda.synchronize()
    assert fn(C.c_longlong(dev[0].numel()), *args) == 0
    bad = (got.view(torch.int64) != want.view(torch.int64)).cpu().numpy()
    assert not bad.any(), (int(bad.sum()), [[float(v).hex() for v in np.asarray(a)[bad][:3]] for a in arrays])


def _hard_quotients():
    """(x, d): integers of 53 bits with x 2^s nearest to an odd multiple of d / 2, and divisors at a binade's ends."""
    rnd = random.Random(7)
    pairs = []
    top = 1 << 53
    for k in range(1, 300):
        for d in (top - k, (1 << 52) + k - 1):
            for x in [1 << 52, (1 << 52) + 1, top - 1, 3 << 51] + [d + j for j in range(-4, 5)] + [
                    rnd.getrandbits(52) | 1 << 52 for _ in range(4)]:
                if 1 << 52 <= x < top:
                    pairs.append((x, d))
    for t in range(60000):
        d = (top - 1 - 2 * rnd.randrange(1 << rnd.randrange(1, 46)), (rnd.getrandbits(46) | 127 << 46) | 1,
             rnd.getrandbits(52) | 1 << 52 | 1)[t % 3]
        if 1 << 52 <= d < top:
            for s in (53, 54):
                inv = pow(2, -s, d)
                pairs += [(x, d) for x in (inv * c % d for c in (1, -1, 3, -3)) if x >> 52 == 1]
    return np.array(pairs, dtype=np.float64).T


def test_quotients_next_to_ties(lib):
    x, d = _hard_quotients()
    for sx, sd in ((1.0, 1.0), (-(2.0**-60), 2.0**-50), (2.0**40, -(2.0**-70))):
        _run(lib.t_div, x * sx, d * sd)


def test_quotients_of_special_operands(lib):
    v = np.array([0.0, -0.0, 1.0, -1.0, 2.0**-300, 2.0**300, 2.0**-1074, 2.0**-1022, 1.7e308, np.inf, -np.inf,
                  1.0 - 2.0**-53, 2.0 - 2.0**-52, (2.0 - 2.0**-52) * 2.0**-300, 3.0])
    x, d = np.meshgrid(v, v)
    x, d = x.ravel(), d.ravel()
    with np.errstate(all="ignore"):
        keep = ~np.isnan(np.divide(x, d, where=d != 0, out=np.full(x.shape, np.nan)))
    # a zero over a negative divisor is not asked for: every divisor of the kernels is positive
    keep &= ~((x == 0) & (d < 0))
    _run(lib.t_div, x[keep], d[keep])


def test_divisors_next_to_one(lib):
    """Every divisor of the range over values of few bits (which tie), neighbours of ties, powers of two and their
    neighbours, values at random and at the ends of the double range."""
    rng = np.random.default_rng(5)
    m = [np.arange(1 << 52, (1 << 53) + 1, 1 << 40), (1 << 52) + np.arange(100), (1 << 53) - np.arange(100),
         rng.integers(1 << 52, 1 << 53, 20000)]
    for n in range(1, 17):  # m n = 2^52 + j modulo 2^53: within j units of a tie
        for j in (0, 1, -1, 2, -2, 15, -15, 255, -255, 256, -256, 257, -257, 511, 513, -511, -513):
            t = ((np.arange(n, 2 * n + 2, dtype=object) << 53) + (1 << 52) + j) // n
            m.append(np.array([x + y for x in t for y in (-1, 0, 1) if 1 << 52 <= x + y <= 1 << 53], dtype=np.int64))
    v = np.concatenate(m).astype(np.float64) * 2.0**-53
    v = np.concatenate([v, -v, v * 2.0**-900, v * 2.0**-1000, v * 2.0**-1040, v * 2.0**1000, v * 2.0**1023 * (2.0 - 2.0**-52),
                        [0.0, -0.0, 2.0**-1074, 2.0**-1022]])
    v = v[np.isfinite(v)]
    for d in [1.0 - k * 2.0**-53 for k in range(17)] + [1.0 + k * 2.0**-52 for k in range(8)]:
        _run(lib.t_div_unit, v, np.full_like(v, d))


def test_square_roots_next_to_ties(lib):
    xs = []
    for shift, lo, hi in ((52, 1 << 104, 1 << 105), (53, 1 << 105, 1 << 106)):
        for c in range(-100, 102, 2):
            roots = [0, 1]  # of N (N + 1) = c modulo 2^shift
            for k in range(1, shift + 1):
                roots = sorted({t for r in roots for t in (r, r + (1 << (k - 1)))
                                if t < (1 << k) and (t * (t + 1) - c) % (1 << k) == 0})
            for r in roots:
                for n in (r, r + (1 << shift)):
                    x = n * (n + 1) - c
                    if lo <= x < hi and x % (1 << shift) == 0:
                        xs.append(math.ldexp(x >> shift, shift - 104))
    xs = np.array(xs)
    _run(lib.t_sqrt, np.concatenate([xs, xs * 0.25, xs * 2.0**100, xs * 2.0**-200]))
