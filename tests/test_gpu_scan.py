"""The one-pass scan where its tiles give up waiting and sum what lies before them themselves (a limit of no polls at
all), and its entry's refusal of overlapping arrays.  The scan's sources are compiled into a library of the test's."""

from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from xkgpu import _lib as L  # noqa: E402
from xkgpu import build as B  # noqa: E402

SOURCE = """
#include "util.cu"
extern "C" int t_scan(const int32_t* in, int32_t* out, long long n, int64_t* sum) {
  XkScratch S(0);
  int64_t* sums;
  int* words;
  XK_TRY(S.get(&sums, scan_sums(n, 1)));
  XK_TRY(S.get(&words, scan_words(n, 1)));
  XK_CUDA(cudaMemsetAsync(words, 0, sizeof(int) * scan_words(n, 1), 0));
  XK_TRY((scan_launch<ScanI32, 0>(ScanI32{in, out, n, sum}, n, 1, sums, words, 0)));
  XK_CUDA(cudaDeviceSynchronize());
  return XK_OK;
}
extern "C" int t_entry(const int32_t* in, int32_t* out, long long n, int64_t* sum) {
  XK_TRY(xk_exclusive_scan_i32(in, out, n, sum, 0));
  XK_CUDA(cudaDeviceSynchronize());
  return XK_OK;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("scan")
    (d / "t.cu").write_text(SOURCE)
    subprocess.run([B.nvcc(), *B.ARCH, *B.FLAGS, "-I", str(B.SRC), "-I", str(B.INCLUDE), "-shared", "-o",
                    str(d / "t.so"), str(d / "t.cu")], check=True, capture_output=True)
    return C.CDLL(str(d / "t.so"))


def _call(fn, a, out, n, total):
    torch.cuda.synchronize()
    return fn(C.c_void_p(a.data_ptr()), C.c_void_p(out.data_ptr()), C.c_longlong(n), C.c_void_p(total.data_ptr()))


@pytest.mark.parametrize("n", [1, 2047, 2049, 300001, 1500000])
def test_prefixes_without_waiting(lib, n):
    h = np.random.default_rng(n).integers(0, 7, n).astype(np.int32)
    a = torch.as_tensor(h, device="cuda")
    want = np.concatenate([[0], np.cumsum(h[:-1])])
    for fn in (lib.t_scan, lib.t_entry):
        out = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        total = torch.zeros(1, dtype=torch.int64, device="cuda")
        assert _call(fn, a, out, n, total) == L.XK_OK
        assert np.array_equal(out.cpu().numpy(), want) and int(total) == int(h.sum())


def test_overlapping_arrays_are_refused(lib):
    n = 5000
    a = torch.ones(2 * n, dtype=torch.int32, device="cuda")
    total = torch.zeros(1, dtype=torch.int64, device="cuda")
    for shift in (0, 1, n - 1):
        assert _call(lib.t_entry, a, a[shift:], n, total) == L.XK_ERR_ARG
        assert _call(lib.t_entry, a[shift:], a, n, total) == L.XK_ERR_ARG
    assert _call(lib.t_entry, a, a[n:], n, total) == L.XK_OK
    assert torch.equal(a[n:], torch.arange(n, dtype=torch.int32, device="cuda")) and torch.all(a[:n] == 1)
