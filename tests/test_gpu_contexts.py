"""What the library keeps between calls (read-back buffer and event, fork and join events, scratch pool) is of the
context it was made in: detection and assembly in several contexts of a device, in turn, after one has gone and from
another thread.  In a process of its own, through the driver API, without torch."""

from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

SCRIPT = """
import ctypes as C, sys, threading
sys.path[:0] = [{root!r}, {pkg!r}]
import numpy as np
from oracle import contact as oc
from xkgpu import _lib as L

cu = C.CDLL("libcuda.so.1")
def ok(code):
    assert code == 0, code
ok(cu.cuInit(0))

def to_dev(a):
    p = C.c_uint64()
    ok(cu.cuMemAlloc_v2(C.byref(p), C.c_size_t(max(a.nbytes, 16))))
    ok(cu.cuMemcpyHtoD_v2(p, a.ctypes.data_as(C.c_void_p), C.c_size_t(a.nbytes)))
    return C.c_void_p(p.value)

rng = np.random.default_rng(3)
n = 60
X = rng.uniform(0.0, 3.0, (n, 1, 3)) + np.stack([np.zeros((n, 3)), rng.normal(0.0, 0.5, (n, 3))], 1)
X, conn, radii = X.reshape(-1, 3), np.arange(2 * n, dtype=np.int32).reshape(-1, 2), np.full(n, 0.3)
lo, hi = oc.segment_aabbs(X, conn, radii, 0.0)
i, j = np.triu_indices(n, 1)
want = np.stack([i, j], 1)[np.all((lo[i] <= hi[j]) & (lo[j] <= hi[i]), axis=1)]
assert 20 < len(want) < n * n

def work():
    m = L.Mesh(2 * n, n, to_dev(X), to_dev(conn), to_dev(radii))
    u = to_dev(np.zeros(12 * n))
    out = to_dev(np.zeros(2 * n * n, np.int32))
    nk, nr, np_ = C.c_int64(), C.c_int64(), C.c_int64()
    for _ in range(2):
        L.call("xk_broadphase", C.byref(m), u, C.byref(L.BPParams(0.0, 1, 0, 0, 0.0)), out, n * n, C.byref(nk),
               C.byref(nr), C.byref(np_), None)
        assert nr.value == len(want) == nk.value
        got = np.zeros((nk.value, 2), np.int32)
        ok(cu.cuMemcpyDtoH_v2(got.ctypes.data_as(C.c_void_p), out, C.c_size_t(got.nbytes)))
        assert np.array_equal(got, want)
    # a mesh without elements: what is left of an assembly is its forks and joins
    empty = [L.Mesh(), L.Section(), L.BeamPlan(), L.ContactPattern(), L.ContactParams(), L.Pairs()]
    a = L.Assembly(*(C.addressof(x) for x in empty), None, u)
    a.R, a.precision = u, L.XK_FP64
    L.call("xk_assemble", C.byref(a), u, None, None, None, None)
    ok(cu.cuCtxSynchronize())

def context():
    c = C.c_void_p()
    ok(cu.cuCtxCreate_v2(C.byref(c), 0, 0))  # and makes it current
    return c

a = context()
work()
b = context()
work()
ok(cu.cuCtxSetCurrent(a))
work()
ok(cu.cuCtxDestroy_v2(b))
c = context()
work()
ok(cu.cuCtxSetCurrent(a))
work()
errors = []
def other():
    try:
        for x in (c, a):
            ok(cu.cuCtxSetCurrent(x))
            work()
    except BaseException as e:
        errors.append(e)
t = threading.Thread(target=other)
t.start()
t.join()
assert not errors, errors
L.call("xk_scratch_trim", 0)
print("contexts ok")
"""


def test_calls_in_several_contexts():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=str(ROOT), pkg=str(ROOT / "xkep-cae_gb300"))],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "contexts ok" in r.stdout, r.stderr[-3000:]
