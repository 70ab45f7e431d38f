"""The detection's scratch pool: two threads on two streams at once, and giving it back in between."""

from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from xkgpu import _lib as L  # noqa: E402
from xkgpu import workloads as W  # noqa: E402
from xkgpu.engine import AssemblyEngine  # noqa: E402


def _detections(name, precision, out, errors):
    try:
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            w = W.config_workload(name, seed=1)
            st = w.strand
            eng = AssemblyEngine(st.coords, st.conn, st.radii, w.section, precision=precision, **w.engine_kwargs())
            for k in range(8):
                u = torch.as_tensor(w.u * (1.0 + 0.2 * k), device="cuda")
                eng.detect(u)
                if k % 3 == 2:
                    L.call("xk_scratch_trim", 0)
            eng.assemble(u, u)
            stream.synchronize()
            h = eng.pair_state()
            out.append({**{k: h[k] for k in ("ea", "eb", "gap", "status", "t1")},
                        "col": eng.pattern.col[: eng.pattern.nnzb].cpu().numpy(),
                        "bcodes": eng.pattern.bcodes[: 4 * eng.pattern.nnzb].cpu().numpy()})
    except Exception as e:  # noqa: BLE001 - raised in the test's own thread
        errors.append(e)


def test_two_threads_detect_at_once():
    jobs = [("strand37", "mixed"), ("strand7", "fp64"), ("strand37c", "fp64")]
    alone, together, errors = [], [[] for _ in jobs], []
    for name, precision in jobs:
        _detections(name, precision, alone, errors)
    threads = [threading.Thread(target=_detections, args=(*job, together[k], errors)) for k, job in enumerate(jobs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for a, (b,) in zip(alone, together):
        for k in a:
            assert np.array_equal(a[k], b[k]), k


def test_trim_refuses_a_negative_size():
    assert L.call("xk_scratch_trim", -1, allow=(L.XK_ERR_ARG,)) == L.XK_ERR_ARG
