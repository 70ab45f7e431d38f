"""The launch-shape tuner has the kernels' own choice among its candidates and can come back to it."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from xkgpu import workloads as W  # noqa: E402
from xkgpu.engine import AssemblyEngine  # noqa: E402


@pytest.mark.parametrize("fastest", [0, 1, 2])
def test_default_block_is_a_candidate(fastest):
    w = W.config_workload("strand7", seed=0)
    st = w.strand
    eng = AssemblyEngine(st.coords, st.conn, st.radii, w.section, precision="mixed", **w.engine_kwargs())
    u = torch.as_tensor(w.u, device="cuda")
    eng.detect(u)
    eng.assemble(u, u)
    R = eng.R.clone()
    eng.tune(reps=1)
    tried = []

    def timed(fn, reps):  # what one candidate after the other takes
        fn(torch.cuda.current_stream())
        tried.append(eng.pairs32.c.block)
        return 1.0 if len(tried) == fastest + 1 else 2.0

    eng._time_calls = timed
    shapes = eng._tune_shapes(1)["pair_block"]
    assert shapes["default"] == 0 and set(shapes["times_ms"]) >= {0, 128, 256}
    assert shapes["chosen"] == tried[fastest] == eng._pair_block
    eng.assemble(u, u)
    assert eng.pairs32.c.block == shapes["chosen"]
    assert torch.allclose(eng.R, R, rtol=1e-6, atol=1e-6 * float(R.abs().max()))
