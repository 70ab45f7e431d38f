"""The assembly as one call: the same pair state and records, bit for bit, as the pair entry points on their own
(which form the segments' values in every pair), on any stream, and the residual without tangent as with it."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from xkgpu import workloads as W  # noqa: E402
from xkgpu.engine import AssemblyEngine  # noqa: E402

COAT = dict(stiffness=1e4, damping=50.0, mu=0.2, k_t_ratio=0.5, dt=0.1)


def _engine(kind, precision):
    if kind == "batch":
        w = W.batch_workload(n_strands=3, d=2.0, pitch=40.0)
    else:
        w = W.config_workload("strand37" if kind == "strand37" else "strand7", seed=3)
    kw = w.engine_kwargs()
    if kind == "coated":
        kw.update(core_radii=0.9 * float(w.strand.radii[0]), coating=COAT)
    st = w.strand
    rng = np.random.default_rng(1)
    u = np.zeros((st.n_nodes, 6))
    u[:, :3] = rng.normal(0.0, 2e-3, (st.n_nodes, 3))
    eng = AssemblyEngine(st.coords, st.conn, st.radii, w.section, precision=precision, **kw)
    u0 = torch.as_tensor(u.ravel(), device="cuda")
    u1 = u0 + torch.as_tensor(rng.normal(0.0, 4e-4, 6 * st.n_nodes), device="cuda")
    eng.detect(u0)
    return eng, u0, u1


def _state(eng):
    torch.cuda.synchronize()
    t = eng.pairs32 if eng.precision else eng.pairs
    out = {k: v.clone() for k, v in t.t.items() if torch.is_tensor(v) and k not in ("defer", "t2")}
    out["rec"] = eng.rec[: 16 * eng.pattern.n_members].clone()
    return out


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("kind", ["strand7", "strand37", "coated", "batch"])
@pytest.mark.parametrize("with_ref", [True, False])
def test_same_bits_as_the_parts(precision, kind, with_ref):
    one, u0, u1 = _engine(kind, precision)
    parts, _, _ = _engine(kind, precision)
    ref = u0 if with_ref else None
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    f = torch.linspace(-1.0, 1.0, u0.numel(), dtype=torch.float64, device="cuda")
    fixed = (torch.arange(u0.numel(), device="cuda") % 5 == 0).to(torch.uint8)
    with torch.cuda.stream(side):
        one.assemble(u1, ref, f, fixed)
    parts.pair_step(u1, ref)
    a, b = _state(one), _state(parts)
    assert a.keys() == b.keys()
    for k in a:
        assert torch.equal(a[k], b[k]), k
    assert torch.all(one.R[fixed.bool()] == 0.0)
    assert abs(one.norm2.item() / torch.dot(one.R, one.R).item() - 1.0) < 1e-12
    # without tangent (from the state after the same detection): the same residual
    third, _, _ = _engine(kind, precision)
    third.assemble(u1, ref, f, fixed, tangent=False)
    assert torch.equal(third.R, one.R)
