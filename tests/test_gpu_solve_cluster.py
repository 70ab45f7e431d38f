"""The one-cluster BiCGStab of small systems against the launch-per-step form: the same bits.

A mesh with further nodes that no element touches has the same system plus empty rows, and is large enough
for the launches; the sums meet the same terms in the same order, so x, the iterations and the residual
are equal.  Sizes: one element, a chunk of 256 products, the rows of one CTA, the line between the forms.
"""

from __future__ import annotations

import warnings

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from xkgpu import strand as S  # noqa: E402
from xkgpu import workloads as W  # noqa: E402
from xkgpu.engine import AssemblyEngine  # noqa: E402
from xkgpu.solve import DeviceLinearSolver  # noqa: E402


def _solve(wires, el, precision, pad, check_every, max_iter):
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        st = S.make_strand(wires, 2.0, 40.0, 1, el, gap=-0.01, allow_coarse=True)
    X = np.concatenate([st.coords, 1e3 + np.arange(3 * pad).reshape(-1, 3)])
    eng = AssemblyEngine(X, st.conn, st.radii, W.circle_section(2.0), layer=st.elem_layer, precision=precision,
                         k_pen=1e4, mu=0.0)
    nd = eng.mesh.ndof
    u = torch.zeros(nd, dtype=torch.float64, device="cuda")
    eng.detect(u)
    eng.assemble(u, u)
    fixed = np.zeros((len(X), 6), np.uint8)
    fixed[:1] = 1
    ds = DeviceLinearSolver(eng, rtol=1e-10, max_iter=max_iter, check_every=check_every, strict=False)
    ds.set_fixed(fixed.ravel())
    b = torch.zeros(nd, dtype=torch.float64, device="cuda")
    b[: st.ndof] = torch.as_tensor(np.random.default_rng(1).normal(size=st.ndof), device="cuda")
    x0 = torch.zeros_like(b)
    x0[: st.ndof] = 1e-6
    x = ds.solve(b, x0)
    return x[: st.ndof], ds.iterations, ds.rel_res


@pytest.mark.parametrize("wires,el", [(1, 1), (1, 41), (1, 42), (1, 171), (7, 16), (7, 47), (19, 17), (7, 95)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_cluster_and_launches_give_the_same_bits(wires, el, precision):
    for check_every, max_iter in ((10, 600), (7, 45)):
        small = _solve(wires, el, precision, 0, check_every, max_iter)
        large = _solve(wires, el, precision, 700, check_every, max_iter)
        assert small[1] == large[1] and small[2] == large[2]
        assert torch.equal(small[0], large[0])
