"""The FP64 beam by two lanes an element, against the oracle at the edges of its warps (15 elements each), at wire
ends and at the largest mesh that takes it; and its bits against the colour launches' at u = 0."""

import numpy as np
import pytest

from conftest import rel_err, sparse_rel_err

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from oracle import beam as ob  # noqa: E402
from xkgpu import _lib as L  # noqa: E402
from xkgpu import workloads as W  # noqa: E402
from xkgpu.device import DeviceBeam, DeviceMesh  # noqa: E402


def _mesh(sizes):
    conn, at = [], 0
    for n in sizes:
        conn.append(at + np.stack([np.arange(n), np.arange(1, n + 1)], 1))
        at += n + 1
    conn = np.concatenate(conn)
    rng = np.random.default_rng(len(conn))
    X = np.cumsum(rng.uniform(0.3, 1.0, (at, 3)), axis=0)
    u = 0.02 * rng.normal(size=(at, 6))
    u[:, 3:] = 0.4 * rng.normal(size=(at, 3))
    sec = W.circle_section(0.2)
    beam = DeviceBeam(DeviceMesh(X, conn, 0.1), sec)
    assert beam.chain_ordered
    return X, conn, u.ravel(), sec, beam


def _run(beam, u, tangent=True):
    f = torch.full((u.size,), 7.0, dtype=torch.float64, device="cuda")
    K = torch.full((36 * beam.nnzb,), 7.0, dtype=torch.float64, device="cuda")
    beam.assemble(torch.as_tensor(u, device="cuda"), L.XK_FP64, f, K if tangent else None)
    return f, K


@pytest.mark.parametrize("sizes", [[1], [14], [15], [16], [1, 1, 28], [30, 31, 3], [7, 640, 1], [9392], [9424]])
def test_beam_by_two_lanes(sizes):
    X, conn, u, sec, beam = _mesh(sizes)
    f, K = _run(beam, u)
    K_ref, f_ref = ob.assemble_beam(X, conn, u, ob.Section(**{**sec, "scf": None}))
    # both round each of some thousand operations once: 1e3 x 2^-53, with room for cancellation
    assert rel_err(f.cpu().numpy(), f_ref) < 1e-12
    assert sparse_rel_err(beam.to_csr(K), K_ref) < 1e-12
    assert torch.equal(_run(beam, u, tangent=False)[0], f)
    f, K = _run(beam, np.zeros_like(u))
    beam.plan.chain_ordered = 0  # by colours
    f0, K0 = _run(beam, np.zeros_like(u))
    assert torch.equal(f, f0) and torch.equal(K, K0)
