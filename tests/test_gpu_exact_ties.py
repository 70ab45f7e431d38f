"""The exact narrowphase where a quotient lies on or next to a rounding tie: its divides must give the operators' bits.

A unit normal's components over its own norm tie easily: the norm is 1 or a few last places beside it, and the
components of a contact at 30 or 60 degrees, or of a frame along the axes, are 1/2, 3/4 and the like.
"""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from oracle import contact as oc  # noqa: E402
from xkgpu import _lib as L  # noqa: E402
from xkgpu.device import DeviceMesh, DevicePairTable, ptr, stream_handle  # noqa: E402
from xkgpu.strand import make_strand  # noqa: E402


def _compare(X, conn, radii, table):
    mesh = DeviceMesh(X, conn, radii)
    dt = DevicePairTable(mesh.device)
    dt.from_host(table)
    cp = L.ContactParams(1.0, 0.5, 0.1, 0.0, 0.0, 1e-6, 1, 0.0, 0.0, 0.0, 0.5, 0.0)
    u = torch.zeros(6 * len(X), dtype=torch.float64, device="cuda")
    L.call("xk_narrowphase", C.byref(mesh.c), C.byref(dt.c), ptr(u), C.byref(cp), 1, stream_handle())
    want, got = oc.update_geometry(table, X), dt.to_host()
    for k in ("s", "t", "gap", "normal", "t1", "t2", "status"):
        assert np.array_equal(got[k], want[k]), (k, int(np.sum(got[k] != want[k])))
    for k in ("normal", "t1", "t2"):  # the signs of zeros too
        assert np.array_equal(np.signbit(got[k]), np.signbit(want[k])), k
    return want


@pytest.mark.parametrize("wires,pitches", [(7, 1), (19, 2)])
def test_strand_contacts_at_60_degrees(wires, pitches):
    st = make_strand(wires, 2.0, 40.0, pitches, 16 * pitches, gap=-0.01)
    table, _, _ = oc.detect(oc.empty_table(), st.coords, st.conn, st.radii, margin=1.0)
    table = _compare(st.coords, st.conn, st.radii, table)
    _compare(st.coords, st.conn, st.radii, table)  # frames transported


def _unit_vectors_with(component, n, rng):
    """Vectors whose first component is `component` and whose norm, as the frame forms it, is 1 or next to it."""
    out = np.zeros((0, 3))
    while len(out) < n:
        y = rng.uniform(-1.0, 1.0, 8 * n) * np.sqrt(1.0 - component**2)
        z = np.sqrt(1.0 - component**2 - y * y)
        v = np.stack([np.full_like(y, component), y, z + rng.integers(-12, 13, y.size) * 2.0**-53], 1)
        d = np.abs(np.sqrt(oc.dot_es(v, v)) - 1.0)
        out = np.concatenate([out, v[(d < 2.0**-48)]])
    return out[:n]


@pytest.mark.parametrize("component", [0.5, 0.75, 0.875, 0.25, 0.625, 1.0 - 2.0**-10, 0.5 + 2.0**-20])
def test_previous_frames_with_few_bits(component):
    n = 4000
    rng = np.random.default_rng(int(component * 1024))
    X = rng.uniform(-1.0, 1.0, (n, 4, 3))
    X[:, 2:] += 2.0 * rng.normal(size=(n, 1, 3))
    X, conn = X.reshape(-1, 3), np.arange(4 * n).reshape(-1, 2)
    radii = np.full(2 * n, 0.2)
    table = oc.new_pairs(np.stack([2 * np.arange(n), 2 * np.arange(n) + 1], 1), conn, radii)
    table = oc.update_geometry(table, X)
    v = _unit_vectors_with(component, n, rng)
    perm = rng.permuted(np.tile(np.arange(3), (n, 1)), axis=1)
    v = np.take_along_axis(v, perm, 1) * rng.choice([-1.0, 1.0], (n, 3))
    # the new normal near the previous one, so that the rotation between them shows a last place of either
    table["normal"] = v
    table["t1"] = np.cross(v, table["normal"][::-1])
    table["t1"] /= np.linalg.norm(table["t1"], axis=1)[:, None]
    _compare(X, conn, radii, table)


def test_distances_whose_mantissa_is_all_ones():
    """A divisor 2^k (1 - 2^-53) has its reciprocal next to a tie: quotients of powers of two show which way it fell.
    The offset of the two closest points is (sqrt(3)/2, 1/2, 0) 2^k itself, of that length: a point inside the first
    segment and the end of the second."""
    c = 0.8660254037844386
    rows = []
    for k in (-3, 0, 1, 5):
        for p in ((0, 1, 2), (1, 0, 2), (2, 0, 1)):
            for sign in (1.0, -1.0):
                x = np.array([[c, 0.5, -1.0], [c, 0.5, 1.0], [0.0, 0.0, 0.0], [-c, -0.5, 0.3]])
                rows.append(sign * 2.0**k * x[:, p])
    X = np.stack(rows)
    n = len(X)
    d = X[:, 0] + 0.5 * (X[:, 1] - X[:, 0])
    dist = np.sqrt(oc.dot_es(d, d))
    assert np.all(np.frexp(dist)[0] == 1.0 - 2.0**-53)
    X, conn = X.reshape(-1, 3), np.arange(4 * n).reshape(-1, 2)
    radii = np.full(2 * n, 0.01)
    table = oc.new_pairs(np.stack([2 * np.arange(n), 2 * np.arange(n) + 1], 1), conn, radii)
    want = oc.update_geometry(table, X)
    assert np.allclose(want["gap"] + 0.02, dist, rtol=1e-15)
    _compare(X, conn, radii, table)
