"""Candidate sets of the broadphase against the oracle's over clouds of every shape.

Equal and different radii (the prescreen margin with and without the sums), long boxes on any axis (the cells
run fastest along it), clouds flat on an axis, all in one cell, spread so far that the cells are coarsened,
given cell sizes, boxes turned round by a negative margin.
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
from xkgpu.device import DeviceMesh, ptr, stream_handle  # noqa: E402


def _cloud(n, shape, rng):
    c = rng.uniform(0.0, 1.0, (n, 3)) * n ** (1.0 / 3.0)
    d = rng.normal(0.0, 0.5, (n, 3))
    if shape in ("long_x", "long_y", "long_z"):
        k = "xyz".index(shape[-1])
        d[:, k] *= 6.0
        c[:, k] *= 4.0
    elif shape == "flat":
        c[:, 2] = d[:, 2] = 0.0
    elif shape == "one_spot":
        c *= 1e-3
    elif shape == "spread":
        c[: n // 2] += 1e5
    elif shape == "mixed_sizes":
        d[::17] *= 20.0
    X = np.stack([c, c + d], 1).reshape(-1, 3)
    conn = np.arange(2 * n).reshape(-1, 2)
    chain = np.arange(1, n) % 3 != 0  # two thirds of the segments begin where their predecessor ends
    conn[1:][chain, 0] = conn[:-1][chain, 1]
    return X, conn


@pytest.mark.parametrize("shape", ["cube", "long_x", "long_y", "long_z", "flat", "one_spot", "spread", "mixed_sizes"])
@pytest.mark.parametrize("n", [2, 33, 700])
@pytest.mark.parametrize("radii", ["equal", "different"])
def test_candidates_against_the_oracle(shape, n, radii):
    rng = np.random.default_rng(n + len(shape))
    X, conn = _cloud(n, shape, rng)
    r = np.full(n, 0.3) if radii == "equal" else rng.uniform(0.05, 0.4, n)
    layer = rng.integers(-1, 4, n)
    mesh = DeviceMesh(X, conn, r, layer)
    u = 0.1 * rng.normal(size=6 * len(X))
    x = oc.deformed_coords(X, u)
    ud = torch.as_tensor(u, device="cuda")
    out = torch.zeros(2 * n * n, dtype=torch.int32, device="cuda")
    for margin, shared, same, pre, pre_margin, cell in ((0.0, 1, 1, 1, 0.0, 0.0), (0.1, 0, 0, 0, 0.0, 0.0),
                                                        (0.0, 1, 0, 1, 0.07, 0.4), (0.0, 0, 1, 1, 0.0, 50.0),
                                                        (-0.35, 1, 1, 1, 0.0, 0.0)):
        bp = L.BPParams(margin, shared, same, pre, pre_margin)
        bp.cell_size = cell
        nk, nr, np_ = C.c_int64(), C.c_int64(), C.c_int64()
        L.call("xk_broadphase", C.byref(mesh.c), ptr(ud), C.byref(bp), ptr(out), n * n, C.byref(nk), C.byref(nr),
               C.byref(np_), stream_handle())
        lo, hi = oc.segment_aabbs(x, conn, r, margin)
        i, j = np.triu_indices(n, 1)
        hit = np.all((lo[i] <= hi[j]) & (lo[j] <= hi[i]), axis=1)
        raw = np.stack([i[hit], j[hit]], 1)
        kw = dict(elem_layer=layer, exclude_same_layer=bool(same), exclude_shared=bool(shared))
        before = oc.filter_candidates(raw, x, conn, r, midpoint_prescreening=False, **kw)
        want = oc.filter_candidates(raw, x, conn, r, midpoint_prescreening=bool(pre), prescreening_margin=pre_margin, **kw)
        assert (nr.value, np_.value) == (len(raw), len(before))
        got = out[: 2 * nk.value].view(-1, 2).cpu().numpy()
        assert np.array_equal(got, want)


@pytest.mark.parametrize("offset", [1e6, 1e8, 1e10, 1e12, 1e14])
@pytest.mark.parametrize("radii", ["equal", "different"])
def test_candidates_far_from_the_origin(offset, radii):
    """The prescreen decides as the exact routine wherever the cloud lies: the float midpoints resolve 2^-48 of the
    position, which passes the width of the undecided band from some 10^8 separations on."""
    n = 700
    rng = np.random.default_rng(int(np.log10(offset)))
    X, conn = _cloud(n, "cube", rng)
    X = X + offset * np.array([1.0, -0.7, 0.3])
    r = np.full(n, 0.3) if radii == "equal" else rng.uniform(0.05, 0.4, n)
    mesh = DeviceMesh(X, conn, r)
    u = 0.1 * rng.normal(size=6 * len(X))
    x = oc.deformed_coords(X, u)
    ud = torch.as_tensor(u, device="cuda")
    out = torch.zeros(2 * n * n, dtype=torch.int32, device="cuda")
    for margin, pre_margin in ((1.0, 0.0), (1.0, 0.07)):  # wide boxes, so that many candidates meet the prescreen's line
        bp = L.BPParams(margin, 1, 0, 1, pre_margin)
        nk, nr, np_ = C.c_int64(), C.c_int64(), C.c_int64()
        L.call("xk_broadphase", C.byref(mesh.c), ptr(ud), C.byref(bp), ptr(out), n * n, C.byref(nk), C.byref(nr),
               C.byref(np_), stream_handle())
        lo, hi = oc.segment_aabbs(x, conn, r, margin)
        i, j = np.triu_indices(n, 1)
        raw = np.stack([i, j], 1)[np.all((lo[i] <= hi[j]) & (lo[j] <= hi[i]), axis=1)]
        want = oc.filter_candidates(raw, x, conn, r, midpoint_prescreening=True, prescreening_margin=pre_margin)
        assert nr.value == len(raw)
        assert np.array_equal(out[: 2 * nk.value].view(-1, 2).cpu().numpy(), want)
