"""The FP64 engine's per-iteration kernels at the sizes and states where they can go wrong.

The pair kernels form the narrowphase with fused operations and hand every pair outside the ordinary
case (near-parallel, degenerate, without a frame) to the exact routine; both against the oracle.  The
one-launch beam at the edges of its warps (31 elements each) and at wire ends, against the oracle.
"""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import rel_err, sparse_rel_err

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from oracle import beam as ob  # noqa: E402
from oracle import contact as oc  # noqa: E402
from xkgpu import _lib as L  # noqa: E402
from xkgpu import workloads as W  # noqa: E402
from xkgpu.device import DeviceBeam, DeviceContactPattern, DeviceMesh, DevicePairTable, ptr, stream_handle  # noqa: E402


def _pairs(n, seed):
    """n separate segment pairs: skew, near-parallel, parallel, point-like and crossing ones in turn."""
    rng = np.random.default_rng(seed)
    X = rng.uniform(-1.0, 1.0, (n, 4, 3))
    X[:, 2:] += 0.5 * rng.normal(size=(n, 1, 3))
    for k in range(n):
        d = X[k, 1] - X[k, 0]
        if k % 7 == 1:  # a small angle on either side of the routine's line
            X[k, 3] = X[k, 2] + d + 0.04 * rng.normal(size=3)
        elif k % 7 == 2:
            X[k, 3] = X[k, 2] + 0.7 * d
        elif k % 7 == 3:
            X[k, 3] = X[k, 2] + 1e-7 * rng.normal(size=3)
        elif k % 7 == 4:  # nearly touching
            X[k, 2:] += 0.5 * (X[k, 0] + X[k, 1]) - 0.5 * (X[k, 2] + X[k, 3]) + 1e-3 * rng.normal(size=3)
    return X.reshape(-1, 3), np.arange(4 * n).reshape(-1, 2)


@pytest.mark.parametrize("n", [1, 31, 33, 257])
@pytest.mark.parametrize("delta,aligned", [(0.0, True), (1e3, True), (0.0, False)])
def test_pair_kernels_against_the_oracle(n, delta, aligned):
    X, conn = _pairs(n, n)
    rng = np.random.default_rng(n + 1)
    ne, nd = 2 * n, 6 * len(X)
    radii = np.full(ne, 0.2)
    keys = np.stack([2 * np.arange(n), 2 * np.arange(n) + 1], 1)
    mesh = DeviceMesh(X, conn, radii)
    table = oc.new_pairs(keys, conn, radii)
    table = oc.update_geometry(table, X, g_on=10.0 if n % 2 else 0.0)  # odd n: every pair active
    for k in range(n):  # frames missing, and not of unit length
        if k % 11 == 5:
            table["t1"][k] = 0.0
        elif k % 11 == 6:
            table["normal"][k] *= 1.5
    dt = DevicePairTable(mesh.device)
    dt.from_host(table)
    pat = DeviceContactPattern(mesh)
    pat.build(dt)
    u_ref = 1e-3 * rng.normal(size=nd)
    u = u_ref + 1e-3 * rng.normal(size=nd)
    k_pen, mu = 50.0, 0.2
    cp = L.ContactParams(k_pen, 0.5, mu, delta, 0.0, 1e-6, 1, 0.0, 0.0, 0.0, 0.5, 0.0)
    dev = lambda x: torch.as_tensor(x, device="cuda")  # noqa: E731
    ud, urd = dev(u), dev(u_ref)
    buf = torch.zeros(16 * max(pat.n_members, 1) + 1, dtype=torch.float64, device="cuda")
    rec = buf if aligned else buf[1:]
    L.call("xk_pair_step", C.byref(mesh.c), C.byref(dt.c), C.byref(pat.c), ptr(ud), ptr(urd), C.byref(cp),
           L.XK_STAGE_ALL, L.XK_FP64, L.XK_OUT_COMBINED, ptr(rec), stream_handle())
    torch.cuda.synchronize()
    h = dt.to_host()
    # the closest point's parameters lose 1 / det (det > 1e-3 ac, else the exact routine): 1e3 x 2e-15, and the
    # normal that error over the distance (above 1e-3 here); the gap takes it squared
    t = oc.update_geometry(table, oc.deformed_coords(X, u), freeze_active_set=True)
    ok = t["gap"] + 0.4 > 1e-3
    for k, tol in (("s", 2e-11), ("t", 2e-11), ("gap", 1e-13)):
        assert np.max(np.abs(h[k] - t[k])) < tol, k
    for k in ("normal", "t1", "t2"):
        assert np.max(np.abs(h[k] - t[k])[ok]) < 1e-8, k
    t, fn, _ = oc.huber_evaluate(t, nd, k_pen, delta)
    t, ff, _, fr = oc.friction_evaluate(t, u, u_ref, nd, k_pen, 0.5, mu)
    for k in ("p_n", "z_t", "q_trial_norm"):
        assert rel_err(h[k], t[k]) < 1e-8, k
    assert np.array_equal(h["status"], t["status"]) and np.array_equal(h["stick"], t["stick"])
    m = pat.members[: pat.n_members].cpu().numpy()
    f = np.zeros(nd)
    r = rec[: 16 * len(m)].view(-1, 16).cpu().numpy()
    c = oc.shape_coeffs(r[:, 9], r[:, 10])
    np.add.at(f, oc.trans_dofs(t["nodes"][m]).ravel(), (c[:, :, None] * r[:, None, 11:14]).ravel())
    assert rel_err(f, fn + ff) < 1e-8
    K = oc._blocks_to_csr(t["nodes"][m], (c[:, :, None] * c[:, None, :])[:, :, :, None, None]
                          * r[:, :9].reshape(-1, 1, 1, 3, 3), nd)
    K_ref = (oc.huber_tangent(t, nd, k_pen, delta) - oc.friction_tangent(t, fr, nd)).tocsr()
    if K_ref.nnz:
        assert sparse_rel_err(K, K_ref) < 1e-8


@pytest.mark.parametrize("n", [1, 33, 700])
def test_exact_narrowphase_gives_the_oracle_bits(n):
    """Every branch of the exact routine (ordinary, near-parallel, degenerate; frames fresh, transported, from
    normals of any length, turned far) and the unit-vector forms of its divides, value for value."""
    X, conn = _pairs(n, n + 5)
    rng = np.random.default_rng(n)
    nd = 6 * len(X)
    radii = np.full(2 * n, 0.2)
    mesh = DeviceMesh(X, conn, radii)
    table = oc.new_pairs(np.stack([2 * np.arange(n), 2 * np.arange(n) + 1], 1), conn, radii)
    dt = DevicePairTable(mesh.device)
    cp = L.ContactParams(1.0, 0.5, 0.1, 0.0, 0.05, 0.1, 1, 0.0, 0.0, 0.0, 0.5, 0.0)
    u = np.zeros(nd)
    for step in range(4):
        if step == 2:
            for k in range(n):  # other lengths, no tangent, a normal turned round
                table["normal"][k] *= (1.0, 1.0 + 2.0**-50, 1.5, -1.0)[k % 4]
                table["t1"][k] *= (1.0, 0.0, 1.0 - 2.0**-40)[k % 3]
        dt.from_host(table)
        ud = torch.as_tensor(u, device="cuda")
        L.call("xk_narrowphase", C.byref(mesh.c), C.byref(dt.c), ptr(ud), C.byref(cp), 1, stream_handle())
        table = oc.update_geometry(table, oc.deformed_coords(X, u), g_on=0.05, g_off=0.1)
        h = dt.to_host()
        for k in ("s", "t", "gap", "normal", "t1", "t2", "status"):
            assert np.array_equal(h[k], table[k]), (step, k)
        u = u + 10.0 ** (-6 + 2 * step) * rng.normal(size=nd)


@pytest.mark.parametrize("wires", [(1,), (30,), (31,), (32, 1), (62, 31), (5, 58, 3), "chain", "branched"])
@pytest.mark.parametrize("scf", [None, 8.0])
def test_beam_against_the_oracle(wires, scf):
    rng = np.random.default_rng(3)
    if wires == "chain":  # elements of a chain against their order along the wire
        conn = np.array([[k + 1, k] if k % 2 else [k, k + 1] for k in range(40)])[::-1]
    elif wires == "branched":
        conn = np.array([[0, k] for k in range(1, 6)] + [[k, k + 5] for k in range(1, 6)])
    else:
        conn, n0 = [], 0
        for ne in wires:
            conn += [[n0 + k, n0 + k + 1] for k in range(ne)]
            n0 += ne + 1
        conn = np.array(conn)
    nn = conn.max() + 1
    X = np.cumsum(rng.uniform(0.3, 1.0, (nn, 3)), axis=0)
    u = 0.02 * rng.normal(size=(nn, 6))
    u[:, 3:] = 0.4 * rng.normal(size=(nn, 3))
    u = u.ravel()
    sec = {**W.circle_section(0.2), "scf": scf}
    mesh = DeviceMesh(X, conn, 0.1)
    beam = DeviceBeam(mesh, sec)
    assert beam.chain_ordered == (wires not in ("chain", "branched"))
    f = torch.full((6 * nn,), 7.0, dtype=torch.float64, device="cuda")
    K = torch.full((36 * beam.nnzb,), 7.0, dtype=torch.float64, device="cuda")
    beam.assemble(torch.as_tensor(u, device="cuda"), L.XK_FP64, f, K)
    K_ref, f_ref = ob.assemble_beam(X, conn, u, ob.Section(**sec))
    # both round each of some thousand operations once: 1e3 x 2^-53, with room for cancellation
    assert rel_err(f.cpu().numpy(), f_ref) < 1e-12
    assert sparse_rel_err(beam.to_csr(K), K_ref) < 1e-12
