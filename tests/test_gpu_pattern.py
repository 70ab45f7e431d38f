"""The contact pattern's lists against a direct construction on the host, whole numbers throughout.

Chains and branched meshes, pair tables in any order, nodes with few and with very many members (the warp's
register sort, its shared-memory sort and the serial path), tables without members or without other pairs, the
element-side arrays and the lower index present or absent, and a row over the 256 columns that are accepted.
"""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from xkgpu import _lib as L  # noqa: E402
from xkgpu.device import DeviceContactPattern, DeviceMesh, DevicePairTable, stream_handle  # noqa: E402


def _mesh(kind, ne, rng):
    if kind == "chain":  # wires of five elements
        conn = np.array([(e + e // 5, e + e // 5 + 1) for e in range(ne)])
    else:  # every third element starts at node 0
        conn = np.array([(0 if e % 3 == 0 else e, e + 1) for e in range(ne)])
    X = rng.normal(size=(conn.max() + 1, 3))
    return DeviceMesh(X, conn, np.full(ne, 0.1)), conn


def _pairs(ne, n, hub, rng):
    ea, eb = rng.integers(0, ne, n), rng.integers(0, ne - 1, n)
    eb = np.where(eb >= ea, eb + 1, eb)
    if hub:  # element 2 meets the first ones in turn
        k = min(hub, n)
        other = np.arange(k) % (ne - 1)
        ea[:k], eb[:k] = 2, np.where(other >= 2, other + 1, other)
    p = rng.permutation(n)
    return ea[p], eb[p]


def _expected(conn, ea, eb, member, nn):
    ne = len(conn)
    members, others = np.nonzero(member)[0], np.nonzero(~member)[0]
    nodes = np.concatenate([conn[ea[members]], conn[eb[members]]], 1)
    inc, einc = [[] for _ in range(nn)], [[] for _ in range(ne)]
    blocks: dict[tuple, list] = {}
    for mi, nd in enumerate(nodes.tolist()):
        einc[ea[members[mi]]].append(2 * mi)
        einc[eb[members[mi]]].append(2 * mi + 1)
        for k in range(4):
            inc[nd[k]].append(4 * mi + k)
            for q in range(4):
                if nd[k] <= nd[q]:
                    blocks.setdefault((nd[k], nd[q]), []).append(16 * mi + 4 * k + q)
    keys = sorted(blocks)
    at = {b: i for i, b in enumerate(keys)}
    low = [[] for _ in range(nn)]
    for v, w in keys:
        if v != w:
            low[w].append(at[v, w])
    terms, fits = [], True
    for v, w in keys:
        t = []
        for e in range(ne):
            for p in range(2):
                if conn[e, p] == v:
                    if w == v:
                        t.append(48 * e + 32 * p - 2**31)
                    if conn[e, 1 - p] == w:
                        t.append(48 * e + 16 - 2**31)
        t += [c for c in blocks[v, w] if (c >> 3) & 1 != (c >> 1) & 1]
        fits &= len(t) <= 4
        terms.append(sorted(t + [-1] * (4 - len(t))))
    return dict(members=members, others=others, nodes=nodes, inc=inc, einc=einc, keys=keys, low=low,
                contrib=[sorted(blocks[b]) for b in keys], terms=terms, fits=fits)


def _split(ptr, flat):
    p, f = ptr.cpu().numpy(), flat.cpu().numpy()
    return [f[a:b].tolist() for a, b in zip(p[:-1], p[1:])]


@pytest.mark.parametrize("kind,ne,n,hub,share", [
    ("chain", 3, 1, 0, 1.0), ("chain", 40, 60, 0, 0.5), ("chain", 40, 60, 0, 0.0), ("chain", 300, 2500, 0, 0.7),
    ("chain", 90, 400, 89, 1.0), ("chain", 70, 900, 600, 1.0), ("star", 20, 90, 0, 0.6), ("star", 60, 700, 0, 0.9)])
@pytest.mark.parametrize("optional", [True, False])
def test_lists_against_direct_construction(kind, ne, n, hub, share, optional):
    rng = np.random.default_rng(ne + n)
    mesh, conn = _mesh(kind, ne, rng)
    ea, eb = _pairs(ne, n, hub, rng)
    status = np.where(rng.random(n) < share, rng.integers(1, 3, n), 0)
    p_n = np.where(rng.random(n) < 0.5 * share, 1.0, 0.0)
    pairs = DevicePairTable(mesh.device, n)
    for k, a in (("ea", ea), ("eb", eb), ("status", status), ("p_n", p_n)):
        pairs.t[k][:n] = torch.as_tensor(a).to(pairs.t[k])
    pairs.set_n(n)
    pat = DeviceContactPattern(mesh)
    if not optional:
        sync = pat._sync_struct

        def without():
            sync()
            pat.c.node_elem_ptr = pat.c.node_elem = pat.c.elem_ptr = pat.c.elem_inc = pat.c.bcodes = None
            pat.c.low_ptr = pat.c.low_blk = None

        pat._sync_struct = without
    for _ in range(2):  # the second build has the mesh's lists and grown arrays
        pat.build(pairs)
    x = _expected(conn, ea, eb, (status != 0) | (p_n > 0), mesh.n_nodes)
    nm, nb = len(x["members"]), len(x["keys"])
    assert (pat.n_members, pat.c.n_others, pat.nnzb) == (nm, n - nm, nb)
    assert pat.n_contrib == sum(map(len, x["contrib"]))
    assert np.array_equal(pat.members[:nm].cpu(), x["members"]) and np.array_equal(pat.others[: n - nm].cpu(), x["others"])
    assert np.array_equal(pat.member_nodes[: 4 * nm].cpu(), x["nodes"].ravel())
    assert _split(pat.inc_ptr, pat.inc) == x["inc"]
    rows = np.array(x["keys"]).reshape(-1, 2)
    assert np.array_equal(pat.blk_row[:nb].cpu(), rows[:, 0]) and np.array_equal(pat.col[:nb].cpu(), rows[:, 1])
    assert np.array_equal(pat.row_ptr.cpu(), np.searchsorted(rows[:, 0], np.arange(mesh.n_nodes + 1)))
    assert _split(pat.blk_ptr[: nb + 1], pat.contrib) == x["contrib"]
    if not optional:
        assert pat.nnzb_full == nb and not pat.c.sides_ok
        return
    assert pat.nnzb_full == nb + sum(map(len, x["low"]))
    assert _split(pat.low_ptr, pat.low_blk) == x["low"]
    assert _split(pat.elem_ptr, pat.elem_inc) == x["einc"]
    assert bool(pat.c.sides_ok) == x["fits"]
    if x["fits"]:
        assert pat.bcodes[: 4 * nb].cpu().numpy().reshape(-1, 4).tolist() == x["terms"]


def test_more_cross_terms_than_a_byte_counts():
    """A block with 256 cross contributions (elements of no length, both ends one node): its list is whole, the
    inline terms are refused, and those of the rows before it stay."""
    conn = np.array([(2 * e, 2 * e + 1) for e in range(24)] + [(48, 49 + e) for e in range(8)] + [(57, 57)] * 16)
    ne, nn = len(conn), 58
    mesh = DeviceMesh(np.random.default_rng(1).normal(size=(nn, 3)), conn, np.full(ne, 0.1))
    ea = np.array([2 * k for k in range(12)] + [24 + e for e in range(8) for _ in range(16)])
    eb = np.array([2 * k + 1 for k in range(12)] + [32 + f for _ in range(8) for f in range(16)])
    n = len(ea)
    pairs = DevicePairTable(mesh.device, n)
    for k, a in (("ea", ea), ("eb", eb), ("status", np.ones(n))):
        pairs.t[k][:n] = torch.as_tensor(a).to(pairs.t[k])
    pairs.set_n(n)
    pat = DeviceContactPattern(mesh)
    for _ in range(2):
        pat.build(pairs)
        x = _expected(conn, ea, eb, np.ones(n, bool), nn)
        nb = len(x["keys"])
        assert pat.nnzb == nb and not x["fits"] and not pat.c.sides_ok
        assert len(x["contrib"][x["keys"].index((48, 57))]) == 256
        assert _split(pat.blk_ptr[: nb + 1], pat.contrib) == x["contrib"]
        codes = pat.bcodes[: 4 * nb].cpu().numpy().reshape(-1, 4).tolist()
        for (v, _), got, want in zip(x["keys"], codes, x["terms"]):
            if v < 48:
                assert got == want


def test_a_row_over_256_columns_is_refused():
    ne = 400
    conn = np.arange(2 * ne).reshape(-1, 2)
    mesh = DeviceMesh(np.random.default_rng(0).normal(size=(2 * ne, 3)), conn, np.full(ne, 0.1))
    for n, ok in ((127, True), (130, False)):  # 2 n + 2 columns in the rows of element 0's nodes
        pairs = DevicePairTable(mesh.device, n)
        pairs.t["eb"][:n] = torch.arange(1, n + 1)
        pairs.t["status"][:n] = 1
        pairs.set_n(n)
        pat = DeviceContactPattern(mesh)
        pat._sync_struct()
        code = L.call("xk_contact_pattern_build", C.byref(mesh.c), C.byref(pairs.c), C.byref(pat.c),
                      stream_handle(None), allow=(L.XK_ERR_OVERFLOW,))
        assert (code == L.XK_OK) == ok
