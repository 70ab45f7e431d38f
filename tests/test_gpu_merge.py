"""The pair-table merge at ragged rows per segment, and the screened detection's pass over the merged rows."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from xkgpu import _lib as L  # noqa: E402
from xkgpu import workloads as W  # noqa: E402
from xkgpu.device import DeviceMesh, DevicePairTable, DevicePairTable32, ptr, stream_handle  # noqa: E402
from xkgpu.engine import AssemblyEngine  # noqa: E402

COUNTS = [0, 0, 1, 31, 32, 33, 64, 65, 97, 2, 0, 130]
FIELDS = ("s", "t", "gap", "lambda_n", "k_pen", "k_t", "p_n", "q_trial_norm", "dissipation", "normal", "t1", "t2", "z_t")


def _rows(rng, ne, counts):
    """Sorted distinct (a, b) with counts[a % len] rows in segment a (as many as there are b > a)."""
    out = []
    for a in range(ne):
        k = min(counts[a % len(counts)], ne - 1 - a)
        out += [(a, b) for b in sorted(rng.choice(np.arange(a + 1, ne), k, replace=False))]
    return np.array(out, dtype=np.int64).reshape(-1, 2)


@pytest.mark.parametrize("drop", [False, True])
@pytest.mark.parametrize("ne,old_counts,new_counts", [(2, [1], [1]), (200, COUNTS, COUNTS[::-1]), (333, COUNTS, [0]),
                                                      (333, [0], COUNTS), (150, [149], [3, 149])])
def test_merge_against_sets(ne, old_counts, new_counts, drop):
    rng = np.random.default_rng(ne)
    old_rows, cands = _rows(rng, ne, old_counts), _rows(rng, ne, new_counts)
    half = rng.random(len(old_rows)) < 0.5  # half of the old rows are candidates again
    cands = np.unique(np.concatenate([cands, old_rows[half]]), axis=0)
    n = len(old_rows)
    old = {"ea": old_rows[:, 0], "eb": old_rows[:, 1], "status": rng.integers(0, 3, n), "stick": rng.random(n) < 0.5}
    for k in FIELDS:
        w = {"normal": 3, "t1": 3, "t2": 3, "z_t": 2}.get(k, 1)
        old[k] = rng.normal(size=(n, w) if w > 1 else n)
    idle = rng.random(n) < 0.4  # pristine rows
    old["status"] = np.where(idle, 0, old["status"])
    for k in ("p_n", "k_pen", "z_t"):
        old[k][idle] = 0.0
    X = np.stack([np.arange(ne + 1.0), np.zeros(ne + 1), np.zeros(ne + 1)], 1)
    mesh = DeviceMesh(X, np.stack([np.arange(ne), np.arange(1, ne + 1)], 1), np.full(ne, 0.1))
    table, out = DevicePairTable(mesh.device, cap=max(n, 16)), DevicePairTable(mesh.device, cap=n + len(cands) + 16)
    table.from_host(old)
    rows = torch.as_tensor(cands.astype(np.int32).ravel().copy(), device="cuda")
    L.call("xk_pairs_merge_pruned" if drop else "xk_pairs_merge", C.byref(mesh.c), C.byref(table.c), ptr(rows),
           len(cands), C.byref(out.c), stream_handle(None))
    out.set_n(out.c.n)
    got = out.to_host()
    is_cand = {tuple(r) for r in cands}
    where = {tuple(r): i for i, r in enumerate(old_rows)}
    stays = [r for i, r in enumerate(map(tuple, old_rows)) if r not in is_cand and not (drop and idle[i])]
    exp = sorted(is_cand | set(stays))
    assert list(zip(got["ea"], got["eb"])) == exp
    src = np.array([where.get(r, -1) for r in exp], dtype=np.int64)
    new = src < 0
    status = np.where(new | np.array([r not in is_cand for r in exp], dtype=bool), 0, old["status"][src] if n else 0)
    assert np.array_equal(got["status"], status)
    assert np.array_equal(got["stick"], new | (old["stick"][src] if n else True))
    for k in FIELDS:
        v = np.zeros_like(got[k])
        if n:
            v[~new] = old[k][src[~new]]
        assert np.array_equal(got[k], v), k


@pytest.mark.parametrize("workload", ["strand7", "strand37"])
@pytest.mark.parametrize("from32", [True, False])
def test_screened_merge_is_merge_then_narrowphase(workload, from32):
    w = W.config_workload(workload, seed=7)
    st = w.strand
    rng = np.random.default_rng(2)
    du = torch.as_tensor(rng.normal(0.0, 1e-2, 6 * st.n_nodes), device="cuda")
    tables = []
    for fused in (True, False):
        eng = AssemblyEngine(st.coords, st.conn, st.radii, w.section, precision="mixed", **w.engine_kwargs())
        u0 = torch.as_tensor(w.u, device="cuda")
        eng.detect(u0)
        eng.assemble(u0 + 0.1 * du, u0)
        u = u0 + du
        if fused:
            if not from32:
                eng.sync_state()
            eng.detect(u)
            tables.append((eng.pairs.to_host(), eng.stats["narrowphase_exact"]))
            continue
        eng.sync_state()
        s = stream_handle(None)
        cands, nc = eng.candidates(u)
        L.call("xk_nodes_prepare", C.byref(eng.mesh.c), ptr(u), ptr(u), ptr(eng.node32), s)
        out = DevicePairTable(eng.device, cap=eng.pairs.n + nc + 16)
        L.call("xk_pairs_merge", C.byref(eng.mesh.c), C.byref(eng.pairs.c), ptr(cands), nc, C.byref(out.c), s)
        out.set_n(out.c.n)
        n_exact = torch.zeros(1, dtype=torch.int32, device="cuda")
        L.call("xk_narrowphase_screened", C.byref(eng.mesh.c), C.byref(out.c), ptr(u), ptr(eng.node32),
               C.byref(eng.cp), ptr(n_exact), s)
        tables.append((out.to_host(), int(n_exact.item())))
    (a, na), (b, nb) = tables
    assert na == nb and a["ea"].size > 0
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("n,kind", [(1, "all"), (255, "some"), (256, "none"), (257, "all"), (3000, "some"),
                                    (70_000, "runs"), (140_001, "all")])
def test_float_table_slots(n, kind):
    """Slots of the float table: members first, both in ascending order; the state comes back to the same pairs."""
    rng = np.random.default_rng(n)
    ne = 600
    k = rng.choice(ne * ne, n, replace=False)
    k.sort()
    d = {"ea": k // ne, "eb": k % ne, "stick": rng.random(n) < 0.5}
    for f in FIELDS:
        w = {"normal": 3, "t1": 3, "t2": 3, "z_t": 2}.get(f, 1)
        d[f] = rng.normal(size=(n, w) if w > 1 else n).astype(np.float32).astype(np.float64)
    mem = {"all": np.ones(n, bool), "none": np.zeros(n, bool), "some": rng.random(n) < 0.2,
           "runs": (np.arange(n) // 700) % 3 == 1}[kind]
    d["status"] = np.where(mem, 1, 0)
    d["p_n"] = np.where(mem, np.abs(d["p_n"]), 0.0)
    X = rng.normal(size=(ne + 1, 3))
    mesh = DeviceMesh(X, np.stack([np.arange(ne), np.arange(1, ne + 1)], 1), np.full(ne, 0.1))
    table = DevicePairTable(mesh.device, cap=n + 16)
    table.from_host(d)
    # the pattern's two lists, which are all that the float table takes from it
    members = torch.as_tensor(np.flatnonzero(mem).astype(np.int32), device="cuda")
    others = torch.as_tensor(np.flatnonzero(~mem).astype(np.int32), device="cuda")
    pat = L.ContactPattern()
    pat.n_nodes, pat.n_members, pat.n_others = ne + 1, members.numel(), others.numel()
    pat.members, pat.others = ptr(members), ptr(others)
    q = DevicePairTable32(mesh.device)
    q.ensure(n)
    s = stream_handle(None)
    L.call("xk_pairs_to32", C.byref(mesh.c), C.byref(table.c), C.byref(pat), C.byref(q.c), s)
    order = np.concatenate([np.flatnonzero(mem), np.flatnonzero(~mem)])
    assert q.c.n == n and q.c.n_members == mem.sum()
    assert np.array_equal(q.t["pair"][:n].cpu().numpy(), order)
    assert np.array_equal(order[q.t["slot"][:n].cpu().numpy()], np.arange(n))
    assert np.array_equal(q.t["gap"][:n].cpu().numpy(), d["gap"][order].astype(np.float32))
    conn = mesh.conn.cpu().numpy().reshape(-1, 2)
    nodes = np.concatenate([conn[d["ea"][order]], conn[d["eb"][order]]], 1)
    assert np.array_equal(q.t["nodes"][: 4 * n].cpu().numpy().reshape(-1, 4), nodes)
    back = DevicePairTable(mesh.device, cap=n + 16)
    back.from_host({**d, **{f: np.zeros_like(d[f]) for f in FIELDS if f != "lambda_n"}})
    L.call("xk_pairs_from32", C.byref(q.c), C.byref(back.c), s)
    got = back.to_host()
    for f in FIELDS:
        if f == "t2":  # the others' is formed again from the normal and t1
            assert np.array_equal(got[f][mem], d[f][mem])
        else:
            assert np.array_equal(got[f], d[f]), f
    assert np.array_equal(got["status"], d["status"]) and np.array_equal(got["stick"], d["stick"])
