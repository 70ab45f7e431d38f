"""The measured cases: what a user of the framework has it do, through its public entry points.

Kinds of case
  assemble  one Newton iteration's assembly (``AssemblyEngine``): the pairs' narrowphase, normal force and
            friction, the beam's internal force, the residual, K_beam and K_c; replayed as a CUDA graph, as
            the Newton drivers run it, or launched eagerly, as a first use or a host solver loop does
  detect    one detection (``AssemblyEngine.detect``): once per increment, on a table with history
  score     the pruning network's scores of a detection's candidates (``PairPruner.logits``)
  train     one full-batch training step of that network (``PairPruner.gradient`` and ``adam``)
  solve     one linear solve of a well-posed increment (``DeviceLinearSolver.solve``)

The strands are the repository's own configurations (``workloads.CONFIGS``) and others of the same family;
``draw`` spreads wire counts (also partly filled outer layers), pitches and discretisations over their range.
Every state is a bent strand (curvature 1/(50 D), the bending runs' arc) with the configurations' seeded noise.
"""

from __future__ import annotations

import functools
import math
import sys
import warnings
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "xkep-cae_gb300"))

from xkgpu import _lib as L  # noqa: E402
from xkgpu import runs, workloads  # noqa: E402
from xkgpu import strand as strands  # noqa: E402
from xkgpu.engine import AssemblyEngine  # noqa: E402
from xkgpu.prune import PairPruner, init_params  # noqa: E402
from xkgpu.solve import DeviceLinearSolver  # noqa: E402

MU, K_T_RATIO, G_ON, G_OFF = 0.1, 0.5, 0.0, 1e-6
COAT = dict(stiffness=1e4, damping=50.0, mu=0.2, k_t_ratio=0.5, dt=0.1)


def _strand(name, kind, precision, n_wires, d, pitch, n_pitches, el, **options):
    return dict(name=name, kind=kind, precision=precision, n_wires=n_wires, d=d, pitch=pitch, n_pitches=n_pitches,
                el=el, **options)


def listed():
    return [
        # the smallest call of a Newton loop: a 7-wire strand, where launches and latency count
        _strand("assemble_7_mixed", "assemble", "mixed", 7, 2.0, 40.0, 1, 16, mode="replay"),
        # an ordinary strand with coated wires: every candidate pair carries a force
        _strand("assemble_91_coated_mixed", "assemble", "mixed", 91, 2.0, 40.0, 4, 32, mode="replay", coated=True),
        # the largest strand configuration
        _strand("assemble_1027_mixed", "assemble", "mixed", 1027, 0.5, 20.0, 4, 24, mode="replay"),
        # many ragged strands in one mesh with a friction coefficient per element, launched eagerly
        dict(name="assemble_batch64_mixed", kind="assemble", precision="mixed", n_strands=64, d=2.0, pitch=40.0,
             mode="eager"),
        # an ordinary strand in double, launched eagerly with loads and clamped ends, default schedules
        _strand("assemble_37_fp64", "assemble", "fp64", 37, 2.0, 40.0, 4, 32, mode="eager"),
        # the largest strand in double
        _strand("assemble_1027_fp64", "assemble", "fp64", 1027, 0.5, 20.0, 4, 24, mode="replay"),
        # detections: an ordinary strand, the largest one, and a large one in double
        _strand("detect_37_mixed", "detect", "mixed", 37, 2.0, 40.0, 4, 32),
        _strand("detect_1027_mixed", "detect", "mixed", 1027, 0.5, 20.0, 4, 24),
        _strand("detect_397_fp64", "detect", "fp64", 397, 0.5, 20.0, 4, 24),
        # the candidates of one detection of the largest strand, scored
        dict(name="score_3200k", kind="score", n=3_197_900),
        # one epoch of the network's training on the labelled pairs of a few small strands
        dict(name="train_200k", kind="train", n=201_347),
        # one Newton step's linear solve of the 7-wire strand
        _strand("solve_7_fp64", "solve", "fp64", 7, 2.0, 40.0, 1, 16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["assemble", "detect", "score", "train", "solve"], [6, 3, 1, 1, 1])[0]
    if kind == "score":
        return dict(kind=kind, n=_log_int(rng, 1_000, 3_197_900))
    if kind == "train":
        return dict(kind=kind, n=_log_int(rng, 1_000, 201_347))
    if kind == "solve":
        return dict(kind=kind, precision=rng.choice(["fp64", "mixed"]), n_wires=7, d=2.0, pitch=40.0,
                    n_pitches=rng.randint(1, 2), el=rng.randint(16, 24))
    precision = rng.choice(["mixed", "mixed", "fp64"])
    if kind == "assemble" and rng.random() < 0.2:
        return dict(kind=kind, precision=precision, n_strands=_log_int(rng, 2, 64), d=2.0, pitch=40.0,
                    mode=rng.choice(["replay", "eager"]))
    options = {}
    if kind == "assemble":
        options["mode"] = rng.choice(["replay", "replay", "eager"])
        if rng.random() < 0.2:
            options["coated"] = True
    d, pitch = rng.choice([(2.0, 40.0), (0.5, 20.0)])
    n_wires = _log_int(rng, 4, 1027)
    n_pitches, el = rng.randint(1, 4), rng.randint(16, 32 if d > 1.0 else 24)
    if options.get("coated"):  # every candidate is a member: the rows of the contact pattern limit the strand
        d, pitch, n_wires, el = 2.0, 40.0, min(n_wires, 91), min(el, 32)
    n_pitches = max(1, min(n_pitches, 98_592 // (n_wires * el)))
    if n_wires * n_pitches * el > 98_592:
        n_wires = 98_592 // (n_pitches * el)
    return dict(kind=kind, precision=precision, n_wires=n_wires, d=d, pitch=pitch, n_pitches=n_pitches, el=el, **options)


# ------------------------------------------------------------------------------------------------ inputs


@functools.lru_cache(maxsize=4)
def _mesh(n_strands, n_wires, d, pitch, n_pitches, el):
    """(strand, bent displacement, mu, k_pen): the parts of a workload that no seed changes."""
    if n_strands:
        w = workloads.batch_workload(n_strands=n_strands, d=d, pitch=pitch)
        return w.strand, np.zeros(w.strand.ndof), w.mu, w.k_pen
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        st = strands.make_strand(n_wires, d, pitch, n_pitches, el * n_pitches, gap=-0.005 * d)
    D = 2.0 * max(w.lay_radius for w in st.wires) + d
    sec = workloads.circle_section(d)
    k_pen = 1e3 * sec["E"] * sec["A"] / workloads.mean_element_length(st.coords, st.conn)
    return st, runs.arc_displacement(st, 1.0 / (50.0 * D)), MU, k_pen


def _mesh_of(case):
    return _mesh(case.get("n_strands", 0), case.get("n_wires", 0), case["d"], case["pitch"], case.get("n_pitches", 0),
                 case.get("el", 0))


def _ends(st):
    """Nodes of one element only: the wires' ends, clamped."""
    return np.flatnonzero(np.bincount(np.asarray(st.conn).ravel(), minlength=st.n_nodes) == 1)


def _last_detection(case, seed):
    """u at the last detection: the bent strand with its noise.  The seed moves the whole strand and stirs it by a
    hair (1e-9 d), so that every value is another one and the candidate set, with it all outputs' sizes, is the
    case's own."""
    st, bend, _, _ = _mesh_of(case)
    fixed, rng = np.random.default_rng(0), np.random.default_rng(seed)
    noise = np.empty((st.n_nodes, 6))
    noise[:, :3] = fixed.normal(0.0, 1e-3 * case["d"], (st.n_nodes, 3))
    noise[:, 3:] = fixed.normal(0.0, 1e-3, (st.n_nodes, 3))
    noise[:, :3] += rng.uniform(-case["d"], case["d"], 3) + rng.normal(0.0, 1e-9 * case["d"], (st.n_nodes, 3))
    return bend + noise.ravel(), rng


def _states(case, seed):
    """u at the last detection, u of the iteration, f_ext and the fixed DOFs (host arrays)."""
    st = _mesh_of(case)[0]
    u0, rng = _last_detection(case, seed)
    step = np.zeros((st.n_nodes, 6))
    step[:, :3] = rng.normal(0.0, 2e-4 * case["d"], (st.n_nodes, 3))
    f_ext = np.zeros((st.n_nodes, 6))
    f_ext[:, :3] = rng.normal(0.0, 1.0, (st.n_nodes, 3))
    fixed = np.zeros((st.n_nodes, 6), dtype=np.uint8)
    fixed[_ends(st)] = 1
    return u0, u0 + step.ravel(), f_ext.ravel(), fixed.ravel()


def _detect_states(case, seed):
    """u of the last detection and of the next two (the oscillation's curvature steps, each with its jitter), and of
    the iteration between."""
    st, bend, _, _ = _mesh_of(case)
    u0 = _last_detection(case, seed)[0]
    rng = np.random.default_rng(1)  # not the seed's: what moves here decides which pairs carry a force later
    jitter = np.zeros((3, st.n_nodes, 6))
    jitter[:, :, :3] = rng.normal(0.0, 3e-4 * case["d"], (3, st.n_nodes, 3))
    us = [u0] + [u0 + (math.cos(2.0 * math.pi * k / 30.0) - 1.0) * bend + jitter[k].ravel() for k in (1, 2)]
    return us, u0 + jitter[0].ravel()


def _features(n, seed):
    """Features as a detection's candidates have them: separation, angle, half length, layers, last gap."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = torch.rand((n, 8), generator=g, device="cuda")
    f = torch.empty((n, 8), device="cuda")
    f[:, 0] = 0.8 + 2.0 * r[:, 0]
    f[:, 1] = 1.0 - 0.4 * r[:, 1]
    f[:, 2] = 0.6 + r[:, 2]
    f[:, 3] = 1.0 / 3.0
    f[:, 4] = (r[:, 4] < 0.02).float()
    f[:, 5] = (f[:, 0] - 1.0 + 0.1 * torch.randn(n, generator=g, device="cuda")).clamp(-2.0, 8.0)
    f[:, 6] = (r[:, 6] < 0.9).float()
    f[:, 7] = 0.0
    y = (f[:, 5] < 0.1).float()
    return f.reshape(-1).contiguous(), y


def _theta(seed):
    th = init_params(seed)
    return (th + np.random.default_rng(seed).normal(0.0, 0.02, th.size)).astype(np.float32)


def _engine(case):
    st, _, mu, k_pen = _mesh_of(case)
    kw = {}
    if case.get("coated"):
        kw = dict(core_radii=0.9 * float(st.radii[0]), coating=COAT)
    eng = AssemblyEngine(st.coords, st.conn, st.radii, workloads.circle_section(case["d"]), layer=st.elem_layer,
                         precision=case["precision"], k_pen=k_pen, k_t_ratio=K_T_RATIO, mu=mu, g_on=G_ON, g_off=G_OFF,
                         **kw)
    eng.autotune = False  # the schedule that the autotuner settles on for strands, without its timing noise
    return eng


def prepare(case, seed):
    kind = case["kind"]
    if kind == "score":
        return dict(kind=kind, n=case["n"], pruner=PairPruner(_theta(seed)), feat=_features(case["n"], seed)[0])
    if kind == "train":
        feat, y = _features(case["n"], seed)
        return dict(kind=kind, n=case["n"], pruner=PairPruner(_theta(seed)), feat=feat, y=y, w=1.0 + 3.0 * y)
    if kind == "solve":
        return _prepare_solve(case, seed)
    eng = _engine(case)
    dev = lambda x: torch.as_tensor(x, device="cuda")  # noqa: E731
    if kind == "detect":
        us, u1 = _detect_states(case, seed)
        eng.detect(dev(us[0]))
        eng.assemble(dev(u1), dev(us[0]))
        return dict(kind=kind, engine=eng, u=[dev(us[1]), dev(us[2])], passes=0)
    u0, u1, f_ext, fixed = (dev(x) for x in _states(case, seed))
    eng.detect(u0)
    eng.end_step()
    s = dict(kind=kind, engine=eng, mode=case["mode"], u=u1, u_ref=u0, f_ext=f_ext, fixed=fixed)
    if case["mode"] == "replay":
        if eng.pattern.c.sides_ok == 1:
            eng.gather_variant = L.XK_GATHER_SIDES
        eng.capture(u1, u0, f_ext, fixed)
    s["results"] = _results(eng)
    return s


def _solve_inputs(case, seed):
    """Loads of a load increment (two smooth modes along every wire, about 1 N a node) and the clamped ends."""
    st = _mesh_of(case)[0]
    rng = np.random.default_rng(seed)
    x = np.asarray(st.coords)[:, 2] / st.length
    f = np.zeros((st.n_nodes, 6))
    for mode in (1, 2):
        f[:, :3] += np.sin(mode * math.pi * x)[:, None] * rng.uniform(-1.0, 1.0, 3)
    fixed = np.zeros((st.n_nodes, 6), dtype=np.uint8)
    fixed[_ends(st)] = 1
    return f.ravel(), fixed.ravel()


def _prepare_solve(case, seed):
    """The first Newton step of a frictionless load increment with k_pen 1e4 N/mm (a positive definite tangent)."""
    st = _mesh_of(case)[0]
    eng = AssemblyEngine(st.coords, st.conn, st.radii, workloads.circle_section(case["d"]), layer=st.elem_layer,
                         precision=case["precision"], k_pen=1e4, k_t_ratio=K_T_RATIO, mu=0.0)
    f_ext, fixed = (torch.as_tensor(x, device="cuda") for x in _solve_inputs(case, seed))
    u = torch.zeros_like(f_ext)
    eng.detect(u)
    b = -eng.assemble(u, u, f_ext, fixed)
    solver = DeviceLinearSolver(eng)
    solver.set_fixed(fixed)
    return dict(kind="solve", engine=eng, solver=solver, b=b)


# ------------------------------------------------------------------------------------------------ one pass

_WIDTH = {"normal": 3, "t1": 3, "t2": 3, "z_t": 2}


def _rows(table, names, n):
    """Views of the first n rows of a structure-of-arrays table."""
    return {k: table.t[k].view(_WIDTH[k], -1)[:, :n] if k in _WIDTH else table.t[k][:n] for k in names}


def _results(eng):
    """The engine's own buffers that an assembly leaves: the table's state, R and its squared norm, K_beam, K_c."""
    table = eng.pairs32 if eng.precision == L.XK_MIXED else eng.pairs
    out = _rows(table, ("s", "t", "gap", "normal", "t1", "p_n", "z_t", "status", "stick"), eng.pairs.n)
    out.update(R=eng.R, norm2=eng.norm2, K_beam=eng.K_beam, K_c=eng.K_c[: 9 * eng.pattern.nnzb])
    return out


def run(state):
    kind = state["kind"]
    if kind == "score":
        return state["pruner"].logits(state["feat"], state["n"])
    if kind == "train":
        p = state["pruner"]
        loss, grad, logit = p.gradient(state["feat"], state["y"], state["w"], state["n"])
        p.adam(grad, 3e-3)
        return dict(loss=loss, grad=grad, logit=logit, theta=p.theta)
    if kind == "solve":
        return state["solver"].solve(state["b"])
    eng = state["engine"]
    if kind == "detect":
        eng.detect(state["u"][state["passes"] % 2])
        state["passes"] += 1
        pat = eng.pattern
        out = _rows(eng.pairs, ("ea", "eb", "s", "t", "gap", "normal", "t1", "t2", "p_n", "z_t", "status"), eng.pairs.n)
        out.update(members=pat.members[: pat.n_members], row_ptr=pat.row_ptr, col=pat.col[: pat.nnzb])
        return out
    if state["mode"] == "replay":
        eng.replay()
    else:
        eng.assemble(state["u"], state["u_ref"], state["f_ext"], state["fixed"])
    return state["results"]


# ------------------------------------------------------------------------------------------------ 64 bits

F64 = torch.float64


def _to(x, dtype=F64):
    return torch.as_tensor(np.ascontiguousarray(x)).to("cuda" if torch.cuda.is_available() else "cpu", dtype)


def _dot(a, b):
    return (a * b).sum(-1)


def _overlaps(lo, hi):
    """Index pairs i < j of the closed boxes [lo, hi] that overlap, sorted: boxes binned by their lower corner in
    cells of the largest extent, each box against the cells that can hold a partner's corner."""
    n = lo.shape[0]
    cell = (hi - lo).max()
    c = ((lo - lo.min(0).values) / cell).floor().long() + 1
    dims = c.max(0).values + 2
    key = (c[:, 2] * dims[1] + c[:, 1]) * dims[0] + c[:, 0]
    order = torch.argsort(key)
    ks = key[order]
    found = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                kk = key + (dz * dims[1] + dy) * dims[0] + dx
                a, b = torch.searchsorted(ks, kk), torch.searchsorted(ks, kk, right=True)
                cnt = b - a
                i = torch.repeat_interleave(torch.arange(n, device=lo.device), cnt)
                off = torch.arange(i.numel(), device=lo.device) - torch.repeat_interleave(cnt.cumsum(0) - cnt, cnt)
                j = order[a[i] + off]
                i, j = i[j > i], j[j > i]
                ok = ((lo[i] <= hi[j]) & (lo[j] <= hi[i])).all(1)
                found.append(i[ok] * n + j[ok])
    k = torch.unique(torch.cat(found))
    return k // n, k % n


def _candidates(st, x):
    """Candidate pairs at node positions x: overlapping boxes, no shared node, not of one layer, and the midpoint test."""
    conn, r = _to(st.conn, torch.long), _to(st.radii)
    a, b = x[conn[:, 0]], x[conn[:, 1]]
    i, j = _overlaps(torch.minimum(a, b) - r[:, None], torch.maximum(a, b) + r[:, None])
    layer = _to(st.elem_layer, torch.long)
    keep = (conn[i][:, :, None] != conn[j][:, None, :]).all(2).all(1) & ((layer[i] != layer[j]) | (layer[i] < 0))
    i, j = i[keep], j[keep]
    mid, half, rs = 0.5 * (a + b), 0.5 * (b - a).norm(dim=1), r[i] + r[j]
    far = ((mid[i] - mid[j]).norm(dim=1) - half[i] - half[j]).clamp_min(0.0)
    keep = far <= rs + 0.5 * rs.mean()
    return i[keep], j[keep]


def _closest(x, nd):
    """Closest points of the segments nd[:, :2] and nd[:, 2:]: parameters, distance, unit normal."""
    p, q, r = x[nd[:, 1]] - x[nd[:, 0]], x[nd[:, 3]] - x[nd[:, 2]], x[nd[:, 0]] - x[nd[:, 2]]
    a, b, c, d, e = _dot(p, p), _dot(p, q), _dot(q, q), _dot(p, r), _dot(q, r)
    det = a * c - b * b
    par = det < 1e-10 * (a * c).clamp_min(1e-30)
    det = torch.where(par, torch.ones_like(det), det)
    su = torch.where(par, torch.zeros_like(det), (b * e - c * d) / det)
    tu = torch.where(par, torch.zeros_like(det), (a * e - b * d) / det)
    s, t = su.clamp(0, 1), torch.where(par, (e / c).clamp(0, 1), tu.clamp(0, 1))
    t = torch.where(((su < 0) | (su > 1)) & ~par, ((b * s + e) / c).clamp(0, 1), t)
    out = ((tu < 0) | (tu > 1)) & ~par
    s = torch.where(out, ((b * t - d) / a).clamp(0, 1), s)
    t = torch.where(out, ((b * s + e) / c).clamp(0, 1), t)
    v = r + s[:, None] * p - t[:, None] * q
    dist = v.norm(dim=1)
    return s, t, dist, v / dist[:, None]


def _frame(n, n_old=None, t_old=None):
    """First tangent of the frame at normal n: the old one turned with the normal, or (fresh rows, n_old zero) the
    projection of the axis that n has least of."""
    ax = torch.zeros_like(n).scatter_(1, n.abs().argmin(1, keepdim=True), 1.0)
    fresh = ax
    if n_old is not None:
        v = torch.linalg.cross(n_old, n, dim=1)
        w = torch.linalg.cross(v, t_old, dim=1)
        turned = t_old + w + torch.linalg.cross(v, w, dim=1) / (1.0 + _dot(n_old, n))[:, None]
        fresh = torch.where((n_old.norm(dim=1) > 0.5)[:, None], turned, ax)
    raw = fresh - _dot(fresh, n)[:, None] * n
    return raw / raw.norm(dim=1, keepdim=True)


def _skew(v):
    z = torch.zeros_like(v[:, 0])
    return torch.stack([z, -v[:, 2], v[:, 1], v[:, 2], z, -v[:, 0], -v[:, 1], v[:, 0], z], 1).view(-1, 3, 3)


def _exp(th):
    a = th.norm(dim=1)[:, None, None]
    S, ok = _skew(th), a > 1e-8
    q = torch.where(ok, a, torch.ones_like(a))
    eye = torch.eye(3, dtype=F64, device=th.device)
    return eye + torch.where(ok, torch.sin(q) / q, torch.ones_like(q)) * S + \
        torch.where(ok, 2.0 * (torch.sin(q / 2) / q) ** 2, 0.5 * torch.ones_like(q)) * (S @ S)


def _log(R):
    """Rotation vectors of rotations by less than pi / 2."""
    v = 0.5 * torch.stack([R[:, 2, 1] - R[:, 1, 2], R[:, 0, 2] - R[:, 2, 0], R[:, 1, 0] - R[:, 0, 1]], 1)
    s = v.norm(dim=1)
    a = torch.atan2(s, 0.5 * (R.diagonal(dim1=1, dim2=2).sum(1) - 1.0))
    return torch.where(s > 1e-12, a / s.clamp_min(1e-300), torch.ones_like(s))[:, None] * v


def _spin(th, inverse):
    """The tangent of the exponential map, or its inverse, by series (rotations here stay well below 1)."""
    S, a2 = _skew(th), _dot(th, th)[:, None, None]
    eye = torch.eye(3, dtype=F64, device=th.device)
    if inverse:
        c = [1 / 12, 1 / 720, 1 / 30240, 1 / 1209600, 1 / 47900160, 691 / 1307674368000, 1 / 74724249600]
        return eye - 0.5 * S + sum(v * a2**k for k, v in enumerate(c)) * (S @ S)
    f = math.factorial
    return eye + sum((-a2) ** k / f(2 * k + 2) for k in range(9)) * S + \
        sum((-a2) ** k / f(2 * k + 3) for k in range(9)) * (S @ S)


def _beam(st, sec, u):
    """Forces (n, 12) and symmetrised tangents (n, 12, 12) of corotational Timoshenko elements."""
    X, conn = _to(st.coords), _to(st.conn, torch.long)
    ua, ub = u.view(-1, 6)[conn[:, 0]], u.view(-1, 6)[conn[:, 1]]
    dx0 = X[conn[:, 1]] - X[conn[:, 0]]
    L0 = dx0.norm(dim=1)
    e0 = dx0 / L0[:, None]
    ez = torch.linalg.cross(e0, torch.zeros_like(e0).scatter_(1, e0.abs().argmin(1, keepdim=True), 1.0), dim=1)
    ez = ez / ez.norm(dim=1, keepdim=True)
    R0 = torch.stack([e0, torch.linalg.cross(ez, e0, dim=1), ez], 1)
    dx = dx0 + ub[:, :3] - ua[:, :3]
    Ld = dx.norm(dim=1)
    ex = dx / Ld[:, None]
    V = _skew(torch.linalg.cross(e0, ex, dim=1))
    eye = torch.eye(3, dtype=F64, device=u.device)
    rod = eye + V + V @ V / (1.0 + _dot(e0, ex))[:, None, None]
    Rc = R0 @ rod.mT
    t1, t2 = (_log(Rc @ _exp(w[:, 3:]) @ R0.mT) for w in (ua, ub))
    E, G, A, Iy, Iz, J = (sec[k] for k in ("E", "G", "A", "Iy", "Iz", "J"))
    K = torch.zeros((L0.numel(), 12, 12), dtype=F64, device=u.device)
    K[:, 0, 0] = K[:, 6, 6] = E * A / L0
    K[:, 0, 6] = K[:, 6, 0] = -E * A / L0
    K[:, 3, 3] = K[:, 9, 9] = G * J / L0
    K[:, 3, 9] = K[:, 9, 3] = -G * J / L0
    for I, kappa, sg, (v1, r1, v2, r2) in ((Iz, sec["kappa_z"], 1.0, (1, 5, 7, 11)), (Iy, sec["kappa_y"], -1.0, (2, 4, 8, 10))):
        phi = 12.0 * E * I / (kappa * G * A * L0 * L0)
        c = E * I / (L0 * (1.0 + phi))
        for i, j, val in ((v1, v1, 12 * c / L0**2), (v1, v2, -12 * c / L0**2), (v2, v2, 12 * c / L0**2),
                          (v1, r1, sg * 6 * c / L0), (v1, r2, sg * 6 * c / L0), (v2, r1, -sg * 6 * c / L0),
                          (v2, r2, -sg * 6 * c / L0), (r1, r1, (4 + phi) * c), (r2, r2, (4 + phi) * c),
                          (r1, r2, (2 - phi) * c)):
            K[:, i, j] = val
            K[:, j, i] = val
    d = torch.zeros((L0.numel(), 12), dtype=F64, device=u.device)
    d[:, 3:6], d[:, 6], d[:, 9:12] = t1, _dot(ub[:, :3] - ua[:, :3], dx + dx0) / (Ld + L0), t2
    f = torch.einsum("nij,nj->ni", K, d)
    dpsi = Rc @ _skew(ex) / Ld[:, None, None]
    B = torch.zeros_like(K)
    B[:, 6, :3], B[:, 6, 6:9] = -ex, ex
    for rows, t, th in ((slice(3, 6), t1, ua[:, 3:]), (slice(9, 12), t2, ub[:, 3:])):
        P = _spin(t, True) @ dpsi
        B[:, rows, :3], B[:, rows, 6:9], B[:, rows, rows] = P, -P, _spin(t, True) @ Rc @ _spin(th, False)
    M = K @ B
    for b in range(4):
        g = _skew(f[:, 3 * b:3 * b + 3]) @ dpsi
        M[:, 3 * b:3 * b + 3, :3] += g
        M[:, 3 * b:3 * b + 3, 6:9] -= g
    T = torch.block_diag(*[torch.ones(3, 3)] * 4).to(M)
    Rb = Rc.repeat(1, 4, 4) * T
    Kg = Rb.mT @ M
    return torch.einsum("nji,nj->ni", Rb, f), 0.5 * (Kg + Kg.mT)


def _upper(n, rows, cols, blocks):
    """Sums of the blocks at equal (row, col), row <= col, in ascending order of (row, col)."""
    keep = rows <= cols
    key, inv = torch.unique(rows[keep] * n + cols[keep], return_inverse=True)
    return torch.zeros((key.numel(), *blocks.shape[1:]), dtype=F64, device=blocks.device).index_add_(0, inv, blocks[keep])


def _exact_assemble(case, seed):
    st, _, mu, k_pen = _mesh_of(case)
    u0, u1, f_ext, fixed = _states(case, seed)
    u0, u1, X = _to(u0), _to(u1), _to(st.coords)
    conn, r = _to(st.conn, torch.long), _to(st.radii)
    n = st.n_nodes
    x0, x1 = X + u0.view(-1, 6)[:, :3], X + u1.view(-1, 6)[:, :3]
    i, j = _candidates(st, x0)
    nd = torch.cat([conn[i], conn[j]], 1)
    coated = bool(case.get("coated"))
    rs = r[i] + r[j]
    core = 0.9 * rs if coated else rs
    thick = rs - core
    _, _, dist, nrm = _closest(x0, nd)
    gap0 = dist - core
    cc0 = (thick - gap0).clamp_min(0.0)
    active = (gap0 <= G_ON) | (coated & (cc0 > 0.0))
    member = active | coated
    tan = _frame(nrm)
    mu = _to(mu)[i] if np.ndim(mu) else torch.full_like(rs, mu)
    z, zc = torch.zeros((i.numel(), 2), dtype=F64, device=X.device), torch.zeros((i.numel(), 2), dtype=F64, device=X.device)
    du = (u1 - u0).view(-1, 6)[:, :3]
    s, t, dist, n1 = _closest(x1, nd)
    gap = dist - core
    p_n = torch.where(active, k_pen * (-gap).clamp_min(0.0), torch.zeros_like(gap))
    cs = torch.stack([1 - s, s, t - 1, -t], 1)
    slip = -torch.einsum("pk,pkc->pc", cs, du[nd])
    kt = k_pen * K_T_RATIO
    cc = (thick - gap).clamp_min(0.0)

    def returned(z, k, limit):
        q = z + k * rel
        qn = q.norm(dim=1)
        stick = qn <= limit
        return torch.where(stick[:, None], q, (limit / qn.clamp_min(1e-300))[:, None] * q), qn, stick

    def stiffness(k, limit, q, qn, stick):
        h = q / q.norm(dim=1, keepdim=True).clamp_min(1e-300)
        eye = torch.eye(2, dtype=F64, device=X.device)
        ratio = (limit / qn.clamp_min(1e-300))[:, None, None]
        D = torch.where(stick[:, None, None], k * eye, ratio * k * (eye - h[:, :, None] * h[:, None, :]))
        return torch.einsum("pab,pai,pbj->pij", D, tv, tv)

    for _ in range(2 if case["mode"] == "replay" else 1):  # recording the graph assembles once
        tan = _frame(n1, nrm, tan)
        nrm = n1
        tv = torch.stack([tan, torch.linalg.cross(n1, tan, dim=1)], 1)
        rel = torch.einsum("pac,pc->pa", tv, slip)
        fric = p_n > 0.0
        q, qn, stick = returned(z, kt, mu * p_n)
        z = torch.where(fric[:, None], q, z)
        if coated:
            qc, qnc, stick_c = returned(zc, COAT["stiffness"] * COAT["k_t_ratio"], COAT["mu"] * COAT["stiffness"] * cc)
            zc = torch.where((cc > 0)[:, None], qc, torch.zeros_like(zc))
    v = p_n[:, None] * n1 + torch.einsum("pa,pac->pc", torch.where(fric[:, None], q, torch.zeros_like(q)), tv)
    full = gap + rs  # the geometric terms take the outer radii
    eye = torch.eye(3, dtype=F64, device=X.device)
    nn = n1[:, :, None] * n1[:, None, :]
    use = (p_n > 0.0)[:, None, None]
    Bl = torch.where(use, k_pen * nn - (p_n / full)[:, None, None] * (eye - nn), torch.zeros_like(nn))
    M = -q[:, :1, None] * n1[:, :, None] * tv[:, 0][:, None, :] - q[:, 1:, None] * tv[:, 1][:, :, None] * n1[:, None, :]
    M = M - q[:, 1:, None] * _skew(tv[:, 0])
    Bf = stiffness(kt, mu * p_n, q, qn, stick) + M / full[:, None, None]
    Bl = Bl - torch.where(use & (q.norm(dim=1) > 0)[:, None, None], Bf, torch.zeros_like(Bf))
    if coated:
        k, c = COAT["stiffness"], COAT["damping"] / COAT["dt"]
        prev = cc0  # the converged step's compression: that of the detection
        touch = (cc > 0) | (prev > 0)
        v = v - torch.where(touch, k * cc + c * (cc - prev), torch.zeros_like(cc))[:, None] * n1
        v = v - torch.einsum("pa,pac->pc", zc, tv)
        pressed = (cc > 0)[:, None, None]
        Bc = (k + c) * nn + stiffness(k * COAT["k_t_ratio"], COAT["mu"] * k * cc, zc, qnc, stick_c)
        Bl = Bl + torch.where(pressed, Bc, torch.zeros_like(Bc))
    fe, Ke = _beam(st, workloads.circle_section(case["d"]), u1)
    R = torch.zeros((n, 6), dtype=F64, device=X.device)
    R.index_add_(0, conn.reshape(-1), fe.view(-1, 2, 6).reshape(-1, 6))
    R[:, :3].index_add_(0, nd.reshape(-1), -(cs[:, :, None] * v[:, None, :]).reshape(-1, 3))
    R = R.view(-1) - _to(f_ext)
    R[_to(fixed, torch.bool)] = 0.0
    rows, cols = conn[:, [0, 0, 1, 1]].reshape(-1), conn[:, [0, 1, 0, 1]].reshape(-1)
    blocks = Ke.view(-1, 2, 6, 2, 6).permute(0, 1, 3, 2, 4).reshape(-1, 6, 6)
    K_beam = _upper(n, rows, cols, blocks)
    m = member.nonzero()[:, 0]
    blocks = (cs[m][:, :, None] * cs[m][:, None, :]).reshape(-1, 1, 1) * Bl[m].repeat_interleave(16, 0)
    K_c = _upper(n, nd[m].repeat_interleave(4, 1).reshape(-1), nd[m].repeat(1, 4).reshape(-1), blocks)
    order = torch.arange(i.numel(), device=X.device)
    if case["precision"] == "mixed":  # the float table holds the contributing pairs first
        order = torch.cat([m, (~member).nonzero()[:, 0]])
    row = lambda x: x[order].T if x.dim() > 1 else x[order]  # noqa: E731
    return dict(s=row(s), t=row(t), gap=row(gap), normal=row(n1), t1=row(tan), p_n=row(p_n), z_t=row(z), status=None,
                stick=None, R=R, norm2=_dot(R, R).reshape(1), K_beam=K_beam.reshape(-1), K_c=K_c.reshape(-1))


def _exact_detect(case, seed):
    """The table after one detection: the pairs of both, the old ones' frames turned on, the state carried over."""
    st, _, mu, k_pen = _mesh_of(case)
    (u0, ua, _), u1 = _detect_states(case, seed)
    X, conn, r = _to(st.coords), _to(st.conn, torch.long), _to(st.radii)
    at = lambda u: X + _to(u).view(-1, 6)[:, :3]  # noqa: E731
    ne = st.n_elems
    i, j = _candidates(st, at(u0))
    old = i * ne + j
    nd = torch.cat([conn[i], conn[j]], 1)
    _, _, dist, n0 = _closest(at(u0), nd)
    active = dist - (r[i] + r[j]) <= G_ON
    s, t, dist, n1 = _closest(at(u1), nd)
    tan = _frame(n1, n0, _frame(n0))
    p_n = torch.where(active, k_pen * (r[i] + r[j] - dist).clamp_min(0.0), torch.zeros_like(dist))
    du = (_to(u1) - _to(u0)).view(-1, 6)[:, :3]
    slip = -torch.einsum("pk,pkc->pc", torch.stack([1 - s, s, t - 1, -t], 1), du[nd])
    tv = torch.stack([tan, torch.linalg.cross(n1, tan, dim=1)], 1)
    q = k_pen * K_T_RATIO * torch.einsum("pac,pc->pa", tv, slip)
    qn = q.norm(dim=1)
    q = torch.where((qn <= mu * p_n)[:, None], q, (mu * p_n / qn.clamp_min(1e-300))[:, None] * q)
    q = torch.where((p_n > 0)[:, None], q, torch.zeros_like(q))
    x = at(ua)
    k, l = _candidates(st, x)
    both = torch.unique(torch.cat([old, k * ne + l]))
    where = torch.searchsorted(both, old)
    carry = lambda v: torch.zeros((both.numel(), *v.shape[1:]), dtype=F64, device=X.device).index_copy_(0, where, v)  # noqa: E731
    n_old, t_old = carry(n1), carry(tan)
    i, j = both // ne, both % ne
    s, t, dist, n1 = _closest(x, torch.cat([conn[i], conn[j]], 1))
    tan = _frame(n1, n_old, t_old)
    row = lambda v: v.T if v.dim() > 1 else v  # noqa: E731
    return dict(ea=None, eb=None, s=row(s), t=row(t), gap=row(dist - (r[i] + r[j])), normal=row(n1), t1=row(tan),
                t2=row(torch.linalg.cross(n1, tan, dim=1)), p_n=row(carry(p_n)), z_t=row(carry(q)), status=None,
                members=None, row_ptr=None, col=None)


def _bf16(x):
    return x.float().to(torch.bfloat16).to(F64)


def _layers(theta):
    out, at = [], 0
    for rows, cols in ((64, 8), (64, 64), (64, 64), (1, 64)):
        W = _bf16(theta[at:at + rows * cols]).view(rows, cols)
        at += rows * cols
        out.append((W, _bf16(theta[at:at + rows])))
        at += rows
    return out


def _network(case, seed):
    """The network's layers and activations: bfloat16 weights and activations, sums in 64 bits."""
    feat, y = _features(case["n"], seed)
    layers = _layers(torch.as_tensor(_theta(seed), device="cuda"))
    acts = [_bf16(feat.view(-1, 8))]
    for W, b in layers[:3]:
        acts.append(_bf16((acts[-1] @ W.T + b).clamp_min(0.0)))
    W, b = layers[3]
    return layers, acts, (acts[-1] @ W.T + b)[:, 0], y


def _exact_train(case, seed):
    layers, acts, logit, y = _network(case, seed)
    y = y.to(F64)
    w, n = 1.0 + 3.0 * y, y.numel()
    loss = (w * (torch.nn.functional.softplus(logit) - y * logit)).sum() / n
    d = (w * (torch.sigmoid(logit) - y) / n)[:, None]
    grads = []
    for k in (3, 2, 1, 0):
        grads = [(d.T @ acts[k]).reshape(-1), d.sum(0)] + grads
        if k:
            d = (d @ layers[k][0]) * (acts[k] > 0)
    grad = torch.cat(grads)
    theta = torch.as_tensor(_theta(seed), device="cuda", dtype=F64)
    step = 3e-3 * grad / (grad.abs() + 1e-8)  # Adam's first step: both corrected moments are the gradient's own
    return dict(loss=loss.reshape(1), grad=grad, logit=logit, theta=theta - step)


def _exact_solve(case, seed):
    """The solution of the assembled system by a dense factorisation in 64 bits (the matrix is the solve's input)."""
    s = _prepare_solve(case, seed)
    eng = s["engine"]
    fixed = _to(_solve_inputs(case, seed)[1], torch.bool)
    K = _to(eng.K_total_csr().toarray())
    K[fixed, :] = 0.0
    K[:, fixed] = 0.0
    K[fixed, fixed] = 1.0
    return torch.linalg.solve(K, s["b"].to(K))


def exact(case, seed):
    with torch.no_grad():
        kind = case["kind"]
        if kind == "assemble":
            return _exact_assemble(case, seed)
        if kind == "detect":
            return _exact_detect(case, seed)
        if kind == "score":
            return _network(case, seed)[2]
        return _exact_train(case, seed) if kind == "train" else _exact_solve(case, seed)


# ------------------------------------------------------------------------------------------------ work


@functools.lru_cache(maxsize=64)
def _counts(n_strands, n_wires, d, pitch, n_pitches, el, coated):
    """(nodes, elements, pairs, contributing pairs, K_c blocks) at the unloaded state of seed 0."""
    case = dict(n_strands=n_strands, n_wires=n_wires, d=d, pitch=pitch, n_pitches=n_pitches, el=el)
    st = _mesh_of(case)[0]
    x = _to(st.coords) + _to(_states(case, 0)[0]).view(-1, 6)[:, :3]
    conn, r = _to(st.conn, torch.long), _to(st.radii)
    i, j = _candidates(st, x)
    nd = torch.cat([conn[i], conn[j]], 1)
    m = nd if coated else nd[_closest(x, nd)[2] - (r[i] + r[j]) <= G_ON]
    rows, cols = m.repeat_interleave(4, 1).reshape(-1), m.repeat(1, 4).reshape(-1)
    blocks = torch.unique((rows * st.n_nodes + cols)[rows <= cols]).numel()
    return st.n_nodes, st.n_elems, int(i.numel()), int(m.shape[0]), int(blocks)


def work(case):
    kind = case["kind"]
    if kind == "score":  # the features in, the scores out; the network's products
        return dict(bytes=case["n"] * 36, flops=case["n"] * 2 * (8 * 64 + 2 * 64 * 64 + 64))
    if kind == "train":  # forward, backward and weight gradients
        return dict(bytes=case["n"] * 44, flops=case["n"] * 6 * (8 * 64 + 2 * 64 * 64 + 64))
    nn, ne, pairs, members, blocks = _counts(case.get("n_strands", 0), case.get("n_wires", 0), case["d"], case["pitch"],
                                             case.get("n_pitches", 0), case.get("el", 0), bool(case.get("coated")))
    size = 4 if case["precision"] == "mixed" else 8
    if kind == "solve":  # the matrix once, the right-hand side and the solution; one product with the matrix
        return dict(bytes=size * (36 * (nn + ne) + 9 * blocks) + 96 * nn, flops=4 * (36 * (nn + ne) + 9 * blocks))
    if kind == "detect":  # the mesh and u in; each pair's state in and out; the contact pattern out
        return dict(bytes=72 * nn + 28 * ne + 300 * pairs + 28 * members + 4 * (nn + blocks), flops=250 * pairs + 60 * ne)
    state = 15 * size + 16  # frame in, frame, parameters and gap out, node numbers
    more = 12 * size + 4  # the contributing pairs' friction state in and out, their second tangent out
    return dict(bytes=state * pairs + more * members + nn * (24 + 96 + 48) + ne * 48 + size * (36 * (nn + ne) + 9 * blocks),
                flops=180 * pairs + 250 * members + 16 * 9 * 2 * members + 1500 * ne)
