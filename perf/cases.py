"""The work that users of this framework have it do, as measurable cases.

A feasibility pump solves the root LP of a model once, scales the model, builds a
projector and then projects one rounded target after another: each projection is
``set_target_unscaled`` -> ``solve`` -> ``get_unscaled``.  The cases cover these calls
through their public entry points, on the synthetic model families of
``pdfp_b200/synthetic.py`` (drawn here on the GPU, so that large models are made quickly):

* ``projection`` -- one projection on a single-model handle, FP64 (the default) or mixed;
* ``batch``      -- one projection of every member of a batch handle;
* ``root_lp``    -- a whole root-LP call (upload, scaling, norm estimate, solve);
* ``scaling``    -- a whole ``scale_problem`` call.

A projection runs a fixed number of evaluation windows of 200 PDHG iterations (its
tolerance is tighter than it reaches), so that every pass does the same work.  The
answer of a mixed handle carries FP32 accuracy and is returned as float32.
"""
import functools
import math

import numpy as np
import scipy.sparse as sp
import torch

from pdfp_b200 import gpu
from pdfp_b200.milp import MILP
from pdfp_b200.params import SolverParameters

FREQ = 200       # PDHG iterations per evaluation window (the default frequency)
EPS = 1e-9       # not reached within the windows run here
ROOT_TOL = 1e-2  # the pump's root-LP tolerance


def listed():
    return [
        # the smallest pump models: a 133-row pure-binary covering model, three windows as
        # in the published p0201 run (400-600 iterations per projection); latency decides
        {"name": "projection cover 133x201", "path": "projection", "model": "cover",
         "rows": 133, "cols": 201, "nnz": 1923, "precision": "fp64", "windows": 3},
        # two concurrent trajectories on a dense equality-knapsack model
        {"name": "batch knapsack 6x56 x2", "path": "batch", "model": "knapsack",
         "rows": 6, "cols": 56, "nnz": 306, "members": 2, "precision": "fp64", "windows": 3},
        # a model near the upper end of what one thread block handles; ragged sizes
        {"name": "projection general 601x1503", "path": "projection", "model": "general",
         "rows": 601, "cols": 1503, "nnz": 15025, "precision": "fp64", "windows": 2},
        # a typical MIPLIB-sized model, in the default precision
        {"name": "projection general 4001x10007", "path": "projection", "model": "general",
         "rows": 4001, "cols": 10007, "nnz": 100025, "precision": "fp64", "windows": 2},
        # the general-integer benchmark model, in both precisions
        {"name": "projection general 20k mixed", "path": "projection", "model": "general",
         "rows": 20000, "cols": 50000, "nnz": 500000, "precision": "mixed", "windows": 2},
        {"name": "projection general 20k fp64", "path": "projection", "model": "general",
         "rows": 20000, "cols": 50000, "nnz": 500000, "precision": "fp64", "windows": 2},
        # Zipf-skewed row lengths, the headline benchmark's family: a model that streams
        # from memory in the mixed form, and one in the default FP64 form
        {"name": "projection zipf 20M mixed", "path": "projection", "model": "zipf",
         "rows": 1000000, "cols": 2000000, "nnz": 20000000, "precision": "mixed", "windows": 2},
        {"name": "projection zipf 6M fp64", "path": "projection", "model": "zipf",
         "rows": 300000, "cols": 600000, "nnz": 6000000, "precision": "fp64", "windows": 1},
        # independent covering and packing models of uneven size in one handle
        {"name": "batch uneven mixed", "path": "batch", "model": "uneven",
         "rows": 24000, "cols": 40000, "nnz": 600000, "members": 8, "precision": "mixed",
         "windows": 2},
        # whole root-LP calls: a small model, and a typical one
        {"name": "root LP cover 133x201", "path": "root_lp", "model": "cover",
         "rows": 133, "cols": 201, "nnz": 1923, "precision": "fp64"},
        {"name": "root LP cover 2k", "path": "root_lp", "model": "cover",
         "rows": 2400, "cols": 4000, "nnz": 60000, "precision": "fp64"},
        # the preconditioner on the general-integer benchmark model
        {"name": "scaling general 20k", "path": "scaling", "model": "general",
         "rows": 20000, "cols": 50000, "nnz": 500000},
    ]


def draw(rng):
    def log_uniform(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    path = rng.choice(["projection", "projection", "projection", "batch", "root_lp", "scaling"])
    case = {"path": path}
    if path in ("projection", "scaling"):
        model = rng.choice(["cover", "general", "zipf"] if path == "projection" else ["general"])
        lo, hi = {"cover": (500, 40_000), "general": (2_000, 1_000_000), "zipf": (50_000, 4_000_000)}[model]
        nnz = log_uniform(lo, hi)
        per_row = {"cover": 14, "general": 25, "zipf": 20}[model] * rng.uniform(0.6, 1.4)
        rows = max(8, int(nnz / per_row))
        case.update(model=model, rows=rows, cols=int(rows * rng.uniform(1.2, 2.6)) + 1, nnz=nnz)
        if path == "projection":
            case.update(precision=rng.choice(["fp64", "mixed"]), windows=rng.choice([1, 2]))
    elif path == "batch":
        model = rng.choice(["knapsack", "uneven"])
        if model == "knapsack":
            rows, binaries = rng.randint(4, 9), rng.randint(30, 70)
            case.update(model=model, rows=rows, cols=binaries + rows, nnz=rows * (binaries + 1),
                        members=rng.randint(2, 6), precision="fp64", windows=rng.choice([1, 2, 3]))
        else:
            cols = log_uniform(2_000, 40_000)
            case.update(model=model, rows=int(0.6 * cols), cols=cols, nnz=int(0.6 * cols) * 25,
                        members=rng.randint(2, 8), precision=rng.choice(["fp64", "mixed"]),
                        windows=rng.choice([1, 2]))
    else:
        nnz = log_uniform(600, 60_000)
        rows = max(8, int(nnz / rng.uniform(10.0, 25.0)))
        case.update(model="cover", rows=rows, cols=int(rows * rng.uniform(1.4, 2.2)) + 1, nnz=nnz,
                    precision="fp64")
    return case


# ---- models ---------------------------------------------------------------------------


def _csr(rows, cols, vals_of, m, n, nnz, g):
    """A canonical scipy CSR matrix, on the host, of exactly nnz distinct positions: those
    given, topped up with uniform ones where some repeat, then thinned at random."""
    key = torch.unique(rows * n + cols)  # sorted
    while len(key) < nnz:
        more = torch.randint(0, m * n, (nnz - len(key),), generator=g, device=key.device)
        key = torch.unique(torch.cat([key, more]))
    if len(key) > nnz:
        keep = torch.randperm(len(key), generator=g, device=key.device)[:nnz]
        key = key[torch.sort(keep).values]
    r = key // n
    ptr = torch.zeros(m + 1, dtype=torch.int64, device=key.device)
    torch.cumsum(torch.bincount(r, minlength=m), 0, out=ptr[1:])
    vals = vals_of(nnz).to(torch.float64)
    A = sp.csr_matrix((vals.cpu().numpy(), (key - r * n).to(torch.int32).cpu().numpy(),
                       ptr.to(torch.int32).cpu().numpy()), shape=(m, n))
    A.has_sorted_indices = True
    A.has_canonical_format = True
    return A


def _model(kind, m, n, nnz, seed):
    """One model and an integer-feasible-looking target point, from the seed alone."""
    dev = "cuda"
    g = torch.Generator(device=dev).manual_seed(int(seed) * 1000003 + m * 31 + n)

    def ints(lo, hi, k):
        return torch.randint(lo, hi, (k,), generator=g, device=dev)

    def uni(k):
        return torch.rand(k, generator=g, device=dev, dtype=torch.float64)

    if kind == "knapsack":  # equality knapsacks with one bounded slack each
        p = n - m
        a = ints(0, 100, m * p).reshape(m, p).to(torch.float64).cpu().numpy()
        A = sp.hstack([sp.csr_matrix(a), sp.eye(m)]).tocsr()
        A.sort_indices()
        return MILP(np.concatenate([np.zeros(p), np.ones(m)]), 0.0, A, np.floor(a.sum(axis=1) / 2.0),
                    ["eq"] * m, np.zeros(n), np.concatenate([np.ones(p), np.full(m, 1000.0)]),
                    np.arange(p))
    if kind in ("cover", "pack"):  # pure binary, coefficients 1..5, spread uniformly
        rows = torch.cat([torch.arange(m, device=dev), ints(0, m, n), ints(0, m, max(nnz - m - n, 0))])
        cols = torch.cat([ints(0, n, m), torch.arange(n, device=dev), ints(0, n, max(nnz - m - n, 0))])
        A = _csr(rows, cols, lambda k: ints(1, 6, k), m, n, nnz, g)
        total = np.asarray(A.sum(axis=1)).ravel()
        c = ints(1, 101, n).to(torch.float64).cpu().numpy()
        if kind == "cover":
            return MILP(c, 0.0, -A, -(1.0 + np.floor(0.3 * total)), ["le"] * m, np.zeros(n),
                        np.ones(n), np.arange(n))
        return MILP(-c, 0.0, A, np.floor(0.5 * total), ["le"] * m, np.zeros(n), np.ones(n),
                    np.arange(n))
    if kind == "general":  # Poisson row lengths, 90% general integers, a quarter equalities
        lengths = torch.poisson(torch.full((m,), nnz / m, device=dev), generator=g).long().clamp_(1, n)
        rows = torch.repeat_interleave(torch.arange(m, device=dev), lengths)
        A = _csr(rows, ints(0, n, len(rows)),
                 lambda k: torch.round(torch.randn(k, generator=g, device=dev, dtype=torch.float64) * 100) / 100 + 0.005,
                 m, n, nnz, g)
        is_int = uni(n).cpu().numpy() < 0.9
        u = np.where(is_int, 10.0, 100.0)
        x0 = np.floor(uni(n).cpu().numpy() * (u + 1.0))
        m_eq = m // 4
        b = A @ x0
        b[: m - m_eq] += 5.0 * uni(m - m_eq).cpu().numpy()
        c = 2.0 * uni(n).cpu().numpy() - 1.0
        return MILP(c, 0.0, A, b, ["le"] * (m - m_eq) + ["eq"] * m_eq, np.zeros(n), u,
                    np.nonzero(is_int)[0])
    # zipf: Zipf(1.5) row lengths capped at 10,000, half binary, half continuous in [0, 1]
    raw = torch.floor(uni(m).clamp_(min=1e-12) ** -2.0).clamp_(max=10000.0)
    lengths = torch.floor(raw * (nnz / raw.sum())).clamp_(1.0, min(10000.0, n)).long()
    rows = torch.repeat_interleave(torch.arange(m, device=dev), lengths)
    A = _csr(rows, ints(0, n, len(rows)), lambda k: 2.0 * uni(k) - 1.0, m, n, nnz, g)
    xf = uni(n).cpu().numpy()
    xf[: n // 2] = np.round(xf[: n // 2])
    b = A @ xf + uni(m).cpu().numpy()
    return MILP(np.zeros(n), 0.0, A, b, ["le"] * m, np.zeros(n), np.ones(n), np.arange(n // 2))


def _members(case):
    """(kind, rows, cols, nonzeros) of each model of a case; an uneven batch spreads its
    members' sizes over a factor of 40 below the given one, covering and packing in turn."""
    if case["path"] != "batch":
        return [(case["model"], case["rows"], case["cols"], case["nnz"])]
    k = case["members"]
    if case["model"] == "knapsack":
        return [("knapsack", case["rows"], case["cols"], case["nnz"])] * k
    out = []
    for p in range(k):
        f = 40.0 ** (-p / max(k - 1, 1))
        n = max(int(case["cols"] * f), 40)
        m = max(int(case["rows"] * f), 24)
        out.append(("cover" if p % 2 == 0 else "pack", m, n, max(int(case["nnz"] * f), m + n)))
    return out


def _models(case, seed):
    if case["model"] == "knapsack" and case["path"] == "batch":  # trajectories of one model
        one = _model(*_members(case)[0], seed)
        return [one] * case["members"]
    return [_model(*mm, seed * 64 + p) for p, mm in enumerate(_members(case))]


def _targets(milp, seed):
    """A rounded target and the same with 5% of its integer entries moved by one, as the
    pump's successive targets are."""
    rng = np.random.default_rng([int(seed), len(milp.c)])
    I = np.asarray(milp.int_idx)
    a = np.zeros(len(milp.c))
    a[I] = np.round(milp.l[I] + rng.random(len(I)) * (milp.u[I] - milp.l[I]))
    b = a.copy()
    idx = I[rng.random(len(I)) < 0.05]
    up = np.minimum(b[idx] + 1, milp.u[idx])
    b[idx] = np.where(up != b[idx], up, np.maximum(b[idx] - 1, milp.l[idx]))
    return a, b


def _con_lb(milp):
    return np.where(milp.is_eq, milp.b, -np.inf)


def _weights(milp, D_c):
    w = np.ones(len(milp.c))
    w[milp.int_idx] = D_c[milp.int_idx]
    return w


def _is_int(milp):
    f = np.zeros(len(milp.c), dtype=np.uint8)
    f[milp.int_idx] = 1
    return f


# ---- the four calls -------------------------------------------------------------------


def prepare(case, seed):
    models = _models(case, seed)
    state = {"case": case, "models": models, "calls": 0}
    if case["path"] in ("root_lp", "scaling"):
        return state
    scaled = [gpu.scale_problem(mm.A, np.zeros(len(mm.c)), mm.l, mm.u, _con_lb(mm), mm.b,
                                bound_objective_rescaling=False) for mm in models]
    problems = [(s.A, s.con_ub, mm.is_eq, _is_int(mm), s.var_lb, s.var_ub, _weights(mm, s.D_c),
                 1.0 / s.D_r) for mm, s in zip(models, scaled)]
    if case["path"] == "projection":
        p = problems[0]
        h = gpu.PDFPState(*p[:7], precision=case["precision"], row_unscale=p[7])
        h.set_col_scale(scaled[0].D_c)
    else:
        h = gpu.PDFPBatch(problems, precision=case["precision"])
        for p, s in enumerate(scaled):
            h.set_col_scale(p, s.D_c)
    # targets and answers in page-locked arrays, as the pump keeps them
    state["targets"] = [[], []]
    state["x"] = []
    for p, mm in enumerate(models):
        for k, t in enumerate(_targets(mm, seed * 64 + p)):
            pinned = gpu.pinned_zeros(len(t))
            pinned[:] = t
            state["targets"][k].append(pinned)
        state["x"].append(gpu.pinned_zeros(len(mm.c)))
    state["handle"] = h
    state["params"] = SolverParameters(eps_optimal_relative=EPS, eps_feasible_relative=EPS,
                                       iteration_limit=FREQ * case["windows"])
    return state


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "root_lp":
        x, slack, status, its = gpu.solve_lp_relaxation(state["models"][0], tolerance=ROOT_TOL,
                                                        precision=case["precision"])
        return {"x": x, "dual_slack": slack, "iterations": its, "optimal": status == "OPTIMAL"}
    if path == "scaling":
        mm = state["models"][0]
        s = gpu.scale_problem(mm.A, mm.c, mm.l, mm.u, _con_lb(mm), mm.b)
        return {"values": s.A.data, "c": s.c, "var_ub": s.var_ub, "con_ub": s.con_ub, "D_r": s.D_r,
                "D_c": s.D_c, "bound_scale": s.bound_scale, "objective_scale": s.objective_scale}
    h, targets = state["handle"], state["targets"][state["calls"] % 2]
    state["calls"] += 1
    kind = np.float32 if case["precision"] == "mixed" else np.float64
    if path == "projection":
        h.set_target_unscaled(targets[0])
        h.solve(state["params"], 1.0)
        x = h.get_unscaled("pdhg_x", out=state["x"][0])
        return {"x": x.astype(kind, copy=False), "iterations": h.total_count}
    for p, t in enumerate(targets):
        h.set_target_unscaled(p, t)
    h.solve(state["params"], 1.0)
    return {"x": [h.get_unscaled(p, "pdhg_x", out=o).astype(kind, copy=False)
                  for p, o in enumerate(state["x"])],
            "iterations": [r["total_count"] for r in h.results]}


def work(case):
    """The algorithm's own bytes and operations.  A PDHG iteration multiplies by A and by
    A' (4 operations per nonzero); with s-byte reals it reads both matrices (an index and
    a value per nonzero), the iterates, anchors and data, and writes the new iterates --
    in FP32 16 nnz + 52 n + 24 m bytes.  A root LP is counted as its first window, whatever
    it takes to converge; a scaling reads the model and writes it back once."""
    total = {"bytes": 0.0, "flops": 0.0}
    for _, m, n, nnz in _members(case):
        if case["path"] == "scaling":
            total["bytes"] += 20.0 * nnz + 64.0 * n + 40.0 * m
            total["flops"] += 44.0 * nnz
            continue
        s = 4.0 if case.get("precision") == "mixed" and sum(q[3] for q in _members(case)) >= 1 << 18 else 8.0
        its = FREQ * case.get("windows", 1)
        total["bytes"] += its * (2 * (4 + s) * nnz + (12 * s + 4) * n + (5 * s + 4) * m)
        total["flops"] += its * (4.0 * nnz + 20.0 * n + 10.0 * m)
    return total


# ---- the same in 64 bits, in plain torch -----------------------------------------------


def _scale64(A, c, lb, ub, clb, cub, rescale):
    """Ten Ruiz rounds, then Pock-Chambolle, then the bound and objective scales."""
    m, n = A.shape
    dev = "cuda"
    ptr = torch.from_numpy(A.indptr.astype(np.int64)).to(dev)
    col = torch.from_numpy(A.indices.astype(np.int64)).to(dev)
    row = torch.repeat_interleave(torch.arange(m, device=dev), ptr[1:] - ptr[:-1])
    v = torch.from_numpy(A.data.copy()).to(dev)
    Dr, Dc = torch.ones(m, dtype=v.dtype, device=dev), torch.ones(n, dtype=v.dtype, device=dev)

    def inv_root(t):
        return torch.where(t < 1e-12, torch.ones_like(t), 1.0 / torch.sqrt(t))

    for k in range(11):
        a = v.abs()
        r, q = torch.zeros_like(Dr), torch.zeros_like(Dc)
        if k < 10:
            r.scatter_reduce_(0, row, a, "amax")
            q.scatter_reduce_(0, col, a, "amax")
        else:
            r.index_add_(0, row, a)
            q.index_add_(0, col, a)
        r, q = inv_root(r), inv_root(q)
        v = v * (r[row] * q[col])
        Dr, Dc = Dr * r, Dc * q
    As = torch.sparse_csr_tensor(ptr, col, v, size=(m, n))
    Dr, Dc = Dr.cpu().numpy(), Dc.cpu().numpy()
    out = {"A": As, "c": c * Dc, "lb": lb / Dc, "ub": ub / Dc, "clb": clb * Dr, "cub": cub * Dr,
           "Dr": Dr, "Dc": Dc, "bs": 1.0, "os": 1.0}
    if rescale:
        two = np.isfinite(clb) & (np.abs(out["clb"] - out["cub"]) > 1e-12)
        sq = np.sum(np.where(two, out["clb"], 0.0) ** 2) + np.sum(out["cub"] ** 2)
        out["bs"], out["os"] = 1.0 / (math.sqrt(sq) + 1.0), 1.0 / (np.linalg.norm(out["c"]) + 1.0)
        for key in ("clb", "cub", "lb", "ub"):
            out[key] = out[key] * out["bs"]
        out["c"] = out["c"] * out["os"]
    return out


def _transpose(A):
    t = A.to_sparse_coo().t().coalesce().to_sparse_csr()
    return torch.sparse_csr_tensor(t.crow_indices(), t.col_indices(), t.values(), size=t.shape)


@functools.lru_cache(maxsize=2)
def _start_vector(m):
    """The norm estimate's start vector: SplitMix64 uniforms through Box-Muller."""
    with np.errstate(over="ignore"):
        z = np.uint64(20240517) + np.arange(1, 2 * m + 1, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z = z ^ (z >> np.uint64(31))
    u = ((z >> np.uint64(11)).astype(np.float64) + 0.5) * 2.0 ** -53
    return np.sqrt(-2.0 * np.log(u[0::2])) * np.cos(6.283185307179586 * u[1::2])


def _norm64(A, At):
    eig = torch.from_numpy(_start_vector(A.shape[0])).to("cuda")
    sq = 1.0
    for _ in range(5000):
        nrm = eig.norm()
        if float(nrm) == 0.0:
            break
        nxt = eig / nrm
        eig = A @ (At @ nxt)
        s = torch.dot(nxt, eig)
        sq = float(s)
        if float((eig - s * nxt).norm()) < 1e-4:
            break
    return math.sqrt(max(sq, 0.0))


class _Restarts:
    """The restart rule and the primal-weight controller of restarted Halpern PDHG."""

    def __init__(self, pw):
        self.pw = self.best_pw = pw
        self.best_gap = math.inf
        self.sum = self.last = 0.0
        self.initial = self.trial = math.inf
        self.inner = self.total = 0

    def due(self, fpe):
        yes = self.total == FREQ
        if self.total > FREQ:
            yes = (fpe <= 0.2 * self.initial or (fpe <= 0.5 * self.initial and fpe > self.trial)
                   or self.inner >= 0.36 * self.total)
        self.trial = fpe
        return yes

    def update(self, dp, dd, rel_p, rel_d):
        eps = 2.220446049250313e-16
        ratio = rel_d / max(rel_p, eps)
        if 1e-16 < dp < 1e12 and 1e-16 < dd < 1e12 and 1e-8 < ratio < 1e8:
            err = math.log(dd) - math.log(dp) - math.log(self.pw)
            self.sum = self.sum * 0.3 + err
            self.pw *= math.exp(0.99 * err + 0.01 * self.sum)
            self.last = err
        else:
            self.pw, self.sum, self.last = self.best_pw, 0.0, 0.0
        gap = abs(math.log10(ratio)) if ratio > 0.0 else math.inf
        if gap < self.best_gap:
            self.best_gap, self.best_pw = gap, self.pw
        self.inner, self.trial = 0, math.inf


def _clamp(v, lo, hi):
    return torch.minimum(torch.maximum(v, lo), hi)


def _project64(milp, target, windows):
    """The first projection of a fresh handle, in 64 bits."""
    dev = "cuda"
    s = _scale64(milp.A, np.zeros(len(milp.c)), milp.l, milp.u, _con_lb(milp), milp.b, False)
    A, At = s["A"], _transpose(s["A"])
    t64 = lambda v: torch.from_numpy(np.ascontiguousarray(v, dtype=np.float64)).to(dev)  # noqa: E731
    b, lb, ub, w = t64(s["cub"]), t64(s["lb"]), t64(s["ub"]), t64(_weights(milp, s["Dc"]))
    eq, ii = torch.from_numpy(np.asarray(milp.is_eq, bool)).to(dev), torch.from_numpy(_is_int(milp) != 0).to(dev)
    unscale, xt = t64(1.0 / s["Dr"]), t64(target / s["Dc"])
    wi = torch.where(ii, w, torch.zeros_like(w))
    step = 0.998 / math.sqrt(1.0 + _norm64(A, At) ** 2)
    rs = _Restarts(1.0)
    n, m = len(lb), len(b)
    cx, cy = torch.zeros(n, dtype=b.dtype, device=dev), torch.zeros(n, dtype=b.dtype, device=dev)
    cz = torch.zeros(m, dtype=b.dtype, device=dev)
    ix, iy, iz = cx, cy, cz
    b_norm = float((b * unscale).norm())
    d_den = 1.0 + float(wi.norm())
    restarted = False
    while rs.total < FREQ * windows:
        for k in range(1, FREQ + 1):
            kk = float(rs.inner + k)
            wt = kk / (kk + 1.0)
            tau, sig = step / rs.pw, step * rs.pw
            t = cx - tau * (At @ cz - cy)
            px = _clamp(t, lb, ub)
            rx = 2.0 * px - cx
            py = _clamp(cy + sig * (xt - rx), -wi, wi)
            ry = 2.0 * py - cy
            raw = cz + sig * (A @ rx - b)
            pz = torch.where(eq, raw, raw.clamp(min=0.0))
            rz = 2.0 * pz - cz
            cx, cy, cz = wt * rx + (1.0 - wt) * ix, wt * ry + (1.0 - wt) * iy, wt * rz + (1.0 - wt) * iz
            if k == FREQ or (k == 1 and restarted):
                dx, dy, dz = px - rx, py - ry, pz - rz
                mv = float(dx.square().sum()) * rs.pw + float(dy.square().sum() + dz.square().sum()) / rs.pw
                fpe = math.sqrt(max(mv + 2.0 * step * float(torch.dot(At @ dz - dy, dx)), 0.0))
                if k == 1:
                    rs.initial, restarted = fpe, False
        viol = A @ px - b
        viol = torch.where(eq, viol.abs(), viol.clamp(min=0.0)) * unscale
        rel_p = float(viol.norm()) / (1.0 + b_norm)
        rel_d = float((At @ pz - py - (px - t) / tau).norm()) / d_den
        rs.inner += FREQ
        rs.total += FREQ
        restarted = rs.due(fpe)
        if restarted:
            dd = math.sqrt(float((iy - py).square().sum() + (iz - pz).square().sum()))
            rs.update(float((ix - px).norm()), dd, rel_p, rel_d)
            cx, cy, cz = px, py, pz
            ix, iy, iz = px, py, pz
    return (px.cpu().numpy()) * s["Dc"]


def _root64(milp):
    dev = "cuda"
    s = _scale64(milp.A, milp.c, milp.l, milp.u, _con_lb(milp), milp.b, True)
    A, At = s["A"], _transpose(s["A"])
    t64 = lambda v: torch.from_numpy(np.ascontiguousarray(v, dtype=np.float64)).to(dev)  # noqa: E731
    c, lb, ub, lo, hi = (t64(s[k]) for k in ("c", "lb", "ub", "clb", "cub"))
    step = 0.998 / _norm64(A, At)
    fin = torch.where(torch.isfinite(lo) & (lo != hi), lo, torch.zeros_like(lo))
    b_norm = math.sqrt(float(fin.square().sum() + hi.square().sum()))
    c_norm = float(c.norm())
    lo0 = torch.where(lo.abs() < 1e19, lo, torch.zeros_like(lo))
    scale = s["bs"] * s["os"]
    rs = _Restarts(1.0)
    cx, cy = torch.zeros_like(c), torch.zeros_like(hi)
    ix, iy, restarted = cx, cy, False
    while True:
        for k in range(1, FREQ + 1):
            kk = float(rs.inner + k)
            wt = kk / (kk + 1.0)
            tau, sig = step / rs.pw, step * rs.pw
            t = cx - tau * (c - At @ cy)
            px = _clamp(t, lb, ub)
            rx = 2.0 * px - cx
            q = cy / sig - A @ rx
            py = (q - _clamp(q, -hi, -lo)) * sig
            ry = 2.0 * py - cy
            cx, cy = wt * rx + (1.0 - wt) * ix, wt * ry + (1.0 - wt) * iy
            if k == FREQ or (k == 1 and restarted):
                dx, dy = px - rx, py - ry
                mv = float(dx.square().sum()) * rs.pw + float(dy.square().sum()) / rs.pw
                fpe = math.sqrt(max(mv + 2.0 * step * float(torch.dot(At @ dy, dx)), 0.0))
                if k == 1:
                    rs.initial, restarted = fpe, False
        slack = (px - t) / tau
        Ax = A @ px
        rel_p = float((Ax - _clamp(Ax, lo, hi)).norm()) / s["bs"] / (1.0 + b_norm)
        rel_d = float((c - At @ py - slack).norm()) / s["os"] / (1.0 + c_norm)
        obj = float(torch.dot(c, px)) / scale
        dual = float(torch.dot(slack, px) + (py.clamp(min=0.0) * lo0 + py.clamp(max=0.0) * hi).sum()) / scale
        gap = abs(obj - dual) / (1.0 + abs(obj) + abs(dual))
        rs.inner += FREQ
        rs.total += FREQ
        if (rel_p <= ROOT_TOL and rel_d <= ROOT_TOL and gap <= ROOT_TOL) or rs.total >= 40_000:
            break
        restarted = rs.due(fpe)
        if restarted:
            rs.update(float((ix - px).norm()), float((iy - py).norm()), rel_p, rel_d)
            cx, cy, ix, iy = px, py, px, py
    return {"x": s["Dc"] * px.cpu().numpy() / s["bs"], "dual_slack": slack.cpu().numpy(),
            "iterations": rs.total, "optimal": rs.total < 40_000}


def exact(case, seed):
    models = _models(case, seed)
    if case["path"] == "root_lp":
        return _root64(models[0])
    if case["path"] == "scaling":
        mm = models[0]
        s = _scale64(mm.A, mm.c, mm.l, mm.u, _con_lb(mm), mm.b, True)
        return {"values": s["A"].values().cpu().numpy(), "c": s["c"], "var_ub": s["ub"],
                "con_ub": s["cub"], "D_r": s["Dr"], "D_c": s["Dc"], "bound_scale": float(s["bs"]),
                "objective_scale": float(s["os"])}
    xs = [_project64(mm, _targets(mm, seed * 64 + p)[0], case["windows"]) for p, mm in enumerate(models)]
    its = FREQ * case["windows"]
    if case["path"] == "projection":
        return {"x": xs[0], "iterations": its}
    return {"x": xs, "iterations": [its] * len(xs)}
