"""The resident window (resident_steps.cuh): a window's steps in one cooperative launch
with the whole handle in shared memory.

CPU: tests/native/resident_check.cpp walks the layout with the kernel's index arithmetic.
GPU: the steps against the per-step launches (PDFP_RESIDENT=0) and the FP64 oracle, and a
batch's members against their single handles, bit for bit."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
import scipy.sparse as sp

from pdfp_b200 import synthetic
from pdfp_b200.params import SolverParameters
from test_layout import rand_csr

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
OUT = os.path.join(ROOT, "_build", "libresident_check.so")


@pytest.fixture(scope="module")
def checker():
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    srcs = [os.path.join(HERE, "native", "resident_check.cpp"),
            os.path.join(ROOT, "pdfp_b200", "csrc", "layout.cpp")]
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-o", OUT] + srcs, check=True)
    lib = C.CDLL(OUT)
    lib.resident_check.restype = C.c_int
    return lib


def check(lib, mats, eqs, n_blocks):
    K = len(mats)
    keep = []
    ms, ns = (C.c_int32 * K)(), (C.c_int32 * K)()
    rps, cis = (C.POINTER(C.c_int32) * K)(), (C.POINTER(C.c_int32) * K)()
    vs, es = (C.POINTER(C.c_double) * K)(), (C.POINTER(C.c_uint8) * K)()
    for p, (A, e) in enumerate(zip(mats, eqs)):
        A = sp.csr_matrix(A)
        A.sort_indices()
        rp = np.ascontiguousarray(A.indptr, dtype=np.int32)
        ci = np.ascontiguousarray(A.indices if A.nnz else np.zeros(1), dtype=np.int32)
        v = np.ascontiguousarray(A.data if A.nnz else np.zeros(1), dtype=np.float64)
        ee = np.ascontiguousarray(e, dtype=np.uint8) if len(e) else np.zeros(1, np.uint8)
        keep += [rp, ci, v, ee]
        ms[p], ns[p] = A.shape
        rps[p] = rp.ctypes.data_as(C.POINTER(C.c_int32))
        cis[p] = ci.ctypes.data_as(C.POINTER(C.c_int32))
        vs[p] = v.ctypes.data_as(C.POINTER(C.c_double))
        es[p] = ee.ctypes.data_as(C.POINTER(C.c_uint8))
    stats = (C.c_int64 * 2)()
    return lib.resident_check(K, ms, ns, rps, cis, vs, es, n_blocks, stats), list(stats)


@pytest.mark.parametrize("n_blocks", [1, 7, 148])
def test_layout(checker, n_blocks):
    rng = np.random.default_rng(5)
    one = [rand_csr(rng, 300, 500, 0.02)]
    long = [rand_csr(rng, 60, 9000, 0.0005, long_rows=4, long_len=7001)]
    # row lengths at the edges of the lanes' rule and of a long row's pieces
    edges = [0, 1, 31, 32, 33, 64, 65, 128, 129, 256, 257, 512, 513, 1023, 1024, 1025, 2048, 2049]
    E = sp.lil_matrix((len(edges), 2100))
    for i, k in enumerate(edges):
        E[i, rng.choice(2100, size=k, replace=False)] = 1.0
    batch = [rand_csr(rng, 80, 60, 0.05), sp.csr_matrix((0, 5)), sp.csr_matrix((7, 0)),
             sp.csr_matrix((4, 6)), rand_csr(rng, 1000, 30, 0.3), sp.csr_matrix(E)]
    for mats, has_long in ((one, False), (long, True), ([sp.csr_matrix(E)], True), (batch, True)):
        rc, stats = check(checker, mats, [rng.random(A.shape[0]) < 0.5 for A in mats], n_blocks)
        assert rc == 0
        assert (stats[1] > 0) == has_long


def _state(probs, precision, monkeypatch, resident):
    from pdfp_b200 import gpu
    monkeypatch.setenv("PDFP_RESIDENT", resident)
    s = gpu.PDFPState(*probs, precision=precision)
    form = gpu.C.c_int32()
    gpu.L.check(gpu.L.lib().pdfp_get_window_form(s._h, gpu.C.byref(form)))
    assert form.value == (4 if resident == "1" else 0)
    return s


def _models():
    """Ragged general model (no size a multiple of a warp or of the SM count), equality
    rows among them; Zipf rows long enough for several pieces; binary covering."""
    g, _, xt = synthetic.general_integer(3, m=1501, n=4013, m_eq=377, mean_row=9.0)
    z, _ = synthetic.zipf_lp(2, m=3001, n=6007, nnz=60_001)
    rng = np.random.default_rng(4)
    zt = np.zeros(6007)
    zt[z.int_idx] = np.round(rng.random(len(z.int_idx)))
    return [("general", g, xt), ("zipf", z, zt)]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("which", [0, 1])
def test_steps_match_per_step_launches_and_oracle(oracle, monkeypatch, precision, which):
    """One and three windows.  FP64: both forms stay within 1e-10 of the oracle after 200
    and 600 steps (each step adds rounding of about 1e-16 relative and does not expand it);
    mixed: within 2e-4 of it, FP32 rounding grown by the same argument."""
    _, milp, xt = _models()[which]
    sc, is_eq, is_int, w = oracle.projector_inputs(milp)
    probs = (sc.A, sc.con_ub, is_eq, is_int, sc.var_lb, sc.var_ub, w)
    for windows in (1, 3):
        prm = SolverParameters(eps_optimal_relative=1e-9, eps_feasible_relative=1e-9,
                               iteration_limit=200 * windows)
        o = oracle.OracleSolvers.PDFPState(*probs)
        o.set_target(xt / sc.D_c)
        o.solve(prm, 1.0)
        tol = 1e-10 if precision == "fp64" else 2e-4
        for resident in ("1", "0"):
            s = _state(probs, precision, monkeypatch, resident)
            s.set_target(xt / sc.D_c)
            s.solve(prm, 1.0)
            assert s.total_count == 200 * windows
            for name in ("pdhg_x", "pdhg_y", "pdhg_z", "current_x", "current_y", "current_z", "dual_slack"):
                a, b = s.get(name), o.get(name)
                assert np.linalg.norm(a - b) <= tol * max(1.0, np.linalg.norm(b)), (resident, windows, name)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batch_members_equal_single_handles(oracle, monkeypatch, precision):
    """Members that stop at different windows, one of them with long rows: with the same
    kernels for the windows' first steps (PDFP_AUTOTUNE=0), the steps of the single
    handles bit for bit in the resident part; whole solves to 1e-12 / 1e-5."""
    from pdfp_b200 import gpu
    monkeypatch.setenv("PDFP_RESIDENT", "1")
    monkeypatch.setenv("PDFP_AUTOTUNE", "0")
    models = synthetic.covering_packing_batch(seed=7, k=4, n_min=3000, n_max=9000)
    models.append(_models()[1][1])
    rng = np.random.default_rng(21)
    probs, targets = [], []
    for m in models:
        sc, is_eq, is_int, w = oracle.projector_inputs(m)
        probs.append((sc.A, sc.con_ub, is_eq, is_int, sc.var_lb, sc.var_ub, w))
        targets.append(np.round(rng.random(len(m.c))) / sc.D_c)
    prm = [SolverParameters(eps_optimal_relative=1e-9, eps_feasible_relative=1e-9,
                            iteration_limit=200 * (1 + p % 3)) for p in range(len(models))]
    b = gpu.PDFPBatch(probs, precision=precision)
    for p, xt in enumerate(targets):
        b.set_target(p, xt)
    b.solve(prm, 1.0)
    tol = 1e-12 if precision == "fp64" else 1e-5
    for p, pr in enumerate(probs):
        s = gpu.PDFPState(*pr, precision=precision)
        s.set_target(targets[p])
        s.solve(prm[p], 1.0)
        assert s.total_count == b.results[p]["total_count"] == 200 * (1 + p % 3)
        x, y = s.pdhg_x, b.get(p, "pdhg_x")
        assert np.linalg.norm(x - y) <= tol * max(1.0, np.linalg.norm(x)), p


# ---- small members: whole windows in a thread-block cluster (cluster_windows.cuh) -------


def _small_models():
    """One, two and several blocks per member; sizes at the edges of a warp's 32 rows; dense
    rows shared by several lanes; rows and columns without entries."""
    out = [synthetic.covering_p0201_like(1), synthetic.markshare_like(2)]
    for seed, m, n, mean in ((3, 31, 33, 4.0), (4, 64, 97, 3.0), (5, 211, 305, 7.5), (6, 601, 1503, 25.0)):
        out.append(synthetic.general_integer(seed, m=m, n=n, m_eq=m // 4, mean_row=mean)[0])
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_small_members_match_oracle_and_their_batch(oracle, precision):
    """One and three windows of each member: against the oracle (the bounds of the resident
    steps' test), and in one batch handle, whose cluster size is another: bit for bit."""
    from pdfp_b200 import gpu
    tol = 1e-10 if precision == "fp64" else 2e-4
    probs, targets, singles = [], [], []
    for k, m in enumerate(_small_models()):
        sc, is_eq, is_int, w = oracle.projector_inputs(m)
        probs.append((sc.A, sc.con_ub, is_eq, is_int, sc.var_lb, sc.var_ub, w))
        rng = np.random.default_rng(30 + k)
        xt = np.zeros(len(m.c))
        xt[m.int_idx] = np.round(m.l[m.int_idx] + rng.random(len(m.int_idx)) * (m.u - m.l)[m.int_idx])
        targets.append(xt / sc.D_c)
    for windows in (1, 3):
        prm = SolverParameters(eps_optimal_relative=1e-9, eps_feasible_relative=1e-9,
                               iteration_limit=200 * windows)
        batch = gpu.PDFPBatch(probs, precision=precision)
        for p, xt in enumerate(targets):
            batch.set_target(p, xt)
        batch.solve(prm, 1.0)
        for p, pr in enumerate(probs):
            s, o = gpu.PDFPState(*pr, precision=precision), oracle.OracleSolvers.PDFPState(*pr)
            form = gpu.C.c_int32()
            gpu.L.check(gpu.L.lib().pdfp_get_window_form(s._h, gpu.C.byref(form)))
            assert form.value == 3
            for h in (s, o):
                h.set_target(targets[p])
                h.solve(prm, 1.0)
            assert s.total_count == batch.results[p]["total_count"]
            for name in ("pdhg_x", "pdhg_y", "pdhg_z", "current_x", "current_y", "current_z", "dual_slack"):
                a, b = s.get(name), o.get(name)
                if s.total_count == 200 * windows:
                    assert np.linalg.norm(a - b) <= tol * max(1.0, np.linalg.norm(b)), (p, windows, name)
                assert np.array_equal(a, batch.get(p, name)), (p, windows, name)


@pytest.mark.gpu
def test_a_row_too_long_for_a_cluster_takes_the_resident_steps(oracle):
    """A row of more than 512 nonzeros, and a member of as many rows as a cluster has no
    warps for: the handle runs its windows resident on the chip instead."""
    from pdfp_b200 import gpu
    rng = np.random.default_rng(8)
    A = sp.random(40, 700, density=0.01, random_state=rng, format="lil")
    A[7, :] = rng.uniform(-1.0, 1.0, size=700)
    A = sp.csr_matrix(A)
    for mat in (A, sp.csr_matrix(sp.random(1900, 2100, density=0.004, random_state=rng))):
        m, n = mat.shape
        b = mat @ rng.random(n) + 0.5
        pr = (mat, b, np.zeros(m, np.uint8), np.ones(n, np.uint8), np.zeros(n), np.ones(n), np.ones(n))
        s, o = gpu.PDFPState(*pr), oracle.OracleSolvers.PDFPState(*pr)
        prm = SolverParameters(eps_optimal_relative=1e-9, eps_feasible_relative=1e-9, iteration_limit=400)
        xt = np.round(rng.random(n))
        for h in (s, o):
            h.set_target(xt)
            h.solve(prm, 1.0)
        assert s.total_count == o.total_count
        assert np.linalg.norm(s.pdhg_x - o.pdhg_x) <= 1e-10 * max(1.0, np.linalg.norm(o.pdhg_x))


@pytest.mark.gpu
def test_long_rows_of_a_mixed_handle_are_summed_in_fp64(oracle, monkeypatch):
    """One row of five pieces over columns fixed at 1: each lane's first entry is 1 and its
    31 others 0.9 * 2^-24, which FP32 additions to 1 drop one by one (together 2.7e-4 of the
    row's violation, all of it) and FP64 ones keep.  z, which grows by sigma times the
    violation in every step, within 5% of the oracle's; products and x_bar carry at most
    160 * 2 * 2^-24 = 1.9e-5 of rounding, 7% of the violation and of either sign."""
    from pdfp_b200 import gpu
    monkeypatch.setenv("PDFP_MIXED_MIN_NNZ", "0")
    n = 5120
    a = np.where(np.arange(n) % 1024 < 32, 1.0, 0.9 * 2.0 ** -24)
    one = np.ones(n)
    pr = (sp.csr_matrix(a[None, :]), np.array([160.0]), np.ones(1, np.uint8), np.zeros(n, np.uint8), one, one, one)
    o = oracle.OracleSolvers.PDFPState(*pr)
    prm = SolverParameters(eps_optimal_relative=1e-6, eps_feasible_relative=1e-6, iteration_limit=200)
    s = _state(pr, "mixed", monkeypatch, "1")
    for h in (s, o):
        h.set_target(one)
        h.set_x(one)
        h.solve(prm, 1.0)
    z, zo = s.get("pdhg_z")[0], o.get("pdhg_z")[0]
    assert zo > 0.0 and abs(z - zo) <= 0.05 * zo


def _wide(seed, m, n, row_len):
    """Few rows of row_len nonzeros over binary columns, one of them an equality."""
    rng = np.random.default_rng(seed)
    A = sp.lil_matrix((m, n))
    for i in range(m):
        A[i, np.sort(rng.choice(n, size=row_len, replace=False))] = rng.uniform(0.5, 2.0, size=row_len)
    A = sp.csr_matrix(A)
    A.sort_indices()
    b = 0.5 * (A @ np.ones(n))
    eq = np.zeros(m, np.uint8)
    eq[0] = 1
    sc = 1.0 / np.sqrt(row_len)
    return (A * sc, b * sc, eq, np.ones(n, np.uint8), np.zeros(n), np.ones(n), np.ones(n)), np.round(rng.random(n))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("m,n,row_len,window_form", [(3, 520, 512, 3), (3, 520, 513, 3), (6, 606, 601, 3),
                                                     (5, 1300, 1025, 3), (3, 3500, 3300, 3), (4, 4092, 4000, 4)])
def test_wide_rows_run_in_a_cluster(oracle, monkeypatch, precision, m, n, row_len, window_form):
    """A small member with rows of any length runs its windows in a cluster (lanes deeper than
    their usual 16 entries), unless it has more slices (128 of 32 columns and 4 rows) than
    eight blocks have warps; to the bounds of the resident steps' test: 1e-10 of the oracle,
    2e-4 in FP32."""
    from pdfp_b200 import gpu
    monkeypatch.setenv("PDFP_MIXED_MIN_NNZ", "0")
    pr, xt = _wide(9, m, n, row_len)
    tol = 1e-10 if precision == "fp64" else 2e-4
    for windows in (1, 3):
        prm = SolverParameters(eps_optimal_relative=1e-6, eps_feasible_relative=1e-6, iteration_limit=200 * windows)
        s, o = gpu.PDFPState(*pr, precision=precision), oracle.OracleSolvers.PDFPState(*pr)
        form = gpu.C.c_int32()
        gpu.L.check(gpu.L.lib().pdfp_get_window_form(s._h, gpu.C.byref(form)))
        assert form.value == window_form
        for h in (s, o):
            h.set_target(xt)
            h.solve(prm, 1.0)
        assert s.total_count == o.total_count
        for name in ("pdhg_x", "pdhg_y", "pdhg_z", "current_x", "current_y", "current_z"):
            a, b = s.get(name), o.get(name)
            assert np.linalg.norm(a - b) <= tol * max(1.0, np.linalg.norm(b)), (windows, name)


@pytest.mark.gpu
def test_members_of_several_sizes_in_clusters_of_their_own(oracle):
    """400 members of one block each beside one of seven: the device time of the batch is at
    most twice that of its parts one after the other (a cluster of seven blocks for every
    member takes eight times the part of the 400), and the members' results are their own
    handles', bit for bit."""
    from pdfp_b200 import gpu
    small = synthetic.covering_p0201_like(1)
    big = synthetic.general_integer(6, m=601, n=1503, m_eq=150, mean_row=25.0)[0]
    inputs = {}
    for m in (small, big):
        sc, is_eq, is_int, w = oracle.projector_inputs(m)
        inputs[id(m)] = (sc.A, sc.con_ub, is_eq, is_int, sc.var_lb, sc.var_ub, w)
    prm = SolverParameters(eps_optimal_relative=1e-9, eps_feasible_relative=1e-9, iteration_limit=400)

    def solved(models):
        b = gpu.PDFPBatch([inputs[id(m)] for m in models], precision="fp64")
        for _ in range(2):  # the second solve is timed
            for p, m in enumerate(models):
                rng = np.random.default_rng(p % 5)
                b.set_target(p, np.round(rng.random(len(m.c))))
            b.solve(prm, 1.0)
        return b

    many = [small] * 400
    both = solved(many[:200] + [big] + many[200:])
    parts = [solved(many), solved([big])]
    assert both.results[0]["device_ms"] <= 2.0 * sum(b.results[0]["device_ms"] for b in parts)
    for p in (0, 3, 199, 200, 201, 400):
        m = big if p == 200 else small
        s = gpu.PDFPState(*inputs[id(m)], precision="fp64")
        for _ in range(2):
            s.set_target(np.round(np.random.default_rng(p % 5).random(len(m.c))))
            s.solve(prm, 1.0)
        for name in ("pdhg_x", "pdhg_z", "current_y"):
            assert np.array_equal(s.get(name), both.get(p, name)), (p, name)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_the_first_solve_pays_for_the_layout(oracle, monkeypatch, precision):
    """The first projection of a new handle, which lays the handle out for the resident window:
    no slower than the same one in per-step launches (best of three handles each), although
    it runs one window only."""
    import time
    milp, _, xt = synthetic.general_integer(1, m=24000, n=60000, m_eq=6000)
    sc, is_eq, is_int, w = oracle.projector_inputs(milp)
    probs = (sc.A, sc.con_ub, is_eq, is_int, sc.var_lb, sc.var_ub, w)
    prm = SolverParameters(eps_optimal_relative=1e-9, eps_feasible_relative=1e-9, iteration_limit=200)
    best = {}
    for resident in ("0", "1") * 4:  # the first of each loads the kernels
        s = _state(probs, precision, monkeypatch, resident)
        s.set_target(xt / sc.D_c)
        t = time.perf_counter()
        s.solve(prm, 1.0)
        best.setdefault(resident, []).append(time.perf_counter() - t)
    assert min(best["1"][1:]) <= min(best["0"][1:])


@pytest.mark.gpu
def test_asking_for_the_window_form_leaves_the_device_alone():
    """pdfp_get_window_form on a handle that has not solved: the answer is 4, and no device
    memory goes to it (a process without the library's memory pool, which would hide it)."""
    import sys
    code = """
import numpy as np, torch
from pdfp_b200 import gpu, synthetic
from oracle import oracle as O
milp = synthetic.general_integer(1)[0]
sc, is_eq, is_int, w = O.projector_inputs(milp)
s = gpu.PDFPState(sc.A, sc.con_ub, is_eq, is_int, sc.var_lb, sc.var_ub, w)
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
form = gpu.C.c_int32()
gpu.L.check(gpu.L.lib().pdfp_get_window_form(s._h, gpu.C.byref(form)))
assert form.value == 4
assert torch.cuda.mem_get_info()[0] == free
"""
    env = dict(os.environ, PDFP_POOL="0", PDFP_AUTOTUNE="0")
    for name in ("PDFP_RESIDENT", "PDFP_STEP_ENGINE", "PDFP_TUNING"):
        env.pop(name, None)
    subprocess.run([sys.executable, "-c", code], check=True, cwd=ROOT, env=env)


def _form(h):
    from pdfp_b200 import gpu
    form = gpu.C.c_int32()
    gpu.L.check(gpu.L.lib().pdfp_get_window_form(h._h, gpu.C.byref(form)))
    return form.value


@pytest.mark.gpu
@pytest.mark.parametrize("precision,m", [("fp64", 24000), ("mixed", 36000)])
def test_near_the_shared_memory_limit(oracle, monkeypatch, precision, m):
    """Handles that fill their blocks' shared memory (600k nonzeros in FP64, 900k mixed), after
    one and three windows: the bounds of the resident steps' test."""
    milp, _, xt = synthetic.general_integer(3, m=m, n=5 * m // 2, m_eq=m // 4)
    sc, is_eq, is_int, w = oracle.projector_inputs(milp)
    probs = (sc.A, sc.con_ub, is_eq, is_int, sc.var_lb, sc.var_ub, w)
    tol = 1e-10 if precision == "fp64" else 2e-4
    s, o = _state(probs, precision, monkeypatch, "1"), oracle.OracleSolvers.PDFPState(*probs)
    for windows in (1, 3):
        prm = SolverParameters(eps_optimal_relative=1e-9, eps_feasible_relative=1e-9, iteration_limit=200 * windows)
        for h in (s, o):
            h.set_target(xt / sc.D_c)
            h.solve(prm, 1.0)
        assert s.total_count == 200 * windows
        for name in ("pdhg_x", "pdhg_z", "current_y"):
            a, b = s.get(name), o.get(name)
            assert np.linalg.norm(a - b) <= tol * max(1.0, np.linalg.norm(b)), (windows, name)


@pytest.mark.gpu
def test_two_resident_handles_in_two_threads(oracle, monkeypatch):
    """Two handles that each take the whole GPU, solved at the same time from two threads on
    their own streams: the results of two others solved one after the other, bit for bit."""
    import threading
    monkeypatch.setenv("PDFP_AUTOTUNE", "0")
    prm = SolverParameters(eps_optimal_relative=1e-9, eps_feasible_relative=1e-9, iteration_limit=1000)
    inputs = []
    for _, milp, xt in _models():
        sc, is_eq, is_int, w = oracle.projector_inputs(milp)
        inputs.append(((sc.A, sc.con_ub, is_eq, is_int, sc.var_lb, sc.var_ub, w), xt / sc.D_c))

    def solve(s, xt, out):
        for _ in range(3):  # each from the iterates of the one before
            s.set_target(xt)
            s.solve(prm, 1.0)
            out.append([s.total_count] + [s.get(name) for name in ("pdhg_x", "current_y", "current_z")])

    results = []
    for together in (False, True):
        work = [(_state(pr, "fp64", monkeypatch, "1"), xt, []) for pr, xt in inputs]
        threads = [threading.Thread(target=solve, args=a) for a in work]
        for t in threads:
            t.start()
            if not together:
                t.join()
        for t in threads:
            t.join()
        results.append([out for _, _, out in work])
    for one, two in zip(*results):
        assert len(one) == len(two) == 3
        for a, b in zip(one, two):
            assert a[0] == b[0] == 1000
            for x, y in zip(a[1:], b[1:]):
                assert np.array_equal(x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_window_of_a_batch_member_equals_its_own_handles(oracle, monkeypatch, precision):
    """One window, before any evaluation can change a step size: the members' iterates are their
    single handles' bit for bit, with rows of one lane, of several and in pieces -- of the
    members whose step size is their single handle's: the norm estimate's last bit is not
    always the same in a batch, whose passes add partial sums of other tiles."""
    from pdfp_b200 import gpu
    monkeypatch.setenv("PDFP_RESIDENT", "1")
    monkeypatch.setenv("PDFP_AUTOTUNE", "0")
    monkeypatch.setenv("PDFP_MIXED_MIN_NNZ", "0")
    models = synthetic.covering_packing_batch(seed=7, k=3, n_min=3000, n_max=9000)
    models += [_models()[0][1], _models()[1][1]]
    assert np.diff(models[-1].A.tocsr().indptr).max() > 1024
    rng = np.random.default_rng(22)
    prm = SolverParameters(eps_optimal_relative=1e-6, eps_feasible_relative=1e-6, iteration_limit=200)
    probs, targets = [], []
    for m in models:
        sc, is_eq, is_int, w = oracle.projector_inputs(m)
        probs.append((sc.A, sc.con_ub, is_eq, is_int, sc.var_lb, sc.var_ub, w))
        targets.append(np.round(rng.random(len(m.c))) / sc.D_c)
    b = gpu.PDFPBatch(probs, precision=precision)
    assert _form(b) == 4
    for p, xt in enumerate(targets):
        b.set_target(p, xt)
    b.solve(prm, 1.0)
    compared = []
    for p, pr in enumerate(probs):
        s = gpu.PDFPState(*pr, precision=precision)
        assert _form(s) == 4
        s.set_target(targets[p])
        s.solve(prm, 1.0)
        if s.last["step_size"] != b.results[p]["step_size"]:
            continue
        compared.append(p)
        for name in ("pdhg_x", "pdhg_y", "pdhg_z"):
            assert np.array_equal(s.get(name), b.get(p, name)), (p, name)
    assert len(compared) >= 3 and len(models) - 1 in compared  # the last one has the long rows
