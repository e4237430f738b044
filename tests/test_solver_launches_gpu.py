"""Solver launches that run many iterations, at the sizes where their shape
changes: fewer rows than blocks, partly filled units, the last cluster and
the first grid size, more rows than the shared memories hold (the graph of
single iterations), and whole-GPU launches of two systems at a time.

Tolerances: the heads of the FP32-inner solve within 1e-8 of the FP64 CG
(the bar of tests/test_mixed_precision_gpu.py); runs of the same solve bit
for bit (the sums are added in a fixed order).
"""
import threading
import time

import numpy as np
import pytest

from ogs5_gb300 import mesh as M
from tests.helpers import rel_max_err, renumber

pytestmark = pytest.mark.gpu

MIXED_RTOL = 1e-8


def _mesh(kind, dims):
    m = M.structured_quad(*dims) if kind == "quad" else (
        M.structured_tet(*dims) if kind == "tet" else M.structured_hex(*dims))
    if kind == "renumbered":
        m, _ = renumber(m, 3)
    return m


def _system(gpu, m, seed=1, stream=None):
    rng = np.random.default_rng(seed)
    ek = np.exp(np.log(1e-5) + 0.7 * rng.standard_normal(m.n_elements))
    eqs = gpu.LinearEQS(gpu.GpuMesh(m), stream=stream)
    eqs.Initialize()
    eqs.GlobalAssembly(gpu.make_params(gpu.GROUNDWATER_FLOW, dt=3600.0, storage=1e-4), ek, np.zeros(m.n_nodes))
    lf, rf = m.face_nodes(0, 0), m.face_nodes(0, 1)
    eqs.SetKnownX(np.concatenate([lf, rf]), np.concatenate([np.full(len(lf), 10.0), np.zeros(len(rf))]),
                  gpu.DIRICHLET_SYMMETRIC)
    return eqs


def _solve(gpu, eqs, n, precision, tol=1e-10, method=None, precond=None):
    eqs.ConfigNumerics(gpu.LS_CG if method is None else method, gpu.PRECOND_JACOBI if precond is None else precond,
                       20000, tol, precision=precision, check_norm_rhs=False)
    x = np.zeros(n)
    it = eqs.Solver(x)
    assert eqs.stats()["status"] == gpu.OK and eqs.stats()["rel_residual"] < tol
    return x, it


SHAPES = [("hex", (2, 2, 2)), ("hex", (5, 3, 2)), ("hex", (24, 24, 25)), ("hex", (25, 25, 24)), ("hex", (60, 50, 41)),
          ("tet", (2, 2, 2)), ("tet", (24, 24, 25)), ("tet", (40, 33, 29)), ("renumbered", (6, 5, 4)),
          ("renumbered", (30, 28, 26)), ("quad", (7, 5)), ("quad", (127, 127)), ("quad", (200, 131))]


@pytest.mark.parametrize("kind,dims", SHAPES)
def test_fp32_refined_over_sizes(gpu, kind, dims):
    m = _mesh(kind, dims)
    eqs = _system(gpu, m)
    x64, it64 = _solve(gpu, eqs, m.n_nodes, gpu.PRECISION_FP64)
    x32, it32 = _solve(gpu, eqs, m.n_nodes, gpu.PRECISION_FP32_REFINED)
    again, _ = _solve(gpu, eqs, m.n_nodes, gpu.PRECISION_FP32_REFINED)
    assert rel_max_err(x32, x64) < MIXED_RTOL
    assert it32 <= 1.3 * it64 + 10
    assert np.array_equal(x32, again)


def test_fp32_refined_larger_than_the_shared_memories(gpu):
    m = M.structured_hex(180, 100, 98)  # 1.81 million rows
    eqs = _system(gpu, m)
    x64, _ = _solve(gpu, eqs, m.n_nodes, gpu.PRECISION_FP64)
    x32, _ = _solve(gpu, eqs, m.n_nodes, gpu.PRECISION_FP32_REFINED)
    assert rel_max_err(x32, x64) < MIXED_RTOL


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_two_threads_solve_at_once(gpu, precision):
    """Launches that fill the GPU, from two streams at a time: each result
    is the one of the system alone."""
    prec = gpu.PRECISION_FP64 if precision == "fp64" else gpu.PRECISION_FP32_REFINED
    meshes = [M.structured_hex(48, 40, 36), M.structured_tet(44, 40, 30)]
    systems = [_system(gpu, m, seed=q) for q, m in enumerate(meshes)]
    alone = [_solve(gpu, e, m.n_nodes, prec)[0] for e, m in zip(systems, meshes)]
    got = [[], []]

    def work(q):
        for _ in range(4):
            got[q].append(_solve(gpu, systems[q], meshes[q].n_nodes, prec)[0])

    threads = [threading.Thread(target=work, args=(q,)) for q in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for q in range(2):
        assert len(got[q]) == 4
        for x in got[q]:
            assert np.array_equal(x, alone[q])


@pytest.mark.parametrize("kind,dims,precision,method", [("quad", (100, 100), "fp64", "cg"),
                                                        ("quad", (100, 100), "fp64", "bicgstab"),
                                                        ("quad", (100, 100), "fp32", "cg"),
                                                        ("hex", (27, 27, 27), "fp32", "cg"),
                                                        ("hex", (17, 17, 17), "fp64", "bicgstab"),
                                                        ("hex", (20, 20, 20), "fp64", "cg"),
                                                        ("tet", (25, 24, 24), "fp64", "bicgstab")])
def test_solves_of_many_threads_run_side_by_side(gpu, kind, dims, precision, method):
    """Eight threads' solves of systems that need a part of the SMs take far
    less than eight times one's (0.95 of it where they take turns, 0.1 to 0.4
    where they do not)."""
    prec = gpu.PRECISION_FP64 if precision == "fp64" else gpu.PRECISION_FP32_REFINED
    meth = gpu.LS_CG if method == "cg" else gpu.LS_BICGSTAB
    m, n, reps = _mesh(kind, dims), 8, 6
    systems = [_system(gpu, m, seed=3) for _ in range(n)]
    alone = [_solve(gpu, e, m.n_nodes, prec, method=meth)[0] for e in systems]
    differ = []

    def work(q):
        for _ in range(reps):
            x = np.zeros(m.n_nodes)
            systems[q].Solver(x)
            if not np.array_equal(x, alone[q]):
                differ.append(q)

    best = {}
    for _ in range(3):
        for count in (1, n):
            threads = [threading.Thread(target=work, args=(q,)) for q in range(count)]
            t0 = time.perf_counter()
            for t in threads:
                t.start()
            for t in threads:
                t.join()
            best[count] = min(best.get(count, 1e9), time.perf_counter() - t0)
    assert not differ
    assert best[n] < 0.7 * n * best[1], best


@pytest.mark.parametrize("precision,method", [("fp32", "cg"), ("fp64", "cg"), ("fp64", "bicgstab")])
def test_threads_with_systems_of_many_sizes(gpu, precision, method):
    """Launches with different amounts of shared memory, set up and started
    by six threads at a time: none changes what another may ask for."""
    prec = gpu.PRECISION_FP64 if precision == "fp64" else gpu.PRECISION_FP32_REFINED
    meth = gpu.LS_CG if method == "cg" else gpu.LS_BICGSTAB
    meshes = [_mesh(k, d) for k, d in (("quad", (60, 40)), ("hex", (14, 10, 8)), ("tet", (8, 6, 5)), ("quad", (60, 40)),
                                       ("hex", (20, 18, 16)), ("tet", (16, 12, 10)))]
    systems = [_system(gpu, m, seed=q) for q, m in enumerate(meshes)]
    alone = [_solve(gpu, e, m.n_nodes, prec, method=meth)[0] for e, m in zip(systems, meshes)]
    got = [[] for _ in meshes]

    def work(q):
        for _ in range(20):
            got[q].append(_solve(gpu, systems[q], meshes[q].n_nodes, prec, method=meth)[0])

    threads = [threading.Thread(target=work, args=(q,)) for q in range(len(meshes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for q in range(len(meshes)):
        assert len(got[q]) == 20
        for x in got[q]:
            assert np.array_equal(x, alone[q])


# FP64: launches of many iterations against the graph of single steps (which
# the timing samples of ogs_gpu_profile keep): the same recurrences with the
# sums grouped differently, so heads solved to 1e-13 agree within 1e-10 (the
# bar of the parity tests) and CG's iteration counts within 2.  BiCGStab's
# are not compared: rounding alone moves them (362 to 435 for the graph form
# over ten assemblies of the 800 x 610 quads, whose atomics land in another
# order each time).
def _both_forms(gpu, eqs, n, method, precond, tol=1e-13, max_iter=20000, x0=None):
    out = []
    for graph in (False, True):
        eqs.ConfigNumerics(method, precond, max_iter, tol, check_norm_rhs=False)
        eqs.profile(graph)
        x = np.zeros(n) if x0 is None else x0.copy()
        it = eqs.Solver(x, allow_fail=True)
        out.append((x, it, eqs.stats()))
    eqs.profile(False)
    return out


@pytest.mark.parametrize("kind,dims", SHAPES + [("hex", (12, 11, 10)), ("quad", (800, 610))])
@pytest.mark.parametrize("method", ["cg", "bicgstab"])
@pytest.mark.parametrize("precond", ["jacobi", "none"])
def test_fp64_over_sizes(gpu, kind, dims, method, precond):
    m = _mesh(kind, dims)
    eqs = _system(gpu, m)
    (x, it, st), (xg, itg, stg) = _both_forms(gpu, eqs, m.n_nodes, gpu.LS_CG if method == "cg" else gpu.LS_BICGSTAB,
                                              gpu.PRECOND_JACOBI if precond == "jacobi" else gpu.PRECOND_NONE)
    assert st["status"] == stg["status"] == gpu.OK and st["rel_residual"] < 1e-13
    assert rel_max_err(x, xg) < 1e-10
    if method == "cg":
        assert abs(it - itg) <= 2


@pytest.mark.parametrize("method", ["cg", "bicgstab"])
def test_fp64_vectors_partly_in_global_memory(gpu, method):
    m = M.structured_hex(180, 100, 98)  # 1.81 million rows
    eqs = _system(gpu, m)
    (x, it, st), (xg, itg, stg) = _both_forms(gpu, eqs, m.n_nodes, gpu.LS_CG if method == "cg" else gpu.LS_BICGSTAB,
                                              gpu.PRECOND_JACOBI)
    assert st["status"] == stg["status"] == gpu.OK
    assert rel_max_err(x, xg) < 1e-10


@pytest.mark.parametrize("kind,dims,method,many", [
    ("quad", (1599, 1599), "cg", True), ("quad", (1799, 1749), "cg", False), ("quad", (1299, 1299), "bicgstab", True),
    ("quad", (1499, 1499), "bicgstab", False), ("tet", (91, 91, 91), "cg", True), ("tet", (99, 99, 99), "cg", False),
    ("tet", (108, 108, 108), "bicgstab", True), ("tet", (119, 119, 119), "bicgstab", False)])
def test_fp64_large_systems_take_the_faster_form(gpu, kind, dims, method, many):
    """On both sides of the row limits: launches of many iterations below,
    single steps above, the same heads."""
    m = _mesh(kind, dims)
    eqs = _system(gpu, m)
    meth = gpu.LS_CG if method == "cg" else gpu.LS_BICGSTAB
    eqs.ConfigNumerics(meth, gpu.PRECOND_JACOBI, 40, 1e-13, check_norm_rhs=False)
    x = np.zeros(m.n_nodes)
    gpu.kernel_launches(reset=True)
    eqs.Solver(x, allow_fail=True)
    launches = gpu.kernel_launches()
    assert eqs.stats()["iterations"] == 40
    assert (launches < 20) == many, launches
    (x, _, st), (xg, _, stg) = _both_forms(gpu, eqs, m.n_nodes, meth, gpu.PRECOND_JACOBI)
    assert st["status"] == stg["status"] == gpu.OK
    assert rel_max_err(x, xg) < 1e-10


@pytest.mark.parametrize("kind,dims", [("hex", (80, 80, 80)), ("tet", (90, 90, 90))])
def test_fp64_scattered_columns_keep_their_cache(gpu, kind, dims):
    """Nodes in random order: the vectors in shared memory leave the gathers
    of the products enough L1.  The launches of many iterations took 1.7 to
    1.9 times as long as single steps where they did not, 0.93 times where
    they do (BiCGStab, which has the most vectors)."""
    m, _ = renumber(_mesh(kind, dims), 3)
    eqs = _system(gpu, m)
    ms = {}
    for graph in (False, True):
        eqs.ConfigNumerics(gpu.LS_BICGSTAB, gpu.PRECOND_JACOBI, 192, 1e-30, check_norm_rhs=False)
        eqs.profile(graph)
        for _ in range(4):
            eqs.Solver(np.zeros(m.n_nodes), allow_fail=True)
            ms[graph] = min(ms.get(graph, 1e9), eqs.stats()["solve_ms"])
    eqs.profile(False)
    assert ms[False] < 1.5 * ms[True], ms
    (x, _, st), (xg, _, stg) = _both_forms(gpu, eqs, m.n_nodes, gpu.LS_BICGSTAB, gpu.PRECOND_JACOBI)
    assert st["status"] == stg["status"] == gpu.OK
    assert rel_max_err(x, xg) < 1e-10


@pytest.mark.parametrize("dims,many", [((80, 80, 77), True), ((88, 88, 88), False)])  # 59 and 81 MB
def test_fp32_large_sell_operators_take_the_faster_form(gpu, dims, many):
    """Tets in random order: launches of many FP32 iterations while the
    SELL-32 operator stays in L2, single iterations above, the same heads as
    the FP64 CG's."""
    m, _ = renumber(M.structured_tet(*dims), 3)
    eqs = _system(gpu, m)
    gpu.kernel_launches(reset=True)
    x, it = _solve(gpu, eqs, m.n_nodes, gpu.PRECISION_FP32_REFINED)
    launches = gpu.kernel_launches()
    assert (launches < it) == many, (launches, it)
    x64, _ = _solve(gpu, eqs, m.n_nodes, gpu.PRECISION_FP64)
    assert rel_max_err(x, x64) < MIXED_RTOL


@pytest.mark.parametrize("dims", [(6, 5, 4), (28, 27, 26)])
@pytest.mark.parametrize("method", ["cg", "bicgstab"])
def test_fp64_ends_as_the_graph_does(gpu, dims, method):
    """Iteration limits, non-finite and zero right-hand sides, and heads near
    the limits of double's range (r . r underflows)."""
    m = M.structured_hex(*dims)
    eqs = _system(gpu, m)
    kind = gpu.LS_CG if method == "cg" else gpu.LS_BICGSTAB
    for limit in (0, 1, 7):
        (x, it, st), (xg, itg, stg) = _both_forms(gpu, eqs, m.n_nodes, kind, gpu.PRECOND_JACOBI, max_iter=limit)
        assert (it, st["status"]) == (itg, stg["status"]) == (limit, gpu.NOT_CONVERGED)
        assert rel_max_err(x, xg) < 1e-10
    x0 = np.zeros(m.n_nodes)
    x0[m.n_nodes // 2 - m.n_nodes // 2 % (dims[0] + 1) + 1] = np.nan  # beside the x = 0 face, not on it
    for (x, it, st) in _both_forms(gpu, eqs, m.n_nodes, kind, gpu.PRECOND_JACOBI, x0=x0):
        assert st["status"] == gpu.NONFINITE
    for head in (0.0, 1e-160, 1e-152, 1e150):
        e = gpu.LinearEQS(eqs.gmesh)
        e.Initialize()
        ek = np.full(m.n_elements, 1.0)
        e.GlobalAssembly(gpu.make_params(gpu.GROUNDWATER_FLOW, dt=1.0, storage=1.0), ek, np.zeros(m.n_nodes))
        lf = m.face_nodes(0, 0)
        e.SetKnownX(lf, np.full(len(lf), head), gpu.DIRICHLET_SYMMETRIC)
        (x, it, st), (xg, itg, stg) = _both_forms(gpu, e, m.n_nodes, kind, gpu.PRECOND_JACOBI, tol=1e-6)
        assert st["status"] == stg["status"] and abs(it - itg) <= 1
        assert np.abs(x - xg).max() <= 1e-6 * np.abs(xg).max()
