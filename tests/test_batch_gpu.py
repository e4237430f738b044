"""Monte-Carlo batch (ogs_gpu_batch_*): one persistent launch assembles and
solves many steady flow realisations of different sizes.

Bar: every realisation's heads within 1e-8 relative of the plain FP64 GPU
path (GpuMesh + LinearEQS: element assembly, symmetric Dirichlet, FP64
Jacobi-CG) on the same field, and the batch's own FP64 residual below its
tolerance.
"""
import time

import numpy as np
import pytest

from ogs5_gb300 import fields
from ogs5_gb300 import mesh as M
from tests.helpers import rel_max_err

pytestmark = pytest.mark.gpu

BATCH_RTOL = 1e-8


def _realisations(sizes, seed=0, var=1.0):
    rng = np.random.default_rng(seed)
    out = []
    for q, (nx, ny, nz) in enumerate(sizes):
        ek = fields.lognormal_k((nx - 1, ny - 1, nz - 1), np.log(1e-5), var,
                                float(rng.uniform(2, 4)), seed=seed * 1000 + q)
        out.append((nx, ny, nz, ek, float(rng.uniform(5, 15)), float(rng.uniform(-1, 1))))
    return out


def _plain_fp64(gpu, nx, ny, nz, ek, hl, hr, tol=1e-13, spacing=(1.0, 1.0, 1.0)):
    m = M.structured_hex(nx - 1, ny - 1, nz - 1, *spacing)
    eqs = gpu.LinearEQS(gpu.GpuMesh(m))
    eqs.Initialize()
    p = gpu.make_params(gpu.GROUNDWATER_FLOW, steady=1)
    eqs.GlobalAssembly(p, ek, np.zeros(m.n_nodes))
    lf, rf = m.face_nodes(0, 0), m.face_nodes(0, 1)
    eqs.SetKnownX(np.concatenate([lf, rf]), np.concatenate([np.full(len(lf), hl), np.full(len(rf), hr)]),
                  gpu.DIRICHLET_SYMMETRIC)
    eqs.ConfigNumerics(gpu.LS_CG, gpu.PRECOND_JACOBI, 20000, tol)
    x = np.zeros(m.n_nodes)
    x[lf], x[rf] = hl, hr
    eqs.Solver(x)
    return x


def test_batch_matches_plain_fp64_path(gpu):
    sizes = [(6, 5, 4), (9, 7, 5), (12, 10, 8), (3, 3, 3), (20, 6, 9), (15, 15, 15)]
    reals = _realisations(sizes, seed=1)
    b = gpu.Batch(reals, tol=1e-11)
    stats = b.solve()
    heads = b.heads()
    for (nx, ny, nz, ek, hl, hr), st, h in zip(reals, stats, heads):
        assert st["status"] == gpu.OK
        assert st["rel_residual"] < 1e-11
        assert st["iterations"] > 0 and st["refinements"] >= 2
        ref = _plain_fp64(gpu, nx, ny, nz, ek, hl, hr)
        assert rel_max_err(h, ref) < BATCH_RTOL, (nx, ny, nz)


def test_batch_homogeneous_linear_profile(gpu):
    """Homogeneous K: h = hl + (hr - hl) x / L exactly in trilinear FE."""
    reals = [(n, 4, 3, np.full((n - 1) * 3 * 2, 2e-4), 3.0, 1.0) for n in (5, 11, 17)]
    b = gpu.Batch(reals, hx=0.5, hy=2.0, hz=1.5, tol=1e-12)
    b.solve()
    for (nx, ny, nz, _, hl, hr), h in zip(reals, b.heads()):
        ix = np.arange(nx * ny * nz) % nx
        exact = hl + (hr - hl) * ix / (nx - 1)
        assert np.abs(h - exact).max() < 1e-9


def test_batch_tunings_agree_and_autotune(gpu):
    sizes = [(10, 8, 6), (14, 9, 7), (7, 7, 7), (18, 12, 5)]
    reals = _realisations(sizes, seed=3, var=2.0)
    b = gpu.Batch(reals, tol=1e-10)
    results = []
    for tr, nt, bps in ((64, 256, 1), (256, 512, 1), (4096, 256, 2)):
        b.set_tuning(tr, nt, bps)
        st = b.solve()
        assert all(s["status"] == gpu.OK for s in st)
        results.append(b.heads_flat())
    for r in results[1:]:
        assert rel_max_err(r, results[0]) < BATCH_RTOL
    t = b.autotune()
    assert t["tile_rows"] in (2048, 4096, 8192) and t["block_threads"] in (256, 512)
    assert t["blocks_per_sm"] >= 1 and t["ms_per_step"] > 0
    st = b.solve()
    assert all(s["status"] == gpu.OK for s in st)
    assert rel_max_err(b.heads_flat(), results[0]) < BATCH_RTOL


def test_batch_zero_rhs_and_not_converged(gpu):
    """h = 0 on both faces: b = 0, CheckNormRHS ends the solve at once with
    x = 0; a max_iter of 3 leaves the other realisations NOT_CONVERGED."""
    reals = [(6, 6, 6, np.full(125, 1e-5), 0.0, 0.0), (8, 6, 5, np.full(7 * 5 * 4, 1e-5), 1.0, 0.0)]
    b = gpu.Batch(reals, tol=1e-10)
    st = b.solve()
    assert st[0]["status"] == gpu.OK and st[0]["iterations"] == 0
    h = b.heads()
    assert np.all(h[0] == 0.0)
    b2 = gpu.Batch(reals, tol=1e-10, max_iter=3)
    st2 = b2.solve(allow_fail=True)
    assert st2[0]["status"] == gpu.OK
    assert st2[1]["status"] == gpu.NOT_CONVERGED


def test_batch_set_k_resolves(gpu):
    sizes = [(8, 7, 6), (11, 5, 4)]
    reals = _realisations(sizes, seed=5)
    b = gpu.Batch(reals, tol=1e-11)
    b.solve()
    new = _realisations(sizes, seed=6)
    b.set_k(np.concatenate([r[3] for r in new]))
    b.solve()
    for (nx, ny, nz, _, hl, hr), (_, _, _, ek, _, _), h in zip(reals, new, b.heads()):
        ref = _plain_fp64(gpu, nx, ny, nz, ek, hl, hr)
        assert rel_max_err(h, ref) < BATCH_RTOL


def test_batch_rejects_bad_input(gpu):
    with pytest.raises(gpu.OgsError):
        gpu.Batch([(2, 5, 5, np.ones(16), 1.0, 0.0)])
    with pytest.raises(ValueError):
        gpu.Batch([(4, 4, 4, np.ones(5), 1.0, 0.0)])


# Where the launch changes its form: one brick and many, bricks cut short at
# the far sides, more realisations than blocks, a box that fills the blocks and
# one that does not fit.
FORMS = {
    "one brick": [(3, 3, 3), (5, 40, 3), (17, 4, 12)],
    "remainders": [(33, 29, 31), (97, 13, 11), (64, 33, 5), (31, 32, 33)],
    "many": [(4 + q % 5, 3 + q % 4, 3 + q % 3) for q in range(400)],
    "one on all blocks": [(98, 98, 98)],
    "large and small": [(12, 10, 8), (96, 96, 96), (40, 40, 40), (7, 6, 5), (64, 60, 62)],
    "more bricks than blocks": [(104, 104, 104), (20, 20, 20)],
}


def _plain_system(gpu, nx, ny, nz, ek, hl, hr, spacing=(1.0, 1.0, 1.0)):
    m = M.structured_hex(nx - 1, ny - 1, nz - 1, *spacing)
    eqs = gpu.LinearEQS(gpu.GpuMesh(m))
    eqs.Initialize()
    eqs.GlobalAssembly(gpu.make_params(gpu.GROUNDWATER_FLOW, steady=1), ek, np.zeros(m.n_nodes))
    lf, rf = m.face_nodes(0, 0), m.face_nodes(0, 1)
    eqs.SetKnownX(np.concatenate([lf, rf]), np.concatenate([np.full(len(lf), hl), np.full(len(rf), hr)]),
                  gpu.DIRICHLET_SYMMETRIC)
    return (*eqs.get_csr(), eqs.get_rhs())


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("spacing", [(1.0, 1.0, 1.0), (0.5, 2.0, 1.5)])
def test_batch_forms(gpu, form, spacing):
    """The residual b - A h with the matrix of the plain path.  Bound: twice
    the solver's 1e-11 (the residual's own rounding is below 1e-12 of b)."""
    reals = _realisations(FORMS[form], seed=11)
    b = gpu.Batch(reals, hx=spacing[0], hy=spacing[1], hz=spacing[2], tol=1e-11)
    stats = b.solve()
    heads = b.heads()
    first = b.heads_flat().copy()
    for q, ((nx, ny, nz, ek, hl, hr), st, h) in enumerate(zip(reals, stats, heads)):
        assert st["status"] == gpu.OK and st["rel_residual"] < 1e-11
        if len(reals) > 50 and q % 13:
            continue
        rp, col, val, rhs = _plain_system(gpu, nx, ny, nz, ek, hl, hr, spacing)
        ax = np.add.reduceat(val * h[col], rp[:-1])
        assert np.linalg.norm(rhs - ax) < 2e-11 * np.linalg.norm(rhs), (nx, ny, nz)
    if form != "more bricks than blocks":
        # sums in a fixed order, whichever blocks a realisation lands on
        b.solve()
        assert np.array_equal(b.heads_flat(), first)


@pytest.mark.parametrize("nx", [1577, 1578])
def test_batch_long_lines(gpu, nx):
    """The longest line that a block holds, and the first that it does not:
    20 iterations against the same 20 of Jacobi-CG in FP64 (the solve itself
    would take tens of thousands).  20 FP32 iterations before the first
    replacement: 1e-5 of the largest head."""
    (_, ny, nz, ek, hl, hr), = _realisations([(nx, 3, 3)], seed=12)
    b = gpu.Batch([(nx, ny, nz, ek, hl, hr)], tol=1e-11, max_iter=20)
    st = b.solve(allow_fail=True)[0]
    assert st["status"] == gpu.NOT_CONVERGED
    rp, col, val, rhs = _plain_system(gpu, nx, ny, nz, ek, hl, hr)
    mul = lambda v: np.add.reduceat(val * v[col], rp[:-1])  # noqa: E731
    row = np.repeat(np.arange(len(rhs)), np.diff(rp))
    dinv = 1.0 / val[row == col]
    ix = np.arange(len(rhs)) % nx
    x = np.where(ix == 0, hl, np.where(ix == nx - 1, hr, 0.0))
    r = rhs - mul(x)
    z = dinv * r
    p, rho = z.copy(), r @ z
    for _ in range(20):
        w = mul(p)
        alpha = rho / (p @ w)
        x += alpha * p
        r -= alpha * w
        z = dinv * r
        rho, old = r @ z, rho
        p = z + rho / old * p
    assert rel_max_err(b.heads()[0], x) < 1e-5
    assert abs(st["rel_residual"] / (np.linalg.norm(r) / np.linalg.norm(rhs)) - 1.0) < 1e-4


@pytest.mark.parametrize("dims", [(9, 8, 7), (24, 24, 24)])
def test_negative_conductivities_solve_as_their_negatives(gpu, dims):
    """A negative definite operator (all conductivities negated) has the same
    heads, by the same iterations: every product changes sign."""
    nx, ny, nz = dims
    ek = fields.lognormal_k((nx - 1, ny - 1, nz - 1), np.log(1e-5), 1.0, 3.0, seed=4)
    got = []
    for k in (ek, -ek):
        b = gpu.Batch([(nx, ny, nz, k, 10.0, 0.0)], tol=1e-10)
        st = b.solve()[0]
        got.append((st["iterations"], st["refinements"], b.heads_flat().copy()))
    assert got[1][:2] == got[0][:2]
    assert np.array_equal(got[1][2], got[0][2])


def test_many_small_boxes_cost_no_more_than_their_iterations(gpu):
    """Boxes of one block each are taken by the blocks themselves (10,000 boxes of
    4^3: 9 ms; each given out under a lock 46 ms, the tile form 35 ms)."""
    rng = np.random.default_rng(0)
    reals = [(4, 4, 4, np.exp(np.log(1e-5) + 0.7 * rng.standard_normal(27)), 10.0, 0.0) for _ in range(10000)]
    b = gpu.Batch(reals, tol=1e-9)
    best = 1e9
    for _ in range(5):
        t = time.perf_counter()
        st = b.solve()
        best = min(best, time.perf_counter() - t)
    assert all(s["status"] == gpu.OK for s in st)
    assert best < 35e-3, best
    heads = b.heads()
    for q in (0, 303, 304, 5000, 9999):
        alone = gpu.Batch([reals[q]], tol=1e-9)
        alone.solve()
        assert rel_max_err(heads[q], alone.heads()[0]) < BATCH_RTOL


@pytest.mark.parametrize("sizes", [
    [(4, 4, 4)] * 1, [(4, 4, 4)] * 303, [(4, 4, 4)] * 304, [(4, 4, 4)] * 305, [(4, 4, 4)] * 700,  # one block each
    [(40, 40, 40)] * 30 + [(5, 5, 5)] * 500,                     # several blocks, then one
    [(90, 90, 90)] * 2 + [(6, 5, 4)] * 3,                        # idle blocks to the end
    [(90, 90, 90)] * 3 + [(30, 30, 30)] * 10 + [(4, 5, 6)] * 400])
def test_every_box_is_solved_once(gpu, sizes):
    reals = _realisations(sizes, seed=7)
    b = gpu.Batch(reals, tol=1e-9)
    for _ in range(2):
        st = b.solve()
        assert all(s["status"] == gpu.OK and s["rel_residual"] < 1e-9 for s in st)
    heads = b.heads()
    for q in sorted({0, len(sizes) // 2, len(sizes) - 1}):
        alone = gpu.Batch([reals[q]], tol=1e-9)
        alone.solve()
        assert rel_max_err(heads[q], alone.heads()[0]) < BATCH_RTOL
