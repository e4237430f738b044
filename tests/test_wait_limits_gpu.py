"""The waits of the many-iteration solver launches, of the ILU(0) tile kernels
and of the batch's groups of blocks, made to run out in ordinary solves by a
limit of one poll (some block always polls more than once before the last
one arrives): the call ends with an error status, every block leaves, and
the next solve, with the kernels' own limits back, gives the result of the
one before bit for bit."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from ogs5_gb300 import build as B
from ogs5_gb300 import fields
from ogs5_gb300 import mesh as M

pytestmark = pytest.mark.gpu


def _system(gpu, m, method, precond, precision):
    rng = np.random.default_rng(1)
    eqs = gpu.LinearEQS(gpu.GpuMesh(m))
    eqs.ConfigNumerics(method, precond, 2000, 1e-10, precision=precision, check_norm_rhs=False)
    eqs.Initialize()
    ek = np.exp(np.log(1e-5) + 0.5 * rng.standard_normal(m.n_elements))
    eqs.GlobalAssembly(gpu.make_params(gpu.GROUNDWATER_FLOW, dt=3600.0, storage=1e-4), ek, np.zeros(m.n_nodes))
    lf, rf = m.face_nodes(0, 0), m.face_nodes(0, 1)
    eqs.SetKnownX(np.concatenate([lf, rf]), np.concatenate([np.full(len(lf), 10.0), np.zeros(len(rf))]),
                  gpu.DIRICHLET_SYMMETRIC)
    return eqs


def _solve(gpu, eqs, n):
    x = np.zeros(n)
    eqs.Solver(x, allow_fail=True)
    return x, eqs.stats()["status"]


# sizes whose blocks wait on one another through global memory: a grid for
# CG, BiCGStab and the FP32-inner CG, tiles for ILU(0)
CASES = [("cg", "hex", (30, 28, 26), False), ("bicgstab", "hex", (30, 28, 26), False), ("fp32", "hex", (30, 28, 26), False),
         ("fp32", "tet", (30, 28, 26), False), ("ilu", "tet", (20, 18, 17), False), ("ilu", "tet", (20, 18, 17), True)]


@pytest.mark.parametrize("what,kind,dims,factorisation", CASES)
def test_a_solve_whose_waits_run_out_ends_with_an_error(gpu, what, kind, dims, factorisation):
    m = M.structured_hex(*dims) if kind == "hex" else M.structured_tet(*dims)
    eqs = _system(gpu, m, gpu.LS_BICGSTAB if what in ("bicgstab", "ilu") else gpu.LS_CG,
                  gpu.PRECOND_ILU0 if what == "ilu" else gpu.PRECOND_JACOBI,
                  gpu.PRECISION_FP32_REFINED if what == "fp32" else gpu.PRECISION_FP64)
    x, status = _solve(gpu, eqs, m.n_nodes)
    assert status == gpu.OK
    for _ in range(2):
        eqs.debug_wait_limit(1, factorisation)
        with pytest.raises(gpu.OgsError) as e:
            eqs.Solver(np.zeros(m.n_nodes))
        assert e.value.status == gpu.CUDA_ERROR
        eqs.debug_wait_limit(0)
        again, status = _solve(gpu, eqs, m.n_nodes)
        assert status == gpu.OK
        assert np.array_equal(again, x)


@pytest.mark.parametrize("sizes", [[(25, 25, 25)], [(40, 30, 20)] * 3 + [(12, 10, 8)] * 5, [(60, 60, 60)] * 4])
def test_a_batch_whose_waits_run_out_ends_with_an_error(gpu, sizes):
    reals = [(nx, ny, nz, fields.lognormal_k((nx - 1, ny - 1, nz - 1), np.log(1e-5), 1.0, 3.0, seed=q), 10.0, 0.0)
             for q, (nx, ny, nz) in enumerate(sizes)]
    b = gpu.Batch(reals, tol=1e-10)
    b.solve()
    x = b.heads_flat().copy()
    for _ in range(2):
        b.debug_wait_limit(1)
        with pytest.raises(gpu.OgsError) as e:
            b.solve()
        assert e.value.status == gpu.CUDA_ERROR
        b.debug_wait_limit(0)
        b.solve()
        assert np.array_equal(b.heads_flat(), x)


def test_blocks_without_work_wait_while_others_progress(gpu):
    """Six boxes that each need more than half of the blocks are solved one
    after the other; the blocks left over wait for all of them.  Their limit
    (8192 polls of about 1 us) is far below that, and far above both what a
    block waits for its own group and the time between two signs of progress."""
    n = 90
    reals = [(n, n, n, fields.lognormal_k((n - 1, n - 1, n - 1), np.log(1e-5), 1.0, 3.0, seed=q), 10.0, 0.0)
             for q in range(6)]
    b = gpu.Batch(reals, tol=1e-10)
    b.solve()
    x = b.heads_flat().copy()
    b.debug_wait_limit(8192)
    b.solve()
    assert np.array_equal(b.heads_flat(), x)


def test_tiles_that_wait_often_but_never_long():
    """The limit of the ILU(0) tile kernels is of the polls of one wait, not
    of a tile's walk through its 22 steps."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-m", "tests.ilu_delay_case"], cwd=root,
                       env=dict(os.environ, OGS_GPU_LIB=B.build(debug=True)), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, (r.stdout[-2000:], r.stderr[-2000:])
    got = [json.loads(x) for x in r.stdout.splitlines() if x.startswith("{")]
    assert got == [{"factorisation": f, "error": "", "equal": True} for f in (False, True)]


def test_wait_limit_rejects_bad_arguments(gpu):
    with pytest.raises(gpu.OgsError):
        _system(gpu, M.structured_hex(2, 2, 2), gpu.LS_CG, gpu.PRECOND_JACOBI,
                gpu.PRECISION_FP64).debug_wait_limit(-1)


@pytest.mark.parametrize("what", ["cg", "bicgstab", "fp32"])
def test_a_wait_that_gave_up_outweighs_the_recorded_end(gpu, what):
    """Block 0 may record the end of a solve after another block gave up on
    the same last wait.  A few rows: one cluster, whose waits are hardware
    barriers, converges beside the record."""
    m = M.structured_hex(6, 5, 4)
    eqs = _system(gpu, m, gpu.LS_BICGSTAB if what == "bicgstab" else gpu.LS_CG, gpu.PRECOND_JACOBI,
                  gpu.PRECISION_FP32_REFINED if what == "fp32" else gpu.PRECISION_FP64)
    eqs.debug_wait_limit(0, recorded=True)
    x, status = _solve(gpu, eqs, m.n_nodes)
    assert status == gpu.CUDA_ERROR
    eqs.debug_wait_limit(0)
    assert _solve(gpu, eqs, m.n_nodes)[1] == gpu.OK
