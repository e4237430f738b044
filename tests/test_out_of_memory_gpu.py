"""A solve that runs out of device memory half way through its allocations (the
failing call is faked) ends with OGS_OOM; made again it has all of its arrays
and gives the heads of a system that never failed."""
import numpy as np
import pytest

from ogs5_gb300 import mesh as M

pytestmark = pytest.mark.gpu

# how many allocations the first solve makes at most: the ILU(0) factor, its
# packed rows and its tile arrays are 21; one FP32 block
CASES = [("ilu", "tet", n) for n in (1, 2, 5, 6, 12, 13, 14, 15, 18, 21)] + [("ilu", "hex", 7)] + [
    ("fp32", "hex", 1), ("fp32", "tet", 1)]


@pytest.mark.parametrize("what,kind,n", CASES)
def test_a_solve_out_of_memory_can_be_made_again(gpu, what, kind, n):
    m = M.structured_tet(11, 9, 8) if kind == "tet" else M.structured_hex(11, 9, 8)
    rng = np.random.default_rng(1)
    ek = np.exp(np.log(1e-5) + 0.5 * rng.standard_normal(m.n_elements))
    lf = m.face_nodes(0, 0)
    gm = gpu.GpuMesh(m)
    heads = []
    for fail in (0, n):
        eqs = gpu.LinearEQS(gm)
        if what == "ilu":
            eqs.ConfigNumerics(gpu.LS_BICGSTAB, gpu.PRECOND_ILU0, 500, 1e-12, check_norm_rhs=False)
        else:
            eqs.ConfigNumerics(gpu.LS_CG, gpu.PRECOND_JACOBI, 2000, 1e-12, precision=gpu.PRECISION_FP32_REFINED,
                               check_norm_rhs=False)
        eqs.Initialize()
        eqs.GlobalAssembly(gpu.make_params(gpu.GROUNDWATER_FLOW, dt=3600.0, storage=1e-4), ek, np.zeros(m.n_nodes))
        eqs.SetKnownX(lf, np.ones(len(lf)), gpu.DIRICHLET_SYMMETRIC)
        x = np.zeros(m.n_nodes)
        if fail:
            gpu.debug_fail_alloc(fail)
            with pytest.raises(gpu.OgsError) as e:
                eqs.Solver(x)
            gpu.debug_fail_alloc(0)
            assert e.value.status == gpu.OOM
            x = np.zeros(m.n_nodes)
        eqs.Solver(x)
        assert eqs.stats()["status"] == gpu.OK
        heads.append(x)
    assert np.abs(heads[1] - heads[0]).max() < 1e-10
