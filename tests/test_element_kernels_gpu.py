"""The tensor-product element kernels at the sizes where they can go wrong:
partly filled warps and blocks, 1 to 3 Gauss points an axis, constant and
varying Jacobians, against the CPU oracle.

Tolerances as everywhere (tests/helpers.py): the kernels add the same
Gauss-point terms in another order, so 1e-12 relative with a floor of 1e-14
times the largest value of the row.
"""
import numpy as np
import pytest

from ogs5_gb300 import mesh as M
from tests.helpers import assert_vector_close
from tests.test_parity_gpu import k_field, oracle_params

pytestmark = pytest.mark.gpu


def _shear(m):
    """Parallelepipeds: constant, full Jacobians (exact in binary)."""
    m.x = m.x + 0.25 * m.y + 0.5 * m.z
    m.y = m.y + 0.125 * m.z
    return m


SHAPES = [(3, 1, 1), (31, 1, 1), (4, 4, 2), (11, 3, 1), (13, 5, 3)]  # 3, 31, 32, 33, 195 cells


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("form,ngauss", [("box", 3), ("sheared", 3), ("distorted", 3), ("box", 1), ("distorted", 1),
                                         ("sheared", 2), ("distorted", 2), ("tet", 3), ("tet distorted", 3)])
def test_gauss_point_flux(gpu, oracle, shape, form, ngauss):
    make = M.structured_tet if form.startswith("tet") else M.structured_hex
    m = make(*shape, 1.0, 2.0, 0.5)
    if form == "sheared":
        m = _shear(m)
    if "distorted" in form:
        # every node moves: with one cell across an axis none is interior
        rng = np.random.default_rng(1)
        m.x, m.y, m.z = (c + 0.1 * s * rng.uniform(-1, 1, c.size) for c, s in zip((m.x, m.y, m.z), (1.0, 2.0, 0.5)))
    ek = k_field(m, 4)
    h = np.random.default_rng(3).uniform(0, 10, m.n_nodes)
    gm = gpu.GpuMesh(m, gauss_points=ngauss)
    eqs = gpu.LinearEQS(gm)
    for pcs, kw in ((gpu.GROUNDWATER_FLOW, {"time_unit_factor": 86400.0}),
                    (gpu.LIQUID_FLOW, {"gravity": 9.81, "gravity_on": 1, "viscosity": 1e-3})):
        p = gpu.make_params(pcs, **kw)
        q = eqs.gp_velocity(p, ek, h)
        qo = oracle.gp_velocity(m, oracle_params(oracle, p), ek, h, ngauss=ngauss)
        assert_vector_close(q.ravel(), qo.ravel())
