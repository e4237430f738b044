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
from tests.helpers import assert_matrix_close, assert_vector_close
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


def _hexes(shape, form):
    m = M.structured_hex(*shape, 1.0, 2.0, 0.5)
    if form == "sheared":
        return _shear(m)
    if form == "distorted":
        rng = np.random.default_rng(1)
        m.x, m.y, m.z = (c + 0.1 * s * rng.uniform(-1, 1, c.size) for c, s in zip((m.x, m.y, m.z), (1.0, 2.0, 0.5)))
    return m


def _system(eqs, oracle_values, m):
    rp, col, val = eqs.get_csr()
    oval, ob = oracle_values(rp, col)
    assert_matrix_close(rp, val, oval)
    assert_vector_close(eqs.get_rhs(), ob)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("form", ["box", "sheared", "distorted"])
@pytest.mark.parametrize("ngauss", [2, 3])
@pytest.mark.parametrize("lumping,theta", [(0, 1.0), (1, 0.6), (0, 0.5)])
def test_hex_transport(gpu, oracle, shape, form, ngauss, lumping, theta):
    m = _hexes(shape, form)
    rng = np.random.default_rng(5)
    gm = gpu.GpuMesh(m, gauss_points=ngauss)
    q = rng.normal(0.0, 1e-5, (m.n_elements, gm.n_gauss, 3))
    q[0] = 0.0  # the dispersion tensor's zero-velocity branch
    c0 = rng.uniform(0.0, 1.0, m.n_nodes)
    p = gpu.make_params(gpu.MASS_TRANSPORT, dt=3600.0, porosity=0.3, alpha_l=1.0, alpha_t=0.1, diffusion=1e-9,
                        decay=1e-6, retardation=1.2, theta=theta, mass_lumping=lumping, time_unit_factor=3.0)
    for stored in (0, 1):
        p.memory_type = stored
        eqs = gpu.LinearEQS(gm)
        eqs.Initialize()
        eqs.GlobalAssembly(p, None, c0, q)
        _system(eqs, lambda rp, col: oracle.assemble(m, rp, col, oracle_params(oracle, p), u0=c0, gp_vel=q,
                                                     ngauss=ngauss), m)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("ngauss", [1, 2, 3])
@pytest.mark.parametrize("lumping,relax", [(0, 0.0), (1, 0.3)])
def test_hex_flow_distorted(gpu, oracle, shape, ngauss, lumping, relax):
    m = _hexes(shape, "distorted")
    m.z = m.z + 1000.0  # the gravity term must not depend on the datum
    ek, u0 = k_field(m, 2), np.random.default_rng(3).uniform(0, 1e5, m.n_nodes)
    p = gpu.make_params(gpu.LIQUID_FLOW, dt=3600.0, storage=1e-9, porosity=0.2, drho_dp=4.4e-10, viscosity=1e-3,
                        density=1000.0, gravity=9.81, gravity_on=1, mass_lumping=lumping, nls_relaxation=relax)
    eqs = gpu.LinearEQS(gpu.GpuMesh(m, gauss_points=ngauss))
    eqs.Initialize()
    eqs.GlobalAssembly(p, ek, u0)
    # the system does not depend on the datum, the oracle's rounding does
    # (2.5e-12 in one entry between z and z - 1000, the same doubles of edge
    # lengths): it is evaluated with the datum taken off, an exact difference
    m.z = m.z - 1000.0
    _system(eqs, lambda rp, col: oracle.assemble(m, rp, col, oracle_params(oracle, p), elem_k=ek, u0=u0,
                                                 ngauss=ngauss), m)


@pytest.mark.parametrize("shape", [(1, 1), (2, 1), (1, 7), (15, 15), (16, 15), (33, 9), (130, 61)])
@pytest.mark.parametrize("pcs,lumping,relax", [("gw", 0, 0.0), ("gw", 1, 0.3), ("liquid", 0, 0.0), ("liquid", 1, 0.0)])
def test_quad_lattice_flow(gpu, oracle, shape, pcs, lumping, relax):
    """Rows of a plane lattice, and the same bit for bit in every assembly."""
    m = M.structured_quad(*shape, 2.0, 0.5)
    ek = k_field(m, 4)
    u = np.random.default_rng(5).uniform(0, 10, m.n_nodes)
    if pcs == "gw":
        p = gpu.make_params(gpu.GROUNDWATER_FLOW, dt=50.0, storage=1e-4, time_unit_factor=86400.0, mass_lumping=lumping,
                            nls_relaxation=relax)
    else:
        p = gpu.make_params(gpu.LIQUID_FLOW, dt=50.0, storage=1e-6, viscosity=1e-3, gravity=9.81, gravity_on=1,
                            mass_lumping=lumping, nls_relaxation=relax)
    gm = gpu.GpuMesh(m)
    got = []
    for _ in range(2):
        eqs = gpu.LinearEQS(gm)
        eqs.Initialize()
        eqs.GlobalAssembly(p, ek, u)
        got.append((eqs.get_csr()[2], eqs.get_rhs()))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    _system(eqs, lambda rp, col: oracle.assemble(m, rp, col, oracle_params(oracle, p), elem_k=ek, u0=u), m)


@pytest.mark.parametrize("columns", ["moved by 4e-12", "written with 12 digits", "of 0.1"])
@pytest.mark.parametrize("shape", [(16, 15), (130, 61)])
def test_quads_that_are_nearly_a_lattice(gpu, oracle, shape, columns):
    """Rectangles of almost the same width: every cell's entries are its own."""
    m = M.structured_quad(*shape, 1.0 if columns == "moved by 4e-12" else 0.1 if columns == "of 0.1" else 1.0 / 3.0, 0.5)
    if columns == "moved by 4e-12":
        xs, col = np.unique(m.x, return_inverse=True)
        xs[2:] += 4e-12 * np.random.default_rng(9).choice([-1.0, 1.0], xs.size - 2)  # the first cell's width is 1
        m.x = xs[col]
    elif columns == "written with 12 digits":
        m.x = np.array([float(f"{v:.11e}") for v in m.x])
    ek, u = k_field(m, 4), np.random.default_rng(5).uniform(0, 10, m.n_nodes)
    p = gpu.make_params(gpu.GROUNDWATER_FLOW, dt=50.0, storage=1e-4, time_unit_factor=86400.0)
    eqs = gpu.LinearEQS(gpu.GpuMesh(m))
    eqs.Initialize()
    eqs.GlobalAssembly(p, ek, u)
    _system(eqs, lambda rp, col: oracle.assemble(m, rp, col, oracle_params(oracle, p), elem_k=ek, u0=u), m)


@pytest.mark.parametrize("shape", [(1, 1, 1), (7, 3, 1), (4, 4, 4), (13, 5, 3)])  # 6, 126, 384, 1170 cells
@pytest.mark.parametrize("form", ["box", "mirrored", "distorted"])
@pytest.mark.parametrize("flux", ["per element", "per point", "mixed"])
@pytest.mark.parametrize("lumping,theta", [(0, 1.0), (1, 1.0), (0, 0.6)])
def test_tet_transport(gpu, oracle, shape, form, flux, lumping, theta):
    m = M.structured_tet(*shape, 1.0, 2.0, 0.5)
    rng = np.random.default_rng(6)
    if form == "mirrored":
        m.x = -m.x
    elif form == "distorted":
        m.x, m.y, m.z = (c + 0.1 * s * rng.uniform(-1, 1, c.size) for c, s in zip((m.x, m.y, m.z), (1.0, 2.0, 0.5)))
    gm = gpu.GpuMesh(m)
    q = rng.normal(0.0, 1e-5, (m.n_elements, gm.n_gauss, 3))
    every = {"per element": slice(None), "per point": slice(0, 0), "mixed": slice(None, None, 2)}[flux]
    q[every] = q[every][:, :1, :]
    q[0] = 0.0  # the dispersion tensor's zero-velocity branch
    c0 = rng.uniform(0.0, 1.0, m.n_nodes)
    p = gpu.make_params(gpu.MASS_TRANSPORT, dt=3600.0, porosity=0.3, alpha_l=1.0, alpha_t=0.1, diffusion=1e-9,
                        decay=1e-6, retardation=1.2, theta=theta, mass_lumping=lumping, time_unit_factor=3.0)
    eqs = gpu.LinearEQS(gm)
    eqs.Initialize()
    eqs.GlobalAssembly(p, None, c0, q)
    _system(eqs, lambda rp, col: oracle.assemble(m, rp, col, oracle_params(oracle, p), u0=c0, gp_vel=q), m)


@pytest.mark.parametrize("lists", ["one run", "two faces", "65 runs", "shuffled", "none"])
@pytest.mark.parametrize("mode", ["row", "symmetric"])
def test_dirichlet_list_orders_and_device_values(gpu, lists, mode):
    """The order of a row list decides only which of a row's values is last;
    matrix values into a device array are those of the host array."""
    torch = pytest.importorskip("torch")
    m = M.structured_hex(15, 9, 7)
    rng = np.random.default_rng(8)
    rows = {"one run": np.arange(0, 60), "two faces": np.concatenate([m.face_nodes(0, 0), m.face_nodes(0, 1)]),
            "65 runs": np.tile(np.arange(3, 40, 5), 65), "shuffled": rng.permutation(np.tile(np.arange(50, 200), 2)),
            "none": np.zeros(0, dtype=np.int64)}[lists]
    vals = rng.uniform(0.0, 1.0, len(rows))
    last = dict(zip(rows.tolist(), vals.tolist()))  # the last occurrence of each row
    out = []
    for r, v in ((rows, vals), (np.array(sorted(last), dtype=np.int64), np.array([last[q] for q in sorted(last)]))):
        eqs = gpu.LinearEQS(gpu.GpuMesh(m))
        eqs.Initialize()
        eqs.GlobalAssembly(gpu.make_params(gpu.GROUNDWATER_FLOW, dt=1.0, storage=1e-3), np.full(m.n_elements, 1e-3),
                           np.zeros(m.n_nodes))
        eqs.SetKnownX(r, v, gpu.DIRICHLET_ROW_ONLY if mode == "row" else gpu.DIRICHLET_SYMMETRIC)
        host = eqs.get_values()
        dev = torch.full((len(host) + 1,), -7.0, dtype=torch.float64, device="cuda")
        eqs.get_values(dev[1:])
        assert np.array_equal(dev[1:].cpu().numpy(), host) and dev[0].item() == -7.0
        out.append((host, eqs.get_rhs()))
    assert np.array_equal(out[0][0], out[1][0])
    if lists in ("one run", "two faces", "none"):  # no row twice: the right-hand side as well
        assert np.array_equal(out[0][1], out[1][1])
