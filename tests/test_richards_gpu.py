"""RICHARDS_FLOW on the GPU (ogs_gpu_assemble_richards, ogs_gpu_richards_step)
against the oracle: the assembled system at a partly unsaturated iterate
within 1e-12 per entry, and a Picard time step with the same number of
iterations and the same heads (1e-10 relative, the linear solves stopping at
1e-13)."""
import time

import numpy as np
import pytest

from ogs5_gb300 import mesh as M
from tests.helpers import SOLUTION_RTOL, assert_matrix_close, assert_vector_close, distort, rel_max_err

pytestmark = pytest.mark.gpu

RHO_G = 1000.0 * 9.81
LINEAR_TOL = 1e-13  # linear solves inside the Picard loops, GPU and oracle


def _mesh(kind):
    if kind == "quad":
        return M.structured_quad(10, 14, 0.2, 0.1)
    if kind == "hex":
        return distort(M.structured_hex(4, 3, 8, 0.5, 0.5, 0.25), 0.1, seed=3)
    if kind == "hex_box":  # axis-aligned boxes: the constant-geometry path
        return M.structured_hex(4, 3, 8, 0.5, 0.5, 0.25)
    return M.structured_tet(3, 3, 5, 0.5, 0.5, 0.3)


def _params(gpu, oracle, **kw):
    base = dict(dt=600.0, storage=1e-6, porosity=0.35, drho_dp=4.4e-10, viscosity=1e-3, density=1000.0,
                time_unit_factor=1.0)
    base.update(kw)
    return (gpu.make_params(gpu.RICHARDS_FLOW, **base), oracle.make_params(pcs_type=3, **base))


def _curves(gpu, oracle, model):
    kw = dict(capillary_model=model, permeability_model=model, pb=5.0e3, slr=0.08, slm=0.98,
              m=0.55 if model == 4 else 1.8, kr_slr=0.08, kr_slm=0.98, kr_m=0.55 if model == 4 else 1.8, kr_min=1e-9)
    return gpu.richards_params(**kw), oracle.richards_params(**kw)


def _pressure(m, seed):
    """hydrostatic-ish profile: saturated below a water table, suction above"""
    rng = np.random.default_rng(seed)
    top = m.z.max() if m.dim == 3 else m.y.max()
    h = (m.z if m.dim == 3 else m.y)
    return RHO_G * (0.4 * top - h) * 4.0 + rng.normal(0.0, 500.0, m.n_nodes)


@pytest.mark.parametrize("kind", ["quad", "hex", "hex_box", "tet"])
@pytest.mark.parametrize("opts", [(4, 0, 0), (4, 1, 1), (6, 1, 0), (6, 0, 1)])
def test_richards_assembly_matches_oracle(gpu, oracle, kind, opts):
    model, gravity, lumping = opts
    m = _mesh(kind)
    rng = np.random.default_rng(7)
    ek = np.exp(np.log(1e-12) + 0.5 * rng.standard_normal(m.n_elements))
    gp, op = _params(gpu, oracle, gravity=9.81 if gravity else 0.0, gravity_on=gravity, mass_lumping=lumping)
    gr, orr = _curves(gpu, oracle, model)
    p_old = _pressure(m, 1)
    p_it = _pressure(m, 2)
    eqs = gpu.LinearEQS(gpu.GpuMesh(m))
    eqs.Initialize()
    eqs.AssembleRichards(gp, gr, ek, p_old, p_it)
    rp, col, val = eqs.get_csr()
    orp, ocol = oracle.build_pattern(m.n_nodes, m.conn)
    assert np.array_equal(rp, orp) and np.array_equal(col, ocol)
    oval, ob = oracle.assemble_richards(m, orp, ocol, op, orr, ek, p_old, p_it)
    assert_matrix_close(rp, val, oval)
    assert_vector_close(eqs.get_rhs(), ob)
    assert (p_it < 0).any() and (p_it > 0).any()  # both branches of CalCoefMass


@pytest.mark.parametrize("kind,method", [("quad", 2), ("hex", 4), ("tet", 1)])
def test_richards_picard_step_matches_oracle(gpu, oracle, kind, method):
    """Infiltration into a dry column: top pressure 0 (saturated), bottom
    held at its suction; one Picard step of dt = 60 s from the dry state."""
    m = _mesh(kind)
    rng = np.random.default_rng(11)
    ek = np.exp(np.log(5e-12) + 0.3 * rng.standard_normal(m.n_elements))
    gp, op = _params(gpu, oracle, dt=60.0, gravity=9.81, gravity_on=1)
    gr, orr = _curves(gpu, oracle, 4)
    vert = m.z if m.dim == 3 else m.y
    p_old = np.full(m.n_nodes, -1.0e4)
    top = np.flatnonzero(vert == vert.max())
    bottom = np.flatnonzero(vert == vert.min())
    rows = np.concatenate([top, bottom])
    vals = np.concatenate([np.zeros(len(top)), np.full(len(bottom), -1.0e4)])
    eqs = gpu.LinearEQS(gpu.GpuMesh(m))
    eqs.ConfigNumerics(gpu.LS_CG, gpu.PRECOND_JACOBI, 5000, LINEAR_TOL, check_norm_rhs=False)
    it = p_old.copy()
    st = eqs.RichardsStep(gp, gr, ek, p_old, it, rows, vals, gpu.DIRICHLET_SYMMETRIC, error_method=method,
                          max_iterations=30, tolerance=1e-3 if method == 4 else 1.0)
    orp, ocol = oracle.build_pattern(m.n_nodes, m.conn)
    oit, info = oracle.richards_picard(m, orp, ocol, op, orr, ek, p_old, p_old, rows, vals, True,
                                       error_method=method, tolerance=1e-3 if method == 4 else 1.0,
                                       max_iterations=30, method=5, precond=1, tol=LINEAR_TOL)
    assert st["converged"] and info["converged"]
    assert st["iterations"] == info["iterations"] and st["iterations"] >= 3
    assert rel_max_err(it, oit) < SOLUTION_RTOL
    # the wetting front: pressures rose from the dry state, top held at 0
    assert np.all(it[top] == 0.0) and it.max() <= 1e-6 and np.mean(it) > -1.0e4


def test_richards_relaxation_and_stagnation(gpu, oracle):
    """nls_relaxation 0.5: relax0 / relax1 weigh the Laplace term and the
    iterate moves half way (theta 0.5), as in the oracle (converges in the
    same number of iterations); from a drier state with a longer step the
    error stops falling by 1 % twice in a row: stagnation, NOT_CONVERGED,
    after the same iterations as the oracle."""
    m = _mesh("quad")
    ek = np.full(m.n_elements, 5e-12)
    gr, orr = _curves(gpu, oracle, 4)
    top = np.flatnonzero(m.y == m.y.max())
    vals = np.zeros(len(top))
    orp, ocol = oracle.build_pattern(m.n_nodes, m.conn)
    eqs = gpu.LinearEQS(gpu.GpuMesh(m))
    eqs.ConfigNumerics(gpu.LS_CG, gpu.PRECOND_JACOBI, 5000, LINEAR_TOL, check_norm_rhs=False)
    for dt, dry, ok in ((10.0, -5.0e3, True), (60.0, -2.0e4, False)):
        gp, op = _params(gpu, oracle, dt=dt, gravity=9.81, gravity_on=1, nls_relaxation=0.5)
        p_old = np.full(m.n_nodes, dry)
        it = p_old.copy()
        st = eqs.RichardsStep(gp, gr, ek, p_old, it, top, vals, gpu.DIRICHLET_SYMMETRIC, error_method=2,
                              max_iterations=40, tolerance=1.0, allow_fail=True)
        oit, info = oracle.richards_picard(m, orp, ocol, op, orr, ek, p_old, p_old, top, vals, True, error_method=2,
                                           tolerance=1.0, max_iterations=40, tol=LINEAR_TOL)
        assert st["iterations"] == info["iterations"]
        assert st["converged"] == info["converged"] == ok and st["diverged"] == info["diverged"] == (not ok)
        assert st["status"] == (gpu.OK if ok else gpu.NOT_CONVERGED)
        if ok:
            assert rel_max_err(it, oit) < SOLUTION_RTOL


def test_richards_rejects_bad_input(gpu):
    m = _mesh("quad")
    eqs = gpu.LinearEQS(gpu.GpuMesh(m))
    p = gpu.make_params(gpu.RICHARDS_FLOW, dt=1.0, viscosity=1e-3)
    z = np.zeros(m.n_nodes)
    with pytest.raises(gpu.OgsError):
        eqs.AssembleRichards(p, gpu.richards_params(capillary_model=5), np.ones(m.n_elements), z, z)
    with pytest.raises(gpu.OgsError):
        eqs.AssembleRichards(p, gpu.richards_params(m=1.5), np.ones(m.n_elements), z, z)
    with pytest.raises(gpu.OgsError):  # RICHARDS_FLOW is not an ogs_gpu_assemble process
        eqs.GlobalAssembly(p, np.ones(m.n_elements), z)


@pytest.mark.parametrize("kind", ["quad", "hex"])
def test_richards_assembly_turned_boxes(gpu, oracle, kind):
    """Boxes along the axes whose first edge runs along y (the node order
    turned by a quarter): a Jacobian that is constant but not diagonal."""
    m = _mesh("quad" if kind == "quad" else "hex_box")
    turn = [1, 2, 3, 0] if kind == "quad" else [1, 2, 3, 0, 5, 6, 7, 4]
    m.conn = np.ascontiguousarray(m.conn[:, turn])
    ek = np.exp(np.log(1e-12) + 0.5 * np.random.default_rng(7).standard_normal(m.n_elements))
    gp, op = _params(gpu, oracle, gravity=9.81, gravity_on=1)
    gr, orr = _curves(gpu, oracle, 4)
    p_old, p_it = _pressure(m, 1), _pressure(m, 2)
    eqs = gpu.LinearEQS(gpu.GpuMesh(m))
    eqs.Initialize()
    eqs.AssembleRichards(gp, gr, ek, p_old, p_it)
    rp, col, val = eqs.get_csr()
    oval, ob = oracle.assemble_richards(m, rp, col, op, orr, ek, p_old, p_it)
    assert_matrix_close(rp, val, oval)
    assert_vector_close(eqs.get_rhs(), ob)


# Suction of a whole mesh, t = (pc / pb)^(1 / (1 - m)), around the limits of the
# form that shares the curves' logarithms (t = 1e-3, Se = 1e-3), saturated,
# and where the general form stays.
_T = [0.0, -1.0, 1e-12, 1e-6, 9.99e-4, 1.001e-3, 0.01, 0.3, 1.0, 7.0, 300.0, 1e4, 1e6, 1e9]


@pytest.mark.parametrize("kind", ["hex", "hex_box", "tet"])
@pytest.mark.parametrize("m_vg", [0.05, 0.3, 0.55, 0.9])
@pytest.mark.parametrize("curves", ["one m", "krel of another m", "krel of another range"])
def test_richards_curves(gpu, oracle, kind, m_vg, curves):
    """One pressure everywhere: the matrix is krel times the flow matrix (dt
    large) or the mass coefficient times the mass matrix (K = 0).  The curves
    in extended precision are the reference.  Bound: 1e-12 for the assembly,
    and for points that keep the general form the rounding it amplifies:
    2^-52 max(t, 1 / t) (2 + |log Se|) / m, eight times, t the larger of the
    curve's and krel's own (Se^(-1 / m) - 1 with its Se and m)."""
    msh = _mesh(kind)
    ld = np.longdouble
    pb, slr, slm = 5.0e3, 0.08, 0.98
    kr_m = m_vg if curves != "krel of another m" else 0.5 * m_vg
    kr_slr = slr if curves != "krel of another range" else 0.02
    gr = gpu.richards_params(capillary_model=4, permeability_model=4, pb=pb, slr=slr, slm=slm, m=m_vg, kr_slr=kr_slr,
                             kr_slm=slm, kr_m=kr_m, kr_min=1e-30)
    eqs = gpu.LinearEQS(gpu.GpuMesh(msh))
    one = np.ones(msh.n_elements)
    zero = np.zeros(msh.n_nodes)

    def matrix(k, t, **kw):
        p = zero - (t if t < 0 else pb * t ** (1.0 - m_vg))
        eqs.Initialize()
        eqs.AssembleRichards(gpu.make_params(gpu.RICHARDS_FLOW, porosity=0.35, viscosity=1.0, **kw), gr, k, p, p)
        return eqs.get_csr()[2], -p[0]

    def flow(k, **kw):
        eqs.Initialize()
        eqs.GlobalAssembly(gpu.make_params(gpu.GROUNDWATER_FLOW, **kw), k, zero)
        return eqs.get_csr()[2]

    lap = flow(one, dt=1.0, storage=0.0)
    mass = flow(0.0 * one, dt=1.0, storage=1.0)
    for t in _T:
        got_l, pc = matrix(one, t, dt=1e300, storage=0.0)
        got_m, _ = matrix(0.0 * one, t, dt=1.0, storage=1e-9)
        eps = ld(2.0) ** -52
        m = ld(m_vg)
        tt = (ld(max(pc, 0.0)) / ld(pb)) ** (1 / (1 - m))
        se = (1 + tt) ** -m
        s = min(max(se * (ld(slm) - ld(slr)) + ld(slr), ld(slr) + eps), ld(slm) - eps)
        se_k = (s - ld(kr_slr)) / (ld(slm) - ld(kr_slr))
        kr = max(np.sqrt(se_k) * (1 - (1 - se_k ** (1 / ld(kr_m))) ** ld(kr_m)) ** 2, ld(1e-30))
        cm = ld(1e-9)
        if pc > 0:
            sc = (s - ld(slr)) / (ld(slm) - ld(slr))
            v1 = sc ** (-1 / m)
            cm = ld(1e-9) * s - ld(0.35) * (m * (s - ld(slr))) / (ld(pb) * (m - 1) * v1 * (v1 - 1) ** -m)
        shared = curves == "one m" and tt > 1.0005e-3 and se > 1e-3
        tk = se_k ** (-1 / ld(kr_m)) - 1
        amp = 0.0 if shared else float(8 * eps * max(tt, tk, 1 / max(tt, eps), 1 / max(tk, eps)) *
                                       (2 - np.log(se)) / min(m, ld(kr_m)))
        if amp > 1e-3:
            continue  # the general form has no digits left there
        tol = 1e-12 + amp
        assert np.abs(got_l - float(kr) * lap).max() <= tol * float(kr) * np.abs(lap).max(), t
        assert np.abs(got_m - float(cm) * mass).max() <= tol * abs(float(cm)) * np.abs(mass).max(), t


@pytest.mark.parametrize("kind", ["quad", "hex", "tet"])
def test_richards_points_of_both_forms_in_a_warp(gpu, kind):
    """Pressures from far below the water table to above it in neighbouring
    nodes, some within the wet limit of the shared form: the same matrix as
    with a krel range that differs in the last place, which keeps every point
    in the general form (1e-9: the general form's own rounding)."""
    msh = _mesh(kind)
    rng = np.random.default_rng(5)
    p = -10.0 ** rng.uniform(-4.0, 4.5, msh.n_nodes)
    p[rng.random(msh.n_nodes) < 0.3] *= -1.0
    p[::7] = -1e-3
    got = []
    for slr in (0.08, 0.08 * (1.0 + 2.0 ** -50)):
        gr = gpu.richards_params(capillary_model=4, permeability_model=4, pb=5.0e3, slr=0.08, slm=0.98, m=0.55,
                                 kr_slr=slr, kr_slm=0.98, kr_m=0.55, kr_min=1e-9)
        eqs = gpu.LinearEQS(gpu.GpuMesh(msh))
        eqs.Initialize()
        eqs.AssembleRichards(gpu.make_params(gpu.RICHARDS_FLOW, dt=600.0, storage=1e-6, porosity=0.35, viscosity=1e-3), gr,
                             np.full(msh.n_elements, 1e-12), p, p)
        got.append(eqs.get_csr()[2])
    assert np.abs(got[0] - got[1]).max() <= 1e-9 * np.abs(got[1]).max()


def test_richards_small_meshes_at_a_water_table(gpu):
    """One wave of blocks whose pressures cross the water table takes no longer
    than with curves of different m, which take the powers at every point (1.3
    times as long where a warp went through both forms)."""
    import torch
    msh = M.structured_quad(60, 50)
    p = torch.linspace(-2e4, 1e4, msh.n_nodes, dtype=torch.float64, device="cuda")
    k = torch.full((msh.n_elements,), 1e-12, dtype=torch.float64, device="cuda")
    eqs = gpu.LinearEQS(gpu.GpuMesh(msh))
    prm = gpu.make_params(gpu.RICHARDS_FLOW, dt=600.0, storage=1e-6, porosity=0.35, viscosity=1e-3)
    best = {}
    for kr_m in (0.55, 0.5):
        gr = gpu.richards_params(capillary_model=4, permeability_model=4, pb=5.0e3, slr=0.08, slm=0.98, m=0.55,
                                 kr_slr=0.08, kr_slm=0.98, kr_m=kr_m, kr_min=1e-9)
        for _ in range(20):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            eqs.AssembleRichards(prm, gr, k, p, p)
            torch.cuda.synchronize()
            best[kr_m] = min(best.get(kr_m, 1e9), time.perf_counter() - t0)
    assert best[0.55] < 1.1 * best[0.5], best
