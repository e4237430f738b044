"""Timed cases: what a program that uses this library has it do.

Every case is one pass through the public Python entry points
(``ogs5_gb300.capi``) on device-resident inputs, the calls a time loop, a
Monte-Carlo study or a request server makes again and again:

    flow       one GROUNDWATER_FLOW step: Initialize, GlobalAssembly, SetKnownX, Solver
    assembly   one LIQUID_FLOW assembly with its Dirichlet rows, matrix and right-hand side read back
    transport  Gauss-point flux of a head field, then one MASS_TRANSPORT step on it
    richards   one RICHARDS_FLOW time step by Picard iteration
    batch      one Monte-Carlo batch: new conductivities, solve, heads
    serve      a burst of flow and transport requests through the server

``listed()`` gives the fixed cases, ``draw(rng)`` others of the same ranges,
``prepare(case, seed)`` what the program has in hand before the call,
``run(state)`` one pass, ``work(case)`` the bytes and operations it cannot do
without, ``exact(case, seed)`` the same outputs by plain torch in 64 bits.
The mesh (node coordinates, connectivity, the device mesh made from them) is
the program's for its whole life and is kept between prepare() calls of one
geometry; conductivities, heads and everything else come from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from ogs5_gb300 import capi, fields
from ogs5_gb300 import mesh as M

DT = 3600.0          # s, implicit-Euler step of the transient decks
STORAGE = 1e-4       # 1/m
HEAD = 10.0          # m, head on x = 0 (0 on the far face)
MEAN_LNK = math.log(1e-5)
POROSITY, ALPHA_L, ALPHA_T, DIFFUSION = 0.3, 1.0, 0.1, 1e-9
RICH_SPACING = (0.25, 0.25, 0.0625)
RICH_MEDIUM = dict(capillary_model=4, permeability_model=4, pb=5.0e3, slr=0.08, slm=0.98, m=0.55, kr_slr=0.08,
                   kr_slm=0.98, kr_m=0.55, kr_min=1e-9)
RICH_FLUID = dict(dt=DT, storage=1e-6, porosity=0.35, drho_dp=4.4e-10, viscosity=1e-3, density=1000.0,
                  time_unit_factor=1.0, gravity=9.81, gravity_on=1)
LIQUID = dict(dt=DT, storage=1e-9, porosity=0.2, drho_dp=4.4e-10, viscosity=1e-3, density=1000.0, gravity=9.81,
              gravity_on=1)


# ------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------
def listed():
    return [
        # the smallest deck, 100 x 100 quads, steady, the default BiCGStab + Jacobi: kernel latency
        dict(name="quad100 flow bicgstab", kind="flow", elem="quad", nx=100, ny=100, nz=0, jitter=0.0, steady=1,
             method="bicgstab", precision="fp64", tol=1e-12),
        # one small realisation or request on an odd-sized box, FP32-inner CG
        dict(name="hex small flow fp32", kind="flow", elem="hex", nx=33, ny=27, nz=21, jitter=0.0, steady=1,
             method="cg", precision="fp32", tol=1e-12),
        # a large 2-D aquifer, steady: thousands of FP64 CG iterations
        dict(name="quad large flow cg", kind="flow", elem="quad", nx=999, ny=701, nz=0, jitter=0.0, steady=1,
             method="cg", precision="fp64", tol=1e-12),
        # the transient deck (1.08M nodes), plain FP64 path
        dict(name="hex deck flow fp64", kind="flow", elem="hex", nx=128, ny=128, nz=64, jitter=0.0, steady=0,
             method="cg", precision="fp64", tol=1e-12),
        # the transient deck with the FP32-inner solver: the headline workload
        dict(name="hex deck flow fp32", kind="flow", elem="hex", nx=128, ny=128, nz=64, jitter=0.0, steady=0,
             method="cg", precision="fp32", tol=1e-12),
        # a fitted (non-affine) hex mesh whose matrix goes to the host program's own solver
        dict(name="hex fitted assembly", kind="assembly", elem="hex", nx=61, ny=53, nz=47, jitter=0.2),
        # solute step on the tet split of the deck, flux from the heads, Jacobi
        dict(name="tet deck transport jacobi", kind="transport", elem="tet", nx=128, ny=128, nz=64, jitter=0.0,
             precond="jacobi", stored=0),
        # the same with ILU(0), on a smaller odd-sized box
        dict(name="tet transport ilu", kind="transport", elem="tet", nx=65, ny=57, nz=41, jitter=0.0,
             precond="ilu", stored=0),
        # solute step on hexes, as the server's transport requests
        dict(name="hex transport jacobi", kind="transport", elem="hex", nx=63, ny=63, nz=63, jitter=0.0,
             precond="jacobi", stored=0),
        # unsaturated flow: a Picard time step
        dict(name="hex richards step", kind="richards", elem="hex", nx=64, ny=64, nz=48),
        # a Monte-Carlo study: uneven boxes of 24 to 96 nodes an edge
        dict(name="monte carlo batch", kind="batch", reals=24, n_lo=24, n_hi=96, sizes=4, tol=1e-11),
        # a burst of requests on mixed meshes
        dict(name="serve burst", kind="serve", requests=24, cells=20000, spread=8, tol=1e-11, sizes=5),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, n_lo, n_hi):
    """Three edge lengths (cells) around the edge of a box of n_lo..n_hi nodes."""
    n = math.exp(rng.uniform(math.log(n_lo), math.log(n_hi)))
    e = n ** (1.0 / 3.0)
    nx = max(6, int(e * rng.uniform(0.7, 1.4)))
    ny = max(6, int(e * rng.uniform(0.7, 1.4)))
    return nx, ny, max(6, int(n / ((nx + 1) * (ny + 1))) - 1)


def draw(rng):
    kind = rng.choice(["flow", "flow", "flow", "assembly", "transport", "transport", "richards", "batch", "serve"])
    if kind == "flow":
        elem = rng.choice(["quad", "hex", "hex", "tet"])
        if elem == "quad":
            n = math.exp(rng.uniform(math.log(2e3), math.log(5e5)))
            a = rng.uniform(0.6, 1.6)
            nx, ny, nz = int(math.sqrt(n) * a), int(math.sqrt(n) / a), 0
        else:
            nx, ny, nz = _box(rng, 4e3, 9e5)
        method = rng.choice(["cg", "cg", "bicgstab"])
        # FP32-inner runs CG; steady 2-D problems of this size are FP64 work
        precision = rng.choice(["fp64", "fp32"]) if method == "cg" and elem != "quad" else "fp64"
        return dict(kind="flow", elem=elem, nx=nx, ny=ny, nz=nz, jitter=rng.choice([0.0, 0.0, 0.2]),
                    steady=rng.choice([0, 1]), method=method, precision=precision, tol=1e-12)
    if kind == "assembly":
        nx, ny, nz = _box(rng, 8e3, 2e5)
        return dict(kind="assembly", elem=rng.choice(["hex", "tet"]), nx=nx, ny=ny, nz=nz,
                    jitter=rng.choice([0.0, 0.2]))
    if kind == "transport":
        elem = rng.choice(["hex", "tet", "tet"])
        nx, ny, nz = _box(rng, 8e3, 3e5)
        return dict(kind="transport", elem=elem, nx=nx, ny=ny, nz=nz, jitter=rng.choice([0.0, 0.2]),
                    precond=rng.choice(["jacobi", "jacobi", "ilu"]), stored=rng.choice([0, 0, 1]))
    if kind == "richards":
        nx, ny, nz = _box(rng, 1e4, 1.5e5)
        return dict(kind="richards", elem="hex", nx=nx, ny=ny, nz=nz)
    if kind == "batch":
        return dict(kind="batch", reals=rng.randint(4, 24), n_lo=24, n_hi=rng.randint(40, 88),
                    sizes=rng.randint(0, 1 << 20), tol=1e-11)
    return dict(kind="serve", requests=rng.randint(8, 24), cells=_logint(rng, 8000, 20000), spread=rng.randint(2, 8),
                tol=1e-11, sizes=rng.randint(0, 1 << 20))


# ------------------------------------------------------------------
# meshes and inputs
# ------------------------------------------------------------------
def _make_mesh(elem, nx, ny, nz, jitter=0.0, spacing=(1.0, 1.0, 1.0)):
    if elem == "quad":
        m = M.structured_quad(nx, ny, *spacing[:2])
    elif elem == "hex":
        m = M.structured_hex(nx, ny, nz, *spacing)
    else:
        m = M.structured_tet(nx, ny, nz, *spacing)
    if jitter:
        # a fitted mesh: interior nodes moved by up to jitter cells on each axis
        rng = np.random.default_rng(nx * 1000003 + ny * 1009 + nz)
        axes = [(m.x, 0), (m.y, 1)] + ([(m.z, 2)] if m.dim == 3 else [])
        inside = np.ones(m.n_nodes, bool)
        for c, _ in axes:
            inside &= (c > c.min()) & (c < c.max())
        for c, a in axes:
            c[inside] += jitter * spacing[a] * rng.uniform(-1.0, 1.0, int(inside.sum()))
    return m


_KEPT = {}


def _kept(key, make):
    """One geometry at a time: what the program makes once and keeps."""
    if key not in _KEPT:
        _KEPT.clear()
        _KEPT[key] = make()
    return _KEPT[key]


def _case_mesh(case):
    spacing = RICH_SPACING if case["kind"] == "richards" else (1.0, 1.0, 1.0)
    key = (case["elem"], case["nx"], case["ny"], case["nz"], case.get("jitter", 0.0), spacing)
    return _kept(key, lambda: _with_device(_make_mesh(*key)))


def _with_device(m):
    return m, capi.GpuMesh(m)


def _conductivity(elem, nx, ny, nz, seed, mean=MEAN_LNK, var=1.0, ell=8.0):
    """Log-normal field on the cells (tets: the field of their parent hex)."""
    shape = (nx, ny) if elem == "quad" else (nx, ny, nz)
    k = fields.lognormal_k_device(shape, mean, var, ell, seed=seed)
    return k.repeat_interleave(6).contiguous() if elem == "tet" else k


def _faces(m):
    lf, rf = m.face_nodes(0, 0), m.face_nodes(0, 1)
    return lf, rf


def _dev(a, dtype=None):
    return torch.tensor(a, device="cuda", dtype=dtype)


def _heads(m, seed):
    """A head field between the faces: the linear profile and a few smooth
    modes that vanish on both faces."""
    rng = np.random.default_rng(seed)
    x, y, z = (_dev(c) for c in (m.x, m.y, m.z))
    lx, ly, lz = (float(c.max() - c.min()) or 1.0 for c in (m.x, m.y, m.z))
    h = HEAD * (1.0 - x / lx)
    for _ in range(4):
        a, i, j, k = rng.uniform(-0.3, 0.3), *(int(v) for v in rng.integers(1, 4, 3))
        h += a * torch.sin(math.pi * i * x / lx) * torch.cos(math.pi * j * y / ly) * torch.cos(math.pi * k * z / lz)
    return h


def _flow_inputs(case, m, seed):
    lf, rf = _faces(m)
    rows = np.concatenate([lf, rf])
    vals = np.concatenate([np.full(len(lf), HEAD), np.zeros(len(rf))])
    u0 = torch.zeros(m.n_nodes, dtype=torch.float64, device="cuda")
    u0[_dev(lf)] = HEAD
    k = _conductivity(case["elem"], case["nx"], case["ny"], case["nz"], seed)
    return k, u0, rows, vals


def _transport_inputs(case, m, seed):
    lf, _ = _faces(m)
    c0 = torch.zeros(m.n_nodes, dtype=torch.float64, device="cuda")
    k = _conductivity(case["elem"], case["nx"], case["ny"], case["nz"], seed)
    return k, _heads(m, seed), c0, lf, np.ones(len(lf))


def _richards_inputs(case, m, seed):
    k = _conductivity("hex", case["nx"], case["ny"], case["nz"], seed, math.log(1e-12), 0.5, 4.0)
    p_old = 9810.0 * (0.5 * case["nz"] * RICH_SPACING[2] - m.z)  # hydrostatic, water table at mid-depth
    top, bot = np.flatnonzero(m.z == m.z.max()), np.flatnonzero(m.z == m.z.min())
    rows = np.concatenate([top, bot])
    vals = np.concatenate([np.full(len(top), -5.0e3), p_old[bot]])
    return k, _dev(p_old), rows, vals


def _batch_sizes(case):
    rng = np.random.default_rng(case["sizes"])
    n = rng.integers(case["n_lo"], case["n_hi"] + 1, case["reals"])
    return [int(v) for v in n], rng.uniform(0.5, 2.0, case["reals"]), rng.uniform(4.0, 16.0, case["reals"])


def _batch_inputs(case, seed):
    ns, var, ell = _batch_sizes(case)
    ks = [fields.lognormal_k_device((n - 1,) * 3, MEAN_LNK, float(v), float(e), seed=seed * 1000 + q)
          for q, (n, v, e) in enumerate(zip(ns, var, ell))]
    return ns, ks


def _serve_classes(case):
    """(elem, cells, kind) of the burst's classes: hex and tet boxes and one
    quad plane around `cells` cells, the larger ones `spread` times that."""
    out = []
    for f in (1, case["spread"]):
        e = max(6, int(round((case["cells"] * f) ** (1.0 / 3.0))))
        out += [("hex", (e + 1, e, e - 1), 0), ("hex", (e + 1, e, e - 1), 1), ("tet", (e, e - 1, e), 0),
                ("tet", (e, e - 1, e), 1)]
    s = max(12, int(round(math.sqrt(case["cells"]))))
    return out + [("quad", (s + 3, s, 0), 0)]


def _serve_order(case):
    rng = np.random.default_rng(case["sizes"])
    return [int(v) for v in rng.integers(0, len(_serve_classes(case)), case["requests"])]


def _serve_inputs(case, seed):
    cls = _serve_classes(case)
    return [(c, _conductivity(cls[c][0], *cls[c][1], seed * 1000 + q)) for q, c in enumerate(_serve_order(case))]


def _steady_flow():
    return capi.make_params(capi.GROUNDWATER_FLOW, steady=1)


def _transport_params(stored=0):
    return capi.make_params(capi.MASS_TRANSPORT, dt=DT, porosity=POROSITY, alpha_l=ALPHA_L, alpha_t=ALPHA_T,
                            diffusion=DIFFUSION, memory_type=1 if stored else 0)


# ------------------------------------------------------------------
# prepare and run
# ------------------------------------------------------------------
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    with torch.cuda.stream(state["stream"]):
        return state["run"](state)


def _state(fn, **kw):
    torch.cuda.current_stream().synchronize()  # inputs were made on this stream, the pass runs on its own
    return dict(run=fn, **kw)


def _system(gm):
    stream = torch.cuda.Stream()
    return stream, capi.LinearEQS(gm, stream=stream)


def _prepare_flow(case, seed):
    m, gm = _case_mesh(case)
    k, u0, rows, vals = _flow_inputs(case, m, seed)
    stream, eqs = _system(gm)
    eqs.ConfigNumerics(capi.LS_CG if case["method"] == "cg" else capi.LS_BICGSTAB, capi.PRECOND_JACOBI, 20000,
                       case["tol"],
                       precision=capi.PRECISION_FP32_REFINED if case["precision"] == "fp32" else capi.PRECISION_FP64)
    p = _steady_flow() if case["steady"] else capi.make_params(capi.GROUNDWATER_FLOW, dt=DT, storage=STORAGE)
    return _state(_run_flow, stream=stream, eqs=eqs, p=p, k=k, u0=u0, x=torch.empty_like(u0), rows=_dev(rows),
                  vals=_dev(vals))


def _run_flow(s):
    eqs = s["eqs"]
    eqs.Initialize()
    eqs.GlobalAssembly(s["p"], s["k"], s["u0"])
    eqs.SetKnownX(s["rows"], s["vals"], capi.DIRICHLET_SYMMETRIC)
    s["x"].copy_(s["u0"])
    eqs.Solver(s["x"])
    return {"heads": s["x"]}


def _prepare_assembly(case, seed):
    m, gm = _case_mesh(case)
    k, u0, rows, vals = _flow_inputs(case, m, seed)
    stream, eqs = _system(gm)
    return _state(_run_assembly, stream=stream, eqs=eqs, p=capi.make_params(capi.LIQUID_FLOW, **LIQUID),
                  k=k * 1e-7, u0=u0 * 9810.0, rows=_dev(rows), vals=_dev(vals * 9810.0),
                  val=torch.empty(gm.nnz, dtype=torch.float64, device="cuda"),
                  rhs=torch.empty(gm.n_rows, dtype=torch.float64, device="cuda"))


def _run_assembly(s):
    eqs = s["eqs"]
    eqs.Initialize()
    eqs.GlobalAssembly(s["p"], s["k"], s["u0"])
    eqs.SetKnownX(s["rows"], s["vals"], capi.DIRICHLET_ROW_ONLY)
    return {"matrix": eqs.get_values(s["val"]), "rhs": eqs.get_rhs(s["rhs"])}


def _prepare_transport(case, seed):
    m, gm = _case_mesh(case)
    k, h, c0, rows, vals = _transport_inputs(case, m, seed)
    stream, eqs = _system(gm)
    eqs.ConfigNumerics(capi.LS_BICGSTAB, capi.PRECOND_ILU0 if case["precond"] == "ilu" else capi.PRECOND_JACOBI, 5000,
                       1e-12, check_norm_rhs=False)
    q = torch.empty((m.n_elements, gm.n_gauss, 3), dtype=torch.float64, device="cuda")
    return _state(_run_transport, stream=stream, eqs=eqs, flow=capi.make_params(capi.GROUNDWATER_FLOW),
                  p=_transport_params(case["stored"]), k=k, h=h, c0=c0, q=q, x=torch.empty_like(c0), rows=_dev(rows),
                  vals=_dev(vals))


def _run_transport(s):
    eqs = s["eqs"]
    eqs.gp_velocity(s["flow"], s["k"], s["h"], s["q"])
    eqs.Initialize()
    eqs.GlobalAssembly(s["p"], None, s["c0"], s["q"])
    eqs.SetKnownX(s["rows"], s["vals"], capi.DIRICHLET_ROW_ONLY)
    s["x"].copy_(s["c0"])
    eqs.Solver(s["x"])
    return {"flux": s["q"], "concentration": s["x"]}


def _prepare_richards(case, seed):
    m, gm = _case_mesh(case)
    k, p_old, rows, vals = _richards_inputs(case, m, seed)
    stream, eqs = _system(gm)
    eqs.ConfigNumerics(capi.LS_CG, capi.PRECOND_JACOBI, 20000, 1e-12, check_norm_rhs=False)
    return _state(_run_richards, stream=stream, eqs=eqs, p=capi.make_params(capi.RICHARDS_FLOW, **RICH_FLUID),
                  r=capi.richards_params(**RICH_MEDIUM), k=k, p_old=p_old, it=torch.empty_like(p_old),
                  rows=_dev(rows), vals=_dev(vals))


def _run_richards(s):
    s["it"].copy_(s["p_old"])
    s["stream"].synchronize()
    s["eqs"].RichardsStep(s["p"], s["r"], s["k"], s["p_old"], s["it"], s["rows"], s["vals"],
                          capi.DIRICHLET_SYMMETRIC, error_method=capi.ENORM, max_iterations=40, tolerance=1.0)
    return {"pressure": s["it"]}


def _prepare_batch(case, seed):
    ns, ks = _batch_inputs(case, seed)
    stream = torch.cuda.Stream()
    torch.cuda.current_stream().synchronize()
    b = capi.Batch([(n, n, n, k, HEAD, 0.0) for n, k in zip(ns, ks)], tol=case["tol"], max_iter=20000,
                   stream=stream.cuda_stream)
    return _state(_run_batch, stream=stream, b=b, k=torch.cat(ks),
                  heads=torch.empty(b.rows, dtype=torch.float64, device="cuda"))


def _run_batch(s):
    s["b"].set_k(s["k"])
    s["b"].solve()
    return {"heads": s["b"].heads_flat(s["heads"])}


def _serve_meshes(case):
    cls = _serve_classes(case)
    key = ("serve", case["cells"], case["spread"])
    return _kept(key, lambda: {c[:2]: _with_device(_make_mesh(c[0], *c[1])) for c in cls})


def _prepare_serve(case, seed):
    meshes = _serve_meshes(case)
    srv = capi.Server(budget_bytes=16 << 30, max_active=16, flags=capi.SERVER_PRIORITY | capi.SERVER_SJF |
                      capi.SERVER_BATCH)
    cids = []
    for elem, dims, kind in _serve_classes(case):
        m, gm = meshes[(elem, dims)]
        lf, rf = _faces(m)
        if kind == 0:
            precision = capi.PRECISION_FP64 if elem == "quad" else capi.PRECISION_FP32_REFINED
            cids.append(srv.add_class(gm, capi.REQUEST_FLOW, _steady_flow(), np.concatenate([lf, rf]),
                                      np.concatenate([np.full(len(lf), HEAD), np.zeros(len(rf))]),
                                      capi.DIRICHLET_SYMMETRIC,
                                      capi.solver_config(capi.LS_CG, capi.PRECOND_JACOBI, 20000,
                                                         precision=precision)))
        else:
            cids.append(srv.add_class(gm, capi.REQUEST_TRANSPORT, _transport_params(), lf, np.ones(len(lf)),
                                      capi.DIRICHLET_ROW_ONLY,
                                      capi.solver_config(capi.LS_BICGSTAB, capi.PRECOND_JACOBI, 5000),
                                      flow_params=capi.make_params(capi.GROUNDWATER_FLOW),
                                      flow_head=HEAD * (1.0 - m.x / m.x.max())))
    reqs = [(cids[c], k, torch.zeros(meshes[_serve_classes(case)[c][:2]][0].n_nodes, dtype=torch.float64,
                                     device="cuda")) for c, k in _serve_inputs(case, seed)]
    return _state(_run_serve, stream=torch.cuda.Stream(), srv=srv, reqs=reqs, tol=case["tol"])


def _run_serve(s):
    ids = [s["srv"].submit(c, k, s["tol"], out) for c, k, out in s["reqs"]]
    s["srv"].drain()
    for i in ids:
        s["srv"].result(i)
    return [out for _, _, out in s["reqs"]]


# ------------------------------------------------------------------
# work
# ------------------------------------------------------------------
def _counts(elem, nx, ny, nz):
    """(nodes, elements, stored entries per row, nodes per element, Gauss points)"""
    if elem == "quad":
        return (nx + 1) * (ny + 1), nx * ny, 9, 4, 9
    n, c = (nx + 1) * (ny + 1) * (nz + 1), nx * ny * nz
    return (n, c, 27, 8, 27) if elem == "hex" else (n, 6 * c, 15, 4, 5)


def _iterations(edge, tol, steady):
    """CG iterations of a flow solve, from those of the decks: a few per cell
    along the longest edge, bounded by the storage term when transient."""
    it = 6.0 * edge * -math.log10(tol) / 11.0
    return it if steady else min(it, 330.0)


def _flow_work(elem, nx, ny, nz, tol, steady, krylov=1):
    n, e, row, nn, _ = _counts(elem, nx, ny, nz)
    it = _iterations(max(nx, ny, nz), tol, steady) / (1 if krylov == 1 else 1.5)
    return 8.0 * (e + 2 * n), 6.0 * nn * nn * e + it * krylov * n * (2.0 * row + 12.0)


def _transport_work(elem, nx, ny, nz):
    n, e, row, nn, gp = _counts(elem, nx, ny, nz)
    return 8.0 * (e + 3 * n + 3 * gp * e), (40.0 * gp + 12.0 * nn * nn) * e + 15 * n * (4.0 * row + 24.0)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        per = [_flow_work("hex", n - 1, n - 1, n - 1, case["tol"], 1) for n in _batch_sizes(case)[0]]
    elif kind == "serve":
        cls = _serve_classes(case)
        per = [(_flow_work(cls[c][0], *cls[c][1], case["tol"], 1) if cls[c][2] == 0 else
                _transport_work(cls[c][0], *cls[c][1])) for c in _serve_order(case)]
    else:
        dims = case["elem"], case["nx"], case["ny"], case["nz"]
        n, e, row, nn, gp = _counts(*dims)
        if kind == "flow":
            per = [_flow_work(*dims, case["tol"], case["steady"], 1 if case["method"] == "cg" else 2)]
        elif kind == "transport":
            per = [_transport_work(*dims)]
        elif kind == "assembly":
            per = [(8.0 * (e + 3 * n + row * n), 6.0 * gp * nn * nn * e)]
        else:  # richards: about 20 Picard iterations of 20 linear ones
            per = [(8.0 * (e + 3 * n), 20.0 * (gp * 150.0 * e + 20 * n * (2.0 * row + 12.0)))]
    return {"bytes": sum(p[0] for p in per), "flops": sum(p[1] for p in per)}


# ------------------------------------------------------------------
# the same in plain torch, 64 bits
# ------------------------------------------------------------------
_HEX = torch.tensor([[1, 1, 1], [-1, 1, 1], [-1, -1, 1], [1, -1, 1], [1, 1, -1], [-1, 1, -1], [-1, -1, -1],
                     [1, -1, -1]], dtype=torch.float64)


def _quadrature(elem):
    """Per integration point: weight, N [nn], dN [dim, nn] (points in the order r, s, t of 3-point Gauss)."""
    if elem == "tet":
        a, grad = 1.0 / 6.0, torch.tensor([[-1, 1, 0, 0], [-1, 0, 1, 0], [-1, 0, 0, 1]], dtype=torch.float64)
        pts = [(0.25, 0.25, 0.25, -2.0 / 15.0), (a, a, a, 0.075), (0.5, a, a, 0.075), (a, 0.5, a, 0.075),
               (a, a, 0.5, 0.075)]
        return [(w, torch.tensor([1 - r - s - t, r, s, t], dtype=torch.float64), grad) for r, s, t, w in pts]
    g, w = [math.sqrt(0.6), 0.0, -math.sqrt(0.6)], [5.0 / 9.0, 8.0 / 9.0, 5.0 / 9.0]
    out, dim = [], 2 if elem == "quad" else 3
    node = _HEX[:4, :2] if dim == 2 else _HEX
    for i in np.ndindex(*(3,) * dim):
        f = [1.0 + node[:, d] * g[i[d]] for d in range(dim)]
        scale = 0.5 ** dim
        n = scale * torch.stack(f).prod(0)
        dn = torch.stack([scale * node[:, d] * torch.stack([f[q] for q in range(dim) if q != d]).prod(0)
                          for d in range(dim)])
        out.append((math.prod(w[q] for q in i), n, dn))
    return out


class _Fem:
    """Element integrals of a mesh and the equation system they add up to."""

    def __init__(self, elem, m):
        self.elem, self.dim, self.n = elem, m.dim, m.n_nodes
        self.conn = torch.from_numpy(np.ascontiguousarray(m.conn)).cuda().long()
        xyz = torch.stack([_dev(c) for c in (m.x, m.y, m.z)[: m.dim]], 1)
        self.xe = xyz[self.conn]  # [E, nn, dim]
        self.quad = [(w, a.cuda(), d.cuda()) for w, a, d in _quadrature(elem)]
        self.lines = None

    def points(self):
        """Per integration point: w |J| [E], N [nn], grad N [E, dim, nn]."""
        last = None
        for w, n, dn in self.quad:
            if last is None or self.elem != "tet":
                j = torch.einsum("ki,eid->ekd", dn, self.xe)
                det = torch.linalg.det(j).abs()
                last = det, torch.linalg.solve(j, dn.expand(len(j), -1, -1))
            yield w * last[0], n, last[1]

    def matrix(self, ke):
        """Element matrices [E, nn, nn] summed into a CSR matrix."""
        if self.lines is None:
            key = (self.conn[:, :, None] * self.n + self.conn[:, None, :]).reshape(-1)
            u, inv = torch.unique(key, return_inverse=True)
            crow = torch.searchsorted(u, torch.arange(self.n + 1, device="cuda") * self.n)
            self.lines = crow, u % self.n, inv, u // self.n
        crow, col, inv, _ = self.lines
        return torch.zeros(len(col), dtype=torch.float64, device="cuda").index_add_(0, inv, ke.reshape(-1))

    def csr(self, val):
        return torch.sparse_csr_tensor(self.lines[0], self.lines[1], val, (self.n, self.n))

    def vector(self, fe):
        return torch.zeros(self.n, dtype=torch.float64, device="cuda").index_add_(0, self.conn.reshape(-1),
                                                                                 fe.reshape(-1))


def _outer(w, n):
    return w[:, None, None] * torch.outer(n, n)


def _pcg(mul, b, dinv, tol, most):
    x = torch.zeros_like(b)
    r = b.clone()
    z = dinv * r
    p, rz, goal = z.clone(), torch.dot(r, z), tol * float(b.norm())
    for it in range(most):
        if it % 25 == 0 and float(r.norm()) <= goal:
            break
        s = mul(p)
        a = rz / torch.dot(p, s)
        x += a * p
        r -= a * s
        z = dinv * r
        new = torch.dot(r, z)
        p = z + (new / rz) * p
        rz = new
    return x


def _pbicgstab(mul, b, dinv, tol, most=400):
    x, r = torch.zeros_like(b), b.clone()
    r0, p, goal = r.clone(), r.clone(), tol * float(b.norm())
    rho = torch.dot(r0, r)
    for _ in range(most):
        if float(r.norm()) <= goal:
            break
        ph = dinv * p
        v = mul(ph)
        a = rho / torch.dot(r0, v)
        s = r - a * v
        sh = dinv * s
        t = mul(sh)
        w = torch.dot(t, s) / torch.dot(t, t)
        x += a * ph + w * sh
        r = s - w * t
        new = torch.dot(r0, r)
        if not bool(new):
            break
        p = r + (new / rho) * (a / w) * (p - w * v)
        rho = new
    return x


def _dirichlet_solve(fem, val, b, rows, vals, symmetric, rounds=3):
    """A x = b with x given on rows, the free rows by Jacobi-preconditioned
    CG or BiCGStab with the residual recomputed between rounds."""
    a = fem.csr(val)
    free = torch.ones(fem.n, dtype=torch.float64, device="cuda")
    free[_dev(rows)] = 0.0
    x = torch.zeros_like(free)
    x[_dev(rows)] = _dev(vals)
    diag = val[fem.lines[3] == fem.lines[1]]
    dinv = 1.0 / diag
    mul = lambda v: free * (a @ v)  # noqa: E731  (v is zero on the given rows)
    for k in range(rounds):
        r = free * (b - a @ x)
        tol = 1e-13 if k == 0 else 1e-6
        x += _pcg(mul, r, dinv, tol, 30000) if symmetric else _pbicgstab(mul, r, dinv, tol)
    return x


def _exact_flow(elem, m, k, u0, rows, vals, steady):
    fem = _Fem(elem, m)
    nn = fem.conn.shape[1]
    ke = torch.zeros(len(fem.conn), nn, nn, dtype=torch.float64, device="cuda")
    me = None if steady else torch.zeros_like(ke)
    for w, n, g in fem.points():
        ke += (w * k)[:, None, None] * (g.transpose(1, 2) @ g)
        if me is not None:
            me += _outer(w * (STORAGE / DT), n)
    b = torch.zeros(fem.n, dtype=torch.float64, device="cuda")
    if me is not None:
        b = fem.vector((me @ u0[fem.conn][:, :, None])[:, :, 0])
        ke += me
    del me
    return _dirichlet_solve(fem, fem.matrix(ke), b, rows, vals, True)


def _exact_assembly(case, seed):
    m = _make_mesh(case["elem"], case["nx"], case["ny"], case["nz"], case["jitter"])
    k, u0, rows, vals = _flow_inputs(case, m, seed)
    mat = (k * 1e-7) * (1.0 / LIQUID["viscosity"])
    u0, vals = u0 * 9810.0, vals * 9810.0
    fem = _Fem(case["elem"], m)
    nn = fem.conn.shape[1]
    ke = torch.zeros(len(fem.conn), nn, nn, dtype=torch.float64, device="cuda")
    me, ge = torch.zeros_like(ke), torch.zeros(len(fem.conn), nn, dtype=torch.float64, device="cuda")
    cm = (LIQUID["storage"] + LIQUID["porosity"] * LIQUID["drho_dp"]) / DT
    for w, n, g in fem.points():
        ke += (w * mat)[:, None, None] * (g.transpose(1, 2) @ g)
        me += _outer(w * cm, n)
        ge -= (w * mat * (LIQUID["density"] * LIQUID["gravity"]))[:, None] * g[:, -1]
    b = fem.vector((me @ u0[fem.conn][:, :, None])[:, :, 0] + ge)
    val = fem.matrix(ke + me)
    _, col, _, row = fem.lines
    given = torch.zeros(fem.n, dtype=torch.bool, device="cuda")
    given[_dev(rows)] = True
    diag = val[row == col]
    b[_dev(rows)] = diag[_dev(rows)] * _dev(vals)
    val[given[row] & (row != col)] = 0.0
    return {"matrix": val, "rhs": b}


def _exact_transport(elem, m, k, h, c0, rows, vals):
    fem = _Fem(elem, m)
    nn, ne = fem.conn.shape[1], len(fem.conn)
    ke = torch.zeros(ne, nn, nn, dtype=torch.float64, device="cuda")
    q = torch.zeros(ne, len(fem.quad), 3, dtype=torch.float64, device="cuda")
    me = torch.zeros_like(ke)
    eye = torch.eye(fem.dim, dtype=torch.float64, device="cuda")
    for i, (w, n, g) in enumerate(fem.points()):
        v = -k[:, None] * (g @ h[fem.conn][:, :, None])[:, :, 0]
        q[:, i, : fem.dim] = v
        s = v.norm(dim=1)
        d = (ALPHA_T * s + DIFFUSION * POROSITY)[:, None, None] * eye
        d += ((ALPHA_L - ALPHA_T) / s)[:, None, None] * (v[:, :, None] * v[:, None, :])
        ke += w[:, None, None] * (g.transpose(1, 2) @ (d @ g))
        ke += w[:, None, None] * (n[None, :, None] * (v[:, None, :] @ g))
        me += _outer(w * (POROSITY / DT), n)
    b = fem.vector((me @ c0[fem.conn][:, :, None])[:, :, 0])
    ke += me
    del me
    return q, _dirichlet_solve(fem, fem.matrix(ke), b, rows, vals, False)


def _exact_richards(case, seed):
    m = _make_mesh("hex", case["nx"], case["ny"], case["nz"], 0.0, RICH_SPACING)
    k, p_old, rows, vals = _richards_inputs(case, m, seed)
    fem = _Fem("hex", m)
    med, flu = RICH_MEDIUM, RICH_FLUID
    vm, eps = med["m"], float(np.finfo(np.float64).eps)
    rng, it = med["slm"] - med["slr"], p_old.clone()
    for _ in range(40):
        ke = torch.zeros(len(fem.conn), 8, 8, dtype=torch.float64, device="cuda")
        me, ge = torch.zeros_like(ke), torch.zeros(len(fem.conn), 8, dtype=torch.float64, device="cuda")
        for w, n, g in fem.points():
            p = it[fem.conn] @ n
            se = (((-p).clamp_min(0.0) / med["pb"]) ** (1.0 / (1.0 - vm)) + 1.0) ** -vm
            sw = (se * rng + med["slr"]).clamp(med["slr"] + eps, med["slm"] - eps)
            eff = (sw - med["slr"]) / rng
            kr = (eff.sqrt() * (1.0 - (1.0 - eff ** (1.0 / vm)) ** vm) ** 2).clamp_min(med["kr_min"])
            v1 = eff ** (-1.0 / vm)
            ds = (vm * (sw - med["slr"])) / (med["pb"] * (vm - 1.0) * v1 * (v1 - 1.0) ** -vm)
            wet = p < 0.0
            sm = torch.where(wet, sw, torch.ones_like(sw))
            cm = flu["storage"] * sm + flu["porosity"] * sm * flu["drho_dp"] + torch.where(
                wet, -flu["porosity"] * ds.clamp_min(-1.0 / eps), torch.zeros_like(sw))
            mat = k * kr / flu["viscosity"]
            ke += (w * mat)[:, None, None] * (g.transpose(1, 2) @ g)
            me += _outer(w * cm / flu["dt"], n)
            ge -= (w * mat * (flu["density"] * flu["gravity"]))[:, None] * g[:, -1]
        b = fem.vector((me @ p_old[fem.conn][:, :, None])[:, :, 0] + ge)
        x = _dirichlet_solve(fem, fem.matrix(ke + me), b, rows, vals, True, rounds=2)
        err = float((it - x).norm())
        it = x
        if err <= 1.0:
            break
    return {"pressure": it}


def exact(case, seed):
    kind = case["kind"]
    if kind == "richards":
        return _exact_richards(case, seed)
    if kind == "assembly":
        return _exact_assembly(case, seed)
    if kind == "batch":
        ns, ks = _batch_inputs(case, seed)
        heads = []
        for n, k in zip(ns, ks):
            m = _make_mesh("hex", n - 1, n - 1, n - 1)
            _, u0, rows, vals = _flow_inputs(dict(elem="hex", nx=n - 1, ny=n - 1, nz=n - 1), m, seed)
            heads.append(_exact_flow("hex", m, k, u0, rows, vals, 1))
        return {"heads": torch.cat(heads)}
    if kind == "serve":
        cls, meshes, out = _serve_classes(case), {}, []
        for c, k in _serve_inputs(case, seed):
            elem, dims, req = cls[c]
            m = meshes.setdefault((elem, dims), _make_mesh(elem, *dims))
            lf, rf = _faces(m)
            if req == 0:
                vals = np.concatenate([np.full(len(lf), HEAD), np.zeros(len(rf))])
                out.append(_exact_flow(elem, m, k, None, np.concatenate([lf, rf]), vals, 1))
            else:
                c0 = torch.zeros(m.n_nodes, dtype=torch.float64, device="cuda")
                c0[_dev(lf)] = 1.0
                out.append(_exact_transport(elem, m, k, _dev(HEAD * (1.0 - m.x / m.x.max())), c0, lf,
                                            np.ones(len(lf)))[1])
        return out
    m = _make_mesh(case["elem"], case["nx"], case["ny"], case["nz"], case["jitter"])
    if kind == "flow":
        k, u0, rows, vals = _flow_inputs(case, m, seed)
        return {"heads": _exact_flow(case["elem"], m, k, u0, rows, vals, case["steady"])}
    k, h, c0, rows, vals = _transport_inputs(case, m, seed)
    q, c = _exact_transport(case["elem"], m, k, h, c0, rows, vals)
    return {"flux": q, "concentration": c}
