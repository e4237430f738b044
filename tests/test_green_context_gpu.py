"""Solves on a stream that has part of the SMs (a stream of a CUDA green
context): launches whose blocks wait on one another do not fit there, so the
solver keeps to single-step graphs, and the heads are those of the same
solve on a stream with the whole GPU."""
import ctypes as C

import numpy as np
import pytest

from ogs5_gb300 import mesh as M
from tests.helpers import rel_max_err

pytestmark = pytest.mark.gpu

RESOURCE_BYTES = 144  # sizeof(CUdevResource)


@pytest.fixture(scope="module")
def part_of_the_sms():
    """A stream with a quarter of the SMs."""
    import torch
    torch.zeros(1, device="cuda")  # the primary context is current
    cu = C.CDLL("libcuda.so.1")
    dev, n = C.c_int(), C.c_uint(1)
    whole, part, rest = (C.create_string_buffer(RESOURCE_BYTES) for _ in range(3))
    desc, ctx, stream = C.c_void_p(), C.c_void_p(), C.c_void_p()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    steps = [lambda: cu.cuDeviceGet(C.byref(dev), 0),
             lambda: cu.cuDeviceGetDevResource(dev, whole, 1),
             lambda: cu.cuDevSmResourceSplitByCount(part, C.byref(n), whole, rest, 0, C.c_uint(sms // 4)),
             lambda: cu.cuDevResourceGenerateDesc(C.byref(desc), part, 1),
             lambda: cu.cuGreenCtxCreate(C.byref(ctx), desc, dev, 1),
             lambda: cu.cuGreenCtxStreamCreate(C.byref(stream), ctx, 1, 0)]
    for k, step in enumerate(steps):
        rc = step()
        if rc != 0:
            pytest.skip(f"no green contexts here (step {k}: {rc})")
    return stream.value


# a cluster's size, a grid's, and one of a row a thread on every SM
SHAPES = [("hex", (7, 6, 5)), ("quad", (60, 60)), ("hex", (30, 28, 26)), ("tet", (30, 28, 26)), ("quad", (200, 131))]


@pytest.mark.parametrize("kind,dims", SHAPES)
@pytest.mark.parametrize("what", ["cg", "bicgstab", "fp32"])
def test_solves_on_part_of_the_sms(gpu, part_of_the_sms, kind, dims, what):
    m = {"hex": M.structured_hex, "quad": M.structured_quad, "tet": M.structured_tet}[kind](*dims)
    rng = np.random.default_rng(2)
    ek = np.exp(np.log(1e-5) + 0.5 * rng.standard_normal(m.n_elements))
    lf, rf = m.face_nodes(0, 0), m.face_nodes(0, 1)
    gm = gpu.GpuMesh(m)
    x = []
    for stream in (None, part_of_the_sms):
        eqs = gpu.LinearEQS(gm, stream=stream)
        eqs.ConfigNumerics(gpu.LS_BICGSTAB if what == "bicgstab" else gpu.LS_CG, gpu.PRECOND_JACOBI, 20000, 1e-13 if
                           what != "fp32" else 1e-11,
                           precision=gpu.PRECISION_FP32_REFINED if what == "fp32" else gpu.PRECISION_FP64,
                           check_norm_rhs=False)
        eqs.Initialize()
        eqs.GlobalAssembly(gpu.make_params(gpu.GROUNDWATER_FLOW, dt=3600.0, storage=1e-4), ek, np.zeros(m.n_nodes))
        eqs.SetKnownX(np.concatenate([lf, rf]), np.concatenate([np.full(len(lf), 10.0), np.zeros(len(rf))]),
                      gpu.DIRICHLET_SYMMETRIC)
        h = np.zeros(m.n_nodes)
        eqs.Solver(h)
        assert eqs.stats()["status"] == gpu.OK
        x.append(h)
    assert rel_max_err(x[1], x[0]) < (1e-8 if what == "fp32" else 1e-10)
