"""ILU(0) on a lattice of two tiles, the first of which pauses 200 us before
each of its last 14 steps, with 1500 polls a wait: a pause takes some 200 to
600 polls, all of them together several thousand.  Child process of
tests/test_wait_limits_gpu.py, with OGS_GPU_LIB pointing at the debug
library; prints the status of the solve and whether the heads are those
without the pauses."""
import json

import numpy as np

from ogs5_gb300 import capi as gpu
from ogs5_gb300 import mesh as M


def main():
    m = M.structured_tet(15, 7, 7)
    gm = gpu.GpuMesh(m)
    assert gm.ilu_tiles == 2
    eqs = gpu.LinearEQS(gm)
    eqs.ConfigNumerics(gpu.LS_BICGSTAB, gpu.PRECOND_ILU0, 200, 1e-10, check_norm_rhs=False)
    eqs.Initialize()
    rng = np.random.default_rng(3)
    ek = np.exp(np.log(1e-5) + 0.5 * rng.standard_normal(m.n_elements))
    eqs.GlobalAssembly(gpu.make_params(gpu.GROUNDWATER_FLOW, dt=3600.0, storage=1e-4), ek, np.zeros(m.n_nodes))
    lf = m.face_nodes(0, 0)
    eqs.SetKnownX(lf, np.ones(len(lf)), gpu.DIRICHLET_ROW_ONLY)
    x = np.zeros(m.n_nodes)
    eqs.Solver(x)
    for factorisation in (False, True):
        eqs.debug_wait_limit(1500, factorisation)
        eqs.debug_ilu_delay(200000)
        y = np.zeros(m.n_nodes)
        try:
            eqs.Solver(y)
            error = ""
        except gpu.OgsError as e:
            error = str(e)
        print(json.dumps({"factorisation": factorisation, "error": error, "equal": bool(np.array_equal(x, y))}))


if __name__ == "__main__":
    main()
