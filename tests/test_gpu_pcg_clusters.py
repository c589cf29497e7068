"""The cluster forms of the persistent Poisson PCG when the launch did not form
the clusters that the plan counts on: the kernel gives the system back
untouched and the two-kernel iteration solves it, with the oracle's bits, in
this solve and in the ones that follow."""
import numpy as np
import pytest

import pyoracle
from picfoam_gb300 import abi, cases, native
from picfoam_gb300.simulation import Simulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(8, 8, 8), (32, 32, 1), (20, 32, 31), (38, 32, 33)])
def test_unplanned_clusters_take_the_streamed_iteration(gpu, n):
    side = [cases.patch(abi.PATCH_EMPTY if n[f // 2] == 1 else abi.PATCH_WALL, 2.0 * f) for f in range(6)]
    mesh = cases.block_mesh(n, tuple(1e-3 * v for v in n), side)
    cfg = cases.base_config(1e-12, [(cases.M_E, -cases.E_CHARGE, 1.0, True)], pcg_tol=1e-9)
    g = Simulation(mesh, cfg, backend=gpu)
    o = Simulation(mesh, cfg, backend=pyoracle.OracleBackend(1))
    rho = 1e-5 * np.random.default_rng(3).standard_normal(g.sizes()[0])
    for ranks in (None, 0, None):       # as planned, told of no cluster, and after that
        if ranks is not None:
            assert native.load().picgpu_test_pcg_ranks(g._h, ranks) == abi.OK
        pg, sg = g.solve_poisson(rho)
        po, so = o.solve_poisson(rho)
        assert sg.pcg_iterations == so.pcg_iterations > 0
        assert sg.pcg_residual_l2 == so.pcg_residual_l2 and sg.pcg_residual_initial == so.pcg_residual_initial
        assert np.array_equal(pg, po)
        assert np.array_equal(g.field(abi.FIELD_E_CELL), o.field(abi.FIELD_E_CELL))
        rho = rho[::-1].copy()
    g.close()
    o.close()
