"""Multigrid solves of lines of more than 65535 tiles of 16 cells: along x and
along y, the axes whose tiles lie in the launch grid."""
import numpy as np
import pytest

from picfoam_gb300 import abi, cases
from picfoam_gb300.simulation import Simulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(1_050_000, 2, 1), (2, 1_050_000, 1)])
def test_long_line(gpu, n):
    side = [cases.patch(abi.PATCH_EMPTY if n[f // 2] == 1 else abi.PATCH_WALL) for f in range(6)]
    mesh = cases.block_mesh(n, tuple(1e-3 * v for v in n), side)
    cfg = cases.base_config(1e-12, [(cases.M_E, -cases.E_CHARGE, 1.0, True)], pcg_tol=1e-3)
    cfg.pcg_precond = abi.PRECOND_MULTIGRID
    sim = Simulation(mesh, cfg, backend=gpu)
    _, st = sim.solve_poisson(1e-6 * np.random.default_rng(1).standard_normal(sim.sizes()[0]))
    assert st.pcg_iterations > 0 and st.pcg_residual_l2 <= 1e-3
    sim.close()
