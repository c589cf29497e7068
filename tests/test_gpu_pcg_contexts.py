"""Poisson solves of contexts of different sizes that live side by side: what one
context's plan sets up for the solver kernel must not be taken from another's.
Four chunks of cells per block (80^3) and two (64^3) share a kernel."""
import numpy as np
import pytest

import pyoracle
from picfoam_gb300 import abi, cases
from picfoam_gb300.simulation import Simulation

pytestmark = pytest.mark.gpu


def make(n, backend, precond=abi.PRECOND_JACOBI):
    mesh = cases.block_mesh((n, n, n), (1e-3 * n,) * 3, [cases.patch(abi.PATCH_WALL, 2.0 * f) for f in range(6)])
    cfg = cases.base_config(1e-12, [(cases.M_E, -cases.E_CHARGE, 1.0, True)], pcg_tol=1e-2)
    cfg.pcg_precond = precond
    return Simulation(mesh, cfg, backend=backend)


@pytest.mark.parametrize("precond", [abi.PRECOND_JACOBI, abi.PRECOND_MULTIGRID])
def test_a_smaller_context_leaves_a_larger_one_working(gpu, precond):
    big, small = make(80, gpu), make(64, gpu, precond)
    rng = np.random.default_rng(2)
    for sim in (big, small, big):
        o = make(80 if sim is big else 64, pyoracle.OracleBackend(8))
        rho = 1e-5 * rng.standard_normal(sim.sizes()[0])
        pg, sg = sim.solve_poisson(rho)
        if sim is big or precond == abi.PRECOND_JACOBI:
            po, so = o.solve_poisson(rho)
            assert sg.pcg_iterations == so.pcg_iterations > 0 and np.array_equal(pg, po)
        else:
            assert sg.pcg_residual_l2 <= 1e-2
        o.close()
    big.close()
    small.close()
