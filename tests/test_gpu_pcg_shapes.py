"""The persistent Poisson PCG over its launch shapes: one block (up to 256
cells), clusters of 8, 4 and 2 blocks per 1024-cell chunk, one block per
chunk, several chunks per block, and the two-kernel iteration beyond; cell
counts at the edges of chunks and shapes.  The oracle runs the same
iteration in the same summation order, so potential, iteration count and
residual are equal bit for bit."""
import numpy as np
import pytest

import pyoracle
from picfoam_gb300 import abi, cases
from picfoam_gb300.simulation import Simulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, sides, tol", [
    ((2, 1, 1), "wall", 1e-10), ((33, 1, 1), "wall", 1e-10), ((256, 1, 1), "wall", 1e-8),
    ((257, 1, 1), "cyclic", 1e-8), ((32, 32, 1), "wall", 1e-10), ((41, 25, 1), "cyclic", 1e-10),
    ((19, 1024, 1), "wall", 1e-2), ((20, 32, 31), "mixed", 1e-10), ((38, 32, 33), "wall", 1e-10),
    ((77, 32, 32), "mixed", 1e-6), ((153, 32, 33), "wall", 1e-4), ((64, 64, 149), "wall", 1e-2),
    ((64, 64, 153), "wall", 1e-2)])
def test_solve_matches_oracle_bit_for_bit(gpu, n, sides, tol):
    side = []
    for a in range(3):
        for _ in range(2):
            if n[a] == 1:
                side.append(cases.patch(abi.PATCH_EMPTY))
            elif sides == "cyclic" or (sides == "mixed" and a == 0):
                side.append(cases.patch(abi.PATCH_CYCLIC))
            else:
                side.append(cases.patch(abi.PATCH_WALL, 3.0 * a))
    box = ()
    if sides == "mixed":
        box = (((2, 2, 2), (5, 4, 6), cases.patch(abi.PATCH_WALL, 10.0)),)
    mesh = cases.block_mesh(n, tuple(1e-3 * v for v in n), side, boxes=box)
    cfg = cases.base_config(1e-12, [(cases.M_E, -cases.E_CHARGE, 1.0, True)], pcg_tol=tol)
    g = Simulation(mesh, cfg, backend=gpu)
    o = Simulation(mesh, cfg, backend=pyoracle.OracleBackend(1))
    rng = np.random.default_rng(5)
    rho = 1e-5 * rng.standard_normal(g.sizes()[0])
    for _ in range(2):      # the second solve: the wait counters were left clean
        pg, sg = g.solve_poisson(rho)
        po, so = o.solve_poisson(rho)
        assert sg.pcg_iterations == so.pcg_iterations > 0
        assert sg.pcg_residual_l2 == so.pcg_residual_l2
        assert np.array_equal(pg, po)
        rho = rho[::-1].copy()
    g.close()
    o.close()
