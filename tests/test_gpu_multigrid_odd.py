"""Multigrid on odd cell counts and around a plate one cell thick, where some
aggregates are not full: no more inner iterations than the piecewise-constant
prolongation took (its counts, with one more for the plate's rounding), and the
solver's tolerance on the FP64 residual."""
import numpy as np
import pytest

from picfoam_gb300 import abi, cases
from picfoam_gb300.simulation import Simulation

pytestmark = pytest.mark.gpu

KINDS = {"w": lambda f: cases.patch(abi.PATCH_WALL, 3.0 * f), "c": lambda f: cases.patch(abi.PATCH_CYCLIC),
         "z": lambda f: cases.patch(abi.PATCH_WALL, 0.0, abi.PHI_ZERO_GRADIENT)}


@pytest.mark.parametrize("n, sides, plate, most", [
    ((33, 33, 33), "wwwwww", False, 20), ((33, 33, 33), "cczwcc", False, 21), ((33, 33, 33), "zzzzzz", False, 19),
    ((65, 65, 65), "cccccc", False, 27), ((61, 97, 1), "wwwwww", False, 17), ((17, 301, 5), "cczwcc", False, 41),
    ((48, 48, 48), "cccccc", True, 20), ((3, 2, 700), "wwwwww", False, 20)])
def test_iterations(gpu, n, sides, plate, most):
    side = [cases.patch(abi.PATCH_EMPTY) if n[f // 2] == 1 else KINDS[sides[f]](f) for f in range(6)]
    boxes = (((0, 0, 10), (n[0], n[1], 11), cases.patch(abi.PATCH_WALL, 5.0)),) if plate else ()
    mesh = cases.block_mesh(n, tuple(1e-3 * v for v in n), side, boxes=boxes)
    cfg = cases.base_config(1e-12, [(cases.M_E, -cases.E_CHARGE, 1.0, True)], pcg_tol=1e-10)
    cfg.pcg_precond = abi.PRECOND_MULTIGRID
    sim = Simulation(mesh, cfg, backend=gpu)
    cells = sim.sizes()[0]
    rho = 1e-6 * (np.random.default_rng(1).standard_normal(cells) + np.sin(np.linspace(0.0, 5.0, cells)))
    if "w" not in sides and not plate:
        rho -= rho.mean()
    _, st = sim.solve_poisson(rho)
    assert st.pcg_residual_l2 <= 1e-10 and 0 < st.pcg_iterations <= most
    sim.close()
