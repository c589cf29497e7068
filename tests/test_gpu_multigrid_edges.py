"""Restriction and linear prolongation of the multigrid solve where they can go
wrong: axes of one cell, odd counts, the edges of the 16- and 32-wide tiles,
levels that are and are not a power of two, every kind of side.  The Jacobi
solve of the same charge density (itself bit-equal to the oracle) is the
reference, with the bound of test_gpu_multigrid.py."""
import pytest

from picfoam_gb300 import abi, cases
from test_gpu_multigrid import TOL, close_potentials, solve_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, sides, box", [
    ((17, 16, 15), "wall", False), ((33, 31, 1), "mixed", False), ((1, 40, 37), "wall", False),
    ((513, 1, 1), "wall", False), ((65, 3, 34), "mixed", True), ((34, 18, 20), "cyclic", True),
    ((16, 2, 49), "cyclic", False), ((97, 64, 5), "mixed", False), ((96, 100, 66), "mixed", True)])
def test_matches_jacobi(gpu, n, sides, box):
    def make():
        side = []
        for a in range(3):
            for s in range(2):
                if n[a] == 1:
                    side.append(cases.patch(abi.PATCH_EMPTY))
                elif sides == "cyclic" or (sides == "mixed" and a == 0):
                    side.append(cases.patch(abi.PATCH_CYCLIC))
                elif sides == "mixed" and s == 1:
                    side.append(cases.patch(abi.PATCH_WALL, 0.0, abi.PHI_ZERO_GRADIENT))
                else:
                    side.append(cases.patch(abi.PATCH_ABSORB, 2.0 * a))
        boxes = [((1, 0, 2), (4, 1, 5), cases.patch(abi.PATCH_FLOATING))] if box else []
        mesh = cases.block_mesh(n, tuple(1e-3 * v for v in n), side, boxes=boxes)
        cfg = cases.base_config(1e-12, [(cases.M_E, -cases.E_CHARGE, 1.0, True)])
        return cases.Case("edges", mesh, cfg, {}, [], {})
    pj, stj, pm, stm = solve_both(gpu, make)
    assert stm.pcg_residual_l2 <= TOL
    assert close_potentials(pj, pm, singular=sides == "cyclic") < 1e-7
    assert stm.pcg_iterations <= stj.pcg_iterations
