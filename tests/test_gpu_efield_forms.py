"""The field kernels on equal boxes against the CPU oracle, bit for bit: rows of
one cell, every kind of side and boxes inside, zero fields and values near the
ends of the range (quotients beside the corrected reciprocal)."""
import numpy as np
import pytest

import pyoracle
from picfoam_gb300 import abi, cases
from picfoam_gb300.simulation import Simulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("n, box", [((7, 1, 1), False), ((33, 5, 1), False), ((9, 8, 7), True), ((20, 17, 13), True)])
def test_field_of_a_potential(gpu, precision, n, box):
    side = [cases.patch(abi.PATCH_EMPTY) if n[s // 2] == 1 else
            cases.patch(*[(abi.PATCH_WALL, 0.0), (abi.PATCH_CYCLIC,), (abi.PATCH_ABSORB, 0.0, abi.PHI_ZERO_GRADIENT)][s // 2])
            for s in range(6)]
    boxes = [((2, 2, 2), (4, 3, 5), cases.patch(abi.PATCH_FLOATING))] if box else []
    mesh = cases.block_mesh(n, tuple(1e-3 * (v + 0.1) for v in n), side, boxes=boxes)
    cfg = cases.base_config(1e-12, [(cases.M_E, -cases.E_CHARGE, 1.0, True)], precision=precision)
    g = Simulation(mesh, cfg, backend=gpu)
    cfg.precision = abi.PREC_FP64
    o = Simulation(mesh, cfg, backend=pyoracle.OracleBackend(1))
    rng = np.random.default_rng(4)
    nc = g.sizes()[0]
    # 1e120: near the largest for which the solve's sums of squares are finite
    for scale in (1.0, 0.0, 1e-230, 1e-300, 1e120):
        rho = rng.standard_normal(nc) * 1e-5 * scale
        phi0 = rng.standard_normal(nc) * scale
        for s in (g, o):
            s.solve_poisson(rho, phi0=phi0)
        for f in (abi.FIELD_E_CELL, abi.FIELD_E_POINT):
            np.testing.assert_array_equal(g.field(f), o.field(f), err_msg=f"scale {scale}")
    g.close()
    o.close()
