"""The persistent Poisson PCG when a wait between its blocks runs out: the solve
returns an error, the copies in flight between the blocks of a cluster have
landed (the kernel ends and the context stays usable), and the solves that
follow have the oracle's bits.  Every launch shape whose blocks wait for one
another: clusters of 8, 4 and 2, a chunk per block, several chunks per block."""
import numpy as np
import pytest

import pyoracle
from picfoam_gb300 import abi, cases, native
from picfoam_gb300.simulation import PicError, Simulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(8, 8, 8), (31, 43, 1), (20, 32, 31), (38, 32, 33), (77, 32, 32), (153, 32, 33)])
def test_a_wait_that_runs_out(gpu, n):
    side = [cases.patch(abi.PATCH_EMPTY if n[f // 2] == 1 else abi.PATCH_WALL, 2.0 * f) for f in range(6)]
    mesh = cases.block_mesh(n, tuple(1e-3 * v for v in n), side)
    cfg = cases.base_config(1e-12, [(cases.M_E, -cases.E_CHARGE, 1.0, True)], pcg_tol=1e-6)
    g = Simulation(mesh, cfg, backend=gpu)
    o = Simulation(mesh, cfg, backend=pyoracle.OracleBackend(4))
    look_once = native.load().picgpu_test_pcg_look_once
    rho = 1e-5 * np.random.default_rng(3).standard_normal(g.sizes()[0])
    for _ in range(3):
        assert look_once(g._h, 1) == abi.OK
        for _ in range(2):
            with pytest.raises(PicError) as e:
                g.solve_poisson(rho)
            assert e.value.status == abi.CUDA_ERROR and "waited too long" in str(e.value)
        assert look_once(g._h, 0) == abi.OK
        pg, sg = g.solve_poisson(rho)
        po, so = o.solve_poisson(rho)
        assert sg.pcg_iterations == so.pcg_iterations > 0 and np.array_equal(pg, po)
        rho = rho[::-1].copy()
    g.close()
    o.close()


@pytest.mark.parametrize("learned", [False, True])
def test_a_failed_solve_leaves_field_and_network(gpu, learned):
    case = cases.electrode_box(n_cells=32, per_cell=4, seed=5)
    case.cfg.learned.enabled = 1 if learned else 0
    case.cfg.learned.train_steps = 20
    case.cfg.learned.train_iters = 2
    look_once = native.load().picgpu_test_pcg_look_once
    g = cases.build(case, backend=gpu)
    for _ in range(4):
        before = g.step(1)
    # a field that is not the gradient of the potential at hand
    kinds = (abi.FIELD_E_CELL, abi.FIELD_E_POINT)
    E = [1.5 * g.field(k) for k in kinds]
    for k, v in zip(kinds, E):
        g.set_field(k, v)
    assert look_once(g._h, 1) == abi.OK
    with pytest.raises(PicError) as e:
        g.step(1)
    assert e.value.status == abi.CUDA_ERROR
    assert all(np.array_equal(v, g.field(k)) for k, v in zip(kinds, E))
    assert look_once(g._h, 0) == abi.OK
    after = g.step(1)
    assert not np.array_equal(E[0], g.field(abi.FIELD_E_CELL))
    assert after.learned_samples == before.learned_samples + (1 if learned else 0)
    g.close()
