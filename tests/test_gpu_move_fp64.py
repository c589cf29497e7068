"""The FP64 mover where its passes can go wrong: fewer particles than lanes,
chunks that end inside a row, several rounds per warp, removed slots, and
tracks whose first face is decided by equal or nearly equal quotients (starts on
faces, edges and corners of tets, zero and denormal velocities, displacements
along a face).  Particles, charge and counters are the CPU oracle's bit for bit
(fixed-point deposit)."""
import numpy as np
import pytest

from picfoam_gb300 import abi, cases
from test_gpu_parity import assert_fields_equal, assert_particles_equal, pair

pytestmark = pytest.mark.gpu


def make(n, N, dims):
    kinds = [abi.PATCH_WALL, abi.PATCH_ABSORB, abi.PATCH_CYCLIC, abi.PATCH_CYCLIC, abi.PATCH_WALL, abi.PATCH_FLOATING]
    side = [cases.patch(abi.PATCH_EMPTY if s // 2 >= dims else kinds[s]) for s in range(6)]
    h = 1e-3
    mesh = cases.block_mesh(n, tuple(h * v for v in n), side)
    dt = 1e-10
    cfg = cases.base_config(dt, [(cases.M_E, -cases.E_CHARGE, 100.0, True), (cases.M_AR, 0.0, 100.0, True)],
                            deposit=abi.DEPOSIT_FIXED_POINT, maxwell=abi.MAXWELL_NONE, E_applied=(2e3, -1e3, 5e2),
                            B=(0.0, 0.01, 0.02))
    rng = np.random.Generator(np.random.Philox(11))
    parts = {}
    for s in range(2):
        tet = rng.integers(0, 12 * n[0] * n[1] * n[2], N).astype(np.int32)
        # a third inside, the rest on faces, edges and corners or a hair off them
        grid = np.array([0.0, 0.0, 0.25, 0.5, 1.0 / 3.0, 1e-17, 1e-300])
        u = np.sort(rng.random((N, 3)), axis=1)
        b = np.stack([u[:, 0], u[:, 1] - u[:, 0], u[:, 2] - u[:, 1]], axis=1)
        on = rng.random(N) < 0.67
        g = grid[rng.integers(0, len(grid), (N, 3))]
        b[on] = np.where(g.sum(axis=1, keepdims=True) <= 1.0, g, 0.25)[on]
        # cells per step: 0, a denormal, 0.3 (thermal), up to 6; some along one axis
        U = rng.standard_normal((N, 3)) * 0.3 * h / dt
        k = rng.integers(0, 8, N)
        U[k == 0] = 0.0
        U[k == 1] *= 1e-305 * dt / h
        U[k == 2] *= 10.0
        U[k == 3, 1:] = 0.0
        U[k == 4] = np.array([0.5, 0.5, -0.5]) * h / dt
        if dims < 3:
            U[:, dims:] *= 0.1
        parts[s] = (tet, b, U)
    return cases.Case("move_fp64", mesh, cfg, parts, [], {})


@pytest.mark.parametrize("n, dims, N", [((5, 4, 3), 3, 1), ((5, 4, 3), 3, 31), ((5, 4, 3), 3, 33), ((9, 1, 1), 1, 129),
                                        ((7, 6, 1), 2, 4000), ((5, 4, 3), 3, 77777), ((31, 30, 29), 3, 1000003)])
def test_bit_equal_to_the_oracle(gpu, oracle_backend, n, dims, N):
    g, o = pair(make(n, N, dims), gpu, oracle_backend, nthreads=8 if N > 1000 else 1)
    for _ in range(2 if N > 100000 else 4):
        sg, so = g.step(1), o.step(1)
        assert sg.tet_steps == so.tet_steps and sg.face_crossings == so.face_crossings
        assert list(sg.n_absorbed) == list(so.n_absorbed) and list(sg.n_particles) == list(so.n_particles)
        assert_particles_equal(g, o, 2)
        assert_fields_equal(g, o)
