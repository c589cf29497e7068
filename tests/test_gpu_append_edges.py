"""The per-cell prefix sums and the append of the MCC secondaries where they can
go wrong: one cell, cell counts around the 4096 items of a scan tile, more
tiles than one look-back step of a warp covers, fewer and more staged
candidates than a tile, and one or both secondaries created.  The CPU oracle
draws the same random numbers, so the counts agree but for acceptances that an
ulp decides (the bounds of test_gpu_collisions.py)."""
import numpy as np
import pytest

from picfoam_gb300 import abi, cases
from test_gpu_collisions import run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, N, create", [
    ((1, 1, 1), 300, (1, 1)), ((15, 21, 13), 3000, (1, 0)), ((16, 16, 16), 60000, (1, 1)),
    ((17, 241, 1), 600000, (0, 1)), ((40, 64, 52), 20000, (1, 1))])
def test_secondaries_match_oracle(gpu, oracle_backend, n, N, create):
    case = cases.electron_swarm(nx=n[0], ny=n[1], nz=n[2], N=N, Ez=0.0, T_e=60.0, precision=abi.PREC_FP64,
                                size=tuple(1e-3 * v for v in n))
    for s in range(6):
        case.mesh.side[s].kind = abi.PATCH_CYCLIC
    case.cfg.mcc.create_electron, case.cfg.mcc.create_ion = create
    g, o, sg, so = run_pair(case, gpu, oracle_backend, 6)
    assert sg[0].mcc_candidates == so[0].mcc_candidates > 0
    for s in range(2):
        start = N if s == 0 else 0
        added = o.count(s) - start
        assert (added > 0) == bool(create[s])
        assert abs(g.count(s) - o.count(s)) <= max(2, added // 100)
        # every slot written once: all parcels in the mesh, and as many
        # distinct velocities as parcels
        tet, _, U = g.get_particles(s)
        assert len(U) == g.count(s) == start + create[s] * (g.count(0) - N if create[0] else g.count(1))
        assert len(U) == 0 or (tet.min() >= 0 and tet.max() < 12 * n[0] * n[1] * n[2])
        assert len(np.unique(U, axis=0)) == len(U)
