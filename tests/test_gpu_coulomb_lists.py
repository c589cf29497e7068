"""Cell lists in particle order at the sizes where the sorting network changes
(32 slots per register and lane) and beyond the largest: the pairs of a
Coulomb step are drawn by list position, so one parcel out of order changes
them.  Cells too large to leave, a shuffled store, both pairings; the CPU oracle
draws the same numbers (bounds of test_gpu_collisions.py)."""
import numpy as np
import pytest

from picfoam_gb300 import abi, cases
from test_gpu_collisions import close_fraction, run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairing", [abi.PAIRING_NANBU_YONEMURA, abi.PAIRING_TAKIZUKA_ABE])
@pytest.mark.parametrize("length", [2, 33, 64, 65, 128, 129, 256, 257, 512, 513, 700])
def test_pairs_of_a_shuffled_store(gpu, oracle_backend, pairing, length):
    case = cases.coulomb_thermalisation(n_cells=2, per_cell=length, L=1e6, pairing=pairing)
    tet, bary, U = case.particles[0]
    p = np.random.default_rng(3).permutation(len(tet))
    case.particles[0] = (tet[p], bary[p], U[p])
    g, o, sg, so = run_pair(case, gpu, oracle_backend, 2)
    for a, b in zip(sg, so):
        assert a.coulomb_pairs == b.coulomb_pairs > 0
    assert close_fraction(g, o, 0, 1e-8) > 0.99
