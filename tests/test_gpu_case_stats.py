"""Per-case sums over particle stores in every order: one case, cases of zero and
one particle, stores in cell order, interleaved and shuffled, counts around the
512 particles of a warp's run.  The sums of the returned particles are the
reference; two FP64 sums of n terms (each good to 3 ulp) differ by at most
(n + 4) 2^-52 of the terms' absolute sum."""
import numpy as np
import pytest

from picfoam_gb300 import abi, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PREC_MIXED, abi.PREC_FP64])
@pytest.mark.parametrize("order", ["cells", "interleaved", "shuffled"])
@pytest.mark.parametrize("counts", [[1], [511, 0, 1, 513], [4096, 4097], [3000, 31, 33, 0, 20000, 7, 500]])
def test_sums_of_the_store(gpu, precision, order, counts):
    n = (4, 2, 3)
    case = cases.swarm_ensemble(n_cases=len(counts), n=n, size=(1e-3, 5e-4, 7.5e-4), counts=np.array(counts),
                                EN_Td=np.full(len(counts), 10.0), seed=5)
    case.cfg.precision = precision
    tet, bary, U = case.particles[0]
    rng = np.random.default_rng(2)
    if order == "shuffled":
        p = rng.permutation(len(tet))
    elif order == "interleaved":
        p = np.argsort(np.arange(len(tet)) % 97, kind="stable")
    else:
        p = np.arange(len(tet))
    case.particles[0] = (tet[p], bary[p], U[p])
    sim = cases.build_ensemble(case)
    out, _ = sim.case_stats(0, len(counts))
    tet, _, U = sim.get_particles(0)
    k = tet // (12 * n[0] * n[1] * n[2])
    for j in range(len(counts)):
        u = U[k == j]
        terms = np.concatenate([np.ones((len(u), 1)), u, (u * u).sum(axis=1)[:, None]], axis=1)
        np.testing.assert_array_less(abs(out[j] - terms.sum(axis=0)),
                                     (len(u) + 4) * 2.0 ** -52 * abs(terms).sum(axis=0) + 1e-300)
        assert out[j, 0] == counts[j]
