"""Contexts with different boundaries that live side by side: each keeps its own
patch kinds and potentials whatever is created after it, in the field solve and
the FP64 mover, and gives the bits of a context that is alone."""
import numpy as np
import pytest

from picfoam_gb300 import abi, cases

pytestmark = pytest.mark.gpu


def make(gpu, kind, phi, precond):
    c = cases.two_species_3d(n_cells=10, per_cell=12, precision=abi.PREC_FP64, deposit=abi.DEPOSIT_FIXED_POINT,
                             dt_factor=2.0, L=0.002, pcg_tol=1e-9)
    for f in range(6):
        c.mesh.side[f] = cases.patch(kind, phi * (f + 1))
    c.cfg.pcg_precond = precond
    return cases.build(c, backend=gpu)


def run(sim):
    sim.initialise_fields()
    st = sim.step(3)
    parts = [sim.get_particles(s) for s in range(2)]
    return [st.wall_hits, list(st.n_absorbed)], [sim.field(abi.FIELD_PHI), sim.field(abi.FIELD_E_CELL)] + [
        v for p in parts for v in p]


@pytest.mark.parametrize("precond", [abi.PRECOND_JACOBI, abi.PRECOND_MULTIGRID])
def test_each_context_keeps_its_patches(gpu, precond):
    kinds = [(abi.PATCH_WALL, 3.0), (abi.PATCH_ABSORB, -40.0)]
    alone = []
    for k in kinds:
        with make(gpu, *k, precond) as sim:
            alone.append(run(sim))
    assert alone[0][0] != alone[1][0]       # the boundaries do differ in what they do
    sims = [make(gpu, *k, precond) for k in kinds]
    for sim, (counts, arrays) in zip(sims, alone):
        got, values = run(sim)
        assert got == counts
        assert all(np.array_equal(a, b) for a, b in zip(values, arrays))
        sim.close()
