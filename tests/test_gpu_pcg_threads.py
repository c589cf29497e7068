"""Contexts that solve at the same time from their own host threads: the
persistent solver kernels of both wait for their own blocks alone, and beside
another context's kernels they give the bits that they give by themselves."""
import threading

import numpy as np
import pytest

from picfoam_gb300 import abi, cases
from picfoam_gb300.simulation import Simulation

pytestmark = pytest.mark.gpu


SIDES = [cases.patch(abi.PATCH_WALL, 2.0 * f) for f in range(6)]


def poisson(n):
    mesh = cases.block_mesh(n, tuple(1e-3 * v for v in n), SIDES)
    cfg = cases.base_config(1e-12, [(cases.M_E, -cases.E_CHARGE, 1.0, True)], pcg_tol=1e-4)
    sim = Simulation(mesh, cfg)
    rho = 1e-5 * np.random.default_rng(n[0]).standard_normal(sim.sizes()[0])
    return sim, lambda: [sim.solve_poisson(rho)[0]]


def steps(n):
    """Particles in motion and the field solve, every run from the same state."""
    case = cases.two_species_3d(n_cells=n, per_cell=10, L=0.05 * n / 64, deposit=abi.DEPOSIT_FIXED_POINT)
    for f in range(6):
        case.mesh.side[f] = SIDES[f]
    sim = cases.build(case)
    start = [sim.get_particles(s) for s in range(2)]

    def run():
        for s in range(2):
            sim.set_particles(s, *start[s])
        sim.set_field(abi.FIELD_PHI, np.zeros(n ** 3))
        sim.initialise_fields()
        sim.step(3)
        return [sim.field(abi.FIELD_PHI)] + [np.sort(sim.get_particles(s)[2], axis=0) for s in range(2)]
    return sim, run


@pytest.mark.parametrize("jobs", [
    [(poisson, (64, 64, 64)), (poisson, (80, 80, 80))],
    [(poisson, (20, 32, 31)), (poisson, (77, 32, 32)), (poisson, (8, 8, 8))],
    [(steps, 40), (poisson, (80, 80, 80)), (steps, 24)]])
def test_solves_side_by_side(gpu, jobs):
    sims, runs = zip(*(make(n) for make, n in jobs))
    alone = [run() for run in runs]
    out, errors = [[] for _ in jobs], []
    gate = threading.Barrier(len(jobs))

    def work(k):
        try:
            gate.wait()
            for _ in range(8):
                out[k].append(runs[k]())
        except Exception as e:     # reported below, from the test's own thread
            errors.append((jobs[k], e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for k in range(len(jobs)):
        for r in out[k]:
            assert all(np.array_equal(a, b) for a, b in zip(r, alone[k]))
    for s in sims:
        s.close()
