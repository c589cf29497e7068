"""A capacity error of a graph step belongs to that call: the regular and graph
steps that follow (with a re-sort due) run.  And the prefix sums of the
collision step give the same results whether a block's predecessors answer or
it adds up their items itself."""
import numpy as np
import pytest

from picfoam_gb300 import abi, cases, native
from picfoam_gb300.simulation import PicError

pytestmark = pytest.mark.gpu


def avalanche():
    """6000 electrons of some 1000 eV in a gas so dense that a step adds 1300
    and later 3000 ions: one step fits the room that is kept free, eight do not."""
    case = cases.swarm_ensemble(n_cases=1, n=(4, 4, 4), size=(0.01, 0.01, 0.01), counts=[6000], EN_Td=[0.0],
                                T_e=1000.0, gas_density=1e23, dt=1e-10)
    case.cfg.sort_interval = 1
    for s in range(6):
        case.mesh.side[s].kind = abi.PATCH_CYCLIC
    return case


@pytest.mark.parametrize("after", ["step", "step_graph"])
def test_capacity_error_does_not_stick(gpu, after):
    sim = cases.build_ensemble(avalanche())
    assert sim.step_graph(1, 1).mcc_ionization > 0
    n = sim.count(0)
    with pytest.raises(PicError) as e:
        sim.step_graph(8, 8)
    assert e.value.status == abi.CAPACITY
    sim.set_step_index(5)      # a re-sort is due
    st = sim.step(1) if after == "step" else sim.step_graph(1, 1)
    assert st.mcc_ionization > 0 and sim.count(0) > n
    sim.close()


@pytest.mark.parametrize("n, N", [((16, 16, 16), 20000), ((40, 64, 52), 60000)])
def test_prefix_sums_without_look_back(gpu, n, N):
    runs = []
    for polls in (None, 0):
        case = cases.electron_swarm(nx=n[0], ny=n[1], nz=n[2], N=N, T_e=60.0, size=tuple(1e-3 * v for v in n))
        sim = cases.build(case)
        if polls is not None:
            assert native.load().picgpu_test_scan_polls(sim._h, polls) == abi.OK
        st = [sim.step(1) for _ in range(4)]
        runs.append(([s.mcc_ionization for s in st], [sim.get_particles(s) for s in range(2)]))
        sim.close()
    assert runs[0][0] == runs[1][0] and sum(runs[0][0]) > 0
    for a, b in zip(*(r[1] for r in runs)):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))
