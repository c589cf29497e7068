"""Workloads of the PIC/MCC library for timing: what a picFoam user runs.

listed() are fixed sizes, draw(rng) gives more of the same ranges.  A case is
a dict of plain values with a "kind":

  pic        an electrostatic PIC run: time steps, then the fields (and the
             parcels) read back, as at a write interval of the time loop
  flight     time steps without a field solve (MaxwellSolver none): pushers in
             applied fields
  swarm      electron swarm with null-collision MCC on a background gas
  coulomb    Coulomb thermalisation of an electron population
  dsmc       binary collisions of a neutral gas
  ensemble   many swarm cases in one context, stepped by CUDA graphs
  poisson    one Poisson solve of a given charge density
  unet       loss gradient or prediction of the warm-start network
"""
import ctypes as C
import math

import numpy as np
import torch

from picfoam_gb300 import abi, cases, native
from picfoam_gb300.simulation import Simulation, pinned_empty

EPS0 = cases.EPS0
PUSHERS = {"boris": abi.PUSHER_BORIS, "boris_nr": abi.PUSHER_BORIS_NR, "vay": abi.PUSHER_VAY,
           "hc": abi.PUSHER_HIGUERA_CARY}


def listed():
    return [
        # the plasma oscillation tutorial's size: a 1-D periodic line in the
        # exact FP64 form, a step per call and the phase space read for
        # plotting; the smallest call, where launches and waits count
        dict(name="oscillation_1d_fp64", kind="pic", nx=128, ny=1, nz=1, ppc=200, species=1, precision="fp64",
             precond="jacobi", wall=False, boxes=False, pusher="boris", steps=1, sort=0, parcels=True),
        # a 2-D gap of odd cell counts between fixed-potential reflecting
        # walls: an ordinary interactive run, written with its parcels
        dict(name="gap_2d_mixed", kind="pic", nx=97, ny=61, nz=1, ppc=30, species=2, precision="mixed",
             precond="jacobi", wall=True, boxes=False, pusher="boris", steps=4, sort=10, parcels=True),
        # the exact form in 3-D, odd cell counts, Vay pusher, parcels written
        dict(name="plasma_3d_fp64", kind="pic", nx=25, ny=23, nz=21, ppc=40, species=2, precision="fp64",
             precond="jacobi", wall=True, boxes=False, pusher="vay", steps=4, sort=10, parcels=True),
        # the two-species benchmark cube: 64^3 cells, 50 + 50 parcels per
        # cell, production settings (FP32 store, multigrid, re-sort)
        dict(name="two_species_64_mixed", kind="pic", nx=64, ny=64, nz=64, ppc=50, species=2, precision="mixed",
             precond="multigrid", wall=True, boxes=False, pusher="boris", steps=10, sort=10, parcels=False),
        # the embedded-electrode geometry at an ordinary size, few parcels
        dict(name="electrode_box_48", kind="pic", nx=48, ny=48, nz=48, ppc=8, species=2, precision="mixed",
             precond="multigrid", wall=True, boxes=True, pusher="boris", steps=5, sort=10, parcels=False),
        # the benchmark population in applied E and B, Higuera-Cary pusher:
        # the particle path alone
        dict(name="flight_64_hc", kind="flight", nx=64, ny=64, nz=64, ppc=100, pusher="hc", steps=10, sort=10),
        # electron swarm of the transport-coefficient study: 32x32x256 cells,
        # about 10M electrons, elastic / excitation / ionisation tables
        dict(name="swarm_10m", kind="swarm", nx=32, ny=32, nz=256, ppc=38, td=10.0, precision="mixed", steps=10,
             sort=10),
        # the thermalization tutorial's physics at benchmark size
        dict(name="coulomb_16", kind="coulomb", nx=16, ppc=400, pairing="nanbu", precision="mixed", steps=4),
        # many small swarm cases over a range of reduced fields in one context
        dict(name="ensemble_64", kind="ensemble", cases=64, nx=16, ny=16, nz=32, ppc=16, steps=20, per_graph=10),
        # Poisson solves of a coupled host code: the default preconditioner
        # with electrodes at 64^3, and the multigrid at the largest mesh
        dict(name="poisson_jacobi_64", kind="poisson", nx=64, ny=64, nz=64, precond="jacobi", sides="wall",
             boxes=True, tol=1e-10),
        dict(name="poisson_mg_128", kind="poisson", nx=128, ny=128, nz=128, precond="multigrid", sides="wall",
             boxes=True, tol=1e-10),
        # one training gradient of the Poisson warm-start network
        dict(name="unet_gradient_64", kind="unet", nx=64, ny=64, nz=64, op="gradient"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_pic(rng):
    precision = rng.choice(["mixed", "mixed", "fp64"])
    dim = rng.choice([1, 2, 3])
    if dim == 1:
        n = (_log_int(rng, 16, 2000), 1, 1)
    elif dim == 2:
        n = (_log_int(rng, 12, 200), _log_int(rng, 12, 200), 1)
    else:
        n = tuple(_log_int(rng, 9, 48) for _ in range(3))
    n_c = n[0] * n[1] * n[2]
    most = 4_000_000 if precision == "mixed" else 500_000
    ppc = max(2, min(_log_int(rng, 4, 200), most // (2 * n_c)))
    precond = rng.choice(["jacobi", "multigrid"])
    return dict(kind="pic", nx=n[0], ny=n[1], nz=n[2], ppc=ppc, species=rng.choice([1, 2]), precision=precision,
                precond=precond, wall=rng.choice([True, False]),
                boxes=dim == 3 and min(n) >= 16 and rng.random() < 0.4,
                pusher=rng.choice(["boris", "boris_nr", "vay", "hc"]), steps=rng.choice([1, 2, 4]), sort=10,
                parcels=precond == "jacobi" and rng.random() < 0.5)


def draw(rng):
    kind = rng.choice(["pic", "pic", "flight", "swarm", "coulomb", "dsmc", "ensemble", "poisson", "poisson", "unet"])
    if kind == "pic":
        return _draw_pic(rng)
    if kind == "flight":
        n = [_log_int(rng, 8, 64) for _ in range(3)]
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], ppc=_log_int(rng, 5, 100),
                    pusher=rng.choice(["boris", "boris_nr", "vay", "hc"]), steps=rng.choice([5, 10]), sort=10)
    if kind == "swarm":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        n = [_log_int(rng, 6, 24), _log_int(rng, 6, 24), _log_int(rng, 16, 200)]
        most = 4_000_000 if precision == "mixed" else 400_000
        ppc = max(2, min(_log_int(rng, 5, 60), most // (n[0] * n[1] * n[2])))
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], ppc=ppc, td=round(math.exp(rng.uniform(2.3, 4.6)), 2),
                    precision=precision, steps=rng.choice([2, 5]), sort=10)
    if kind == "coulomb":
        return dict(kind=kind, nx=rng.randint(5, 14), ppc=_log_int(rng, 30, 400),
                    pairing=rng.choice(["nanbu", "takizuka"]), precision=rng.choice(["mixed", "fp64"]),
                    steps=rng.choice([1, 2, 3]))
    if kind == "dsmc":
        return dict(kind=kind, nx=rng.randint(6, 24), ppc=_log_int(rng, 8, 60),
                    precision=rng.choice(["mixed", "fp64"]), xs=rng.choice(["hs", "vhs"]), steps=rng.choice([1, 2]))
    if kind == "ensemble":
        per = rng.choice([5, 10])
        return dict(kind=kind, cases=rng.randint(3, 40), nx=_log_int(rng, 6, 16), ny=_log_int(rng, 6, 16),
                    nz=_log_int(rng, 8, 40), ppc=_log_int(rng, 4, 30), steps=2 * per, per_graph=per)
    if kind == "poisson":
        sides = rng.choice(["wall", "cyclic", "mixed"])
        n = [_log_int(rng, 13, 80) for _ in range(3)]
        if rng.random() < 0.3:
            n = [_log_int(rng, 30, 300), _log_int(rng, 30, 300), 1]
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], precond=rng.choice(["jacobi", "multigrid"]), sides=sides,
                    boxes=min(n) >= 16 and rng.random() < 0.4, tol=1e-10)
    m = [rng.choice([16, 32, 48, 64]) for _ in range(2)]
    return dict(kind="unet", nx=m[0], ny=m[1], nz=32, op=rng.choice(["gradient", "forward"]))


# ------------------------------------------------------------- set-up -----
def _sides(wall, n):
    """Fixed-potential specular walls or periodic sides; empty across one cell."""
    out = []
    for a in range(3):
        for k in range(2):
            if n[a] == 1:
                out.append(cases.patch(abi.PATCH_EMPTY))
            elif wall:
                out.append(cases.patch(abi.PATCH_WALL, 0.0))
            else:
                out.append(cases.patch(abi.PATCH_CYCLIC))
    return out


def _boxes(n):
    """Two reflecting electrodes at 100 V and 0 V inside the block."""
    e = [max(v // 12, 1) for v in n]
    boxes = []
    for lo, phi in (([v // 4 for v in n], 100.0), ([(2 * v) // 3 for v in n], 0.0)):
        boxes.append((tuple(lo), tuple(l + k for l, k in zip(lo, e)), cases.patch(abi.PATCH_WALL, phi)))
    return boxes


def _writes_parcels(case):
    return bool(case.get("parcels")) or case["kind"] in ("coulomb", "dsmc")


def _context(case, seed):
    """The library context with its parcels placed on the device."""
    kind = case["kind"]
    n = (case["nx"], case.get("ny", case["nx"]), case.get("nz", case["nx"]))
    mixed = case.get("precision", "mixed") == "mixed"
    prec = abi.PREC_MIXED if mixed else abi.PREC_FP64
    keep = []
    if kind in ("pic", "flight"):
        density, T = 1e15, (2.0, 0.03)
        h = 0.05 / 64
        length = tuple(h * v for v in n)
        wall = case.get("wall", False)
        mesh = cases.block_mesh(n, length, _sides(wall, n), boxes=_boxes(n) if case.get("boxes") else ())
        weight = density * h ** 3 / case["ppc"]
        dt = 0.1 / cases.plasma_frequency(density)
        species = [(cases.M_E, -cases.E_CHARGE, weight, True), (cases.M_AR, cases.E_CHARGE, weight, True)]
        species = species[:case.get("species", 1)]
        cfg = cases.base_config(dt, species, pusher=PUSHERS[case["pusher"]], precision=prec, B=(0.0, 0.0, 0.01),
                                deposit=abi.DEPOSIT_FIXED_POINT, seed=seed)
        if kind == "flight":
            cfg.maxwell_solver = abi.MAXWELL_NONE
            for a, e in enumerate((0.0, 200.0, 1000.0)):
                cfg.E_applied[a] = e
        elif len(species) == 1:
            cfg.space_charge = cases.E_CHARGE * density   # immobile neutralising background
        if case.get("precond") == "multigrid":
            cfg.pcg_precond = abi.PRECOND_MULTIGRID
        init = cases.init_config(abi.INIT_EQUIPARTITION, seed=seed, number_density=(density,) * len(species),
                                 temperature=T[:len(species)], electron_volt=True, solve_fields=kind == "pic",
                                 leapfrog=kind == "pic")
    elif kind == "swarm":
        size = tuple(v * 0.02 / 32 for v in n)
        gas = 1e21
        one = cases.electron_swarm(nx=n[0], ny=n[1], nz=n[2], N=1, Ez=case["td"] * 1e-21 * gas, gas_density=gas,
                                   seed=seed, precision=prec, size=size)
        for s in range(6):
            one.mesh.side[s] = cases.patch(abi.PATCH_CYCLIC)
        mesh, cfg, keep = one.mesh, one.cfg, one.keepalive
        n_c = n[0] * n[1] * n[2]
        init = cases.init_config(abi.INIT_EQUIPARTITION, seed=seed,
                                 number_density=(case["ppc"] * n_c / (size[0] * size[1] * size[2]), 0.0),
                                 temperature=(2.0, 0.03), electron_volt=True)
    elif kind == "coulomb":
        one = cases.coulomb_thermalisation(n_cells=n[0], per_cell=1, n=1e18, precision=prec, seed=seed,
                                           pairing=abi.PAIRING_NANBU_YONEMURA if case["pairing"] == "nanbu"
                                           else abi.PAIRING_TAKIZUKA_ABE)
        mesh, cfg = one.mesh, one.cfg
        cfg.species[0].weight = 1e18 * 1e-4 ** 3 / (n[0] ** 3 * case["ppc"])
    else:  # dsmc
        one = cases.neutral_gas(n_cells=n[0], per_cell=1, L=1e-4 * n[0], precision=prec, seed=seed,
                                cross_section=abi.XS_HARD_SPHERE if case["xs"] == "hs"
                                else abi.XS_VARIABLE_HARD_SPHERE, omega=0.5 if case["xs"] == "hs" else 0.81)
        mesh, cfg = one.mesh, one.cfg
        cfg.species[0].weight = 1e21 * 1e-12 / case["ppc"]
    cfg.sort_interval = case.get("sort", 0)
    sim = Simulation(mesh, cfg, keepalive=keep)
    if not _writes_parcels(case):
        sim.initialise(init)     # picInitialise on the device
        return sim
    # a population placed by the host program: the same count in every cell
    rng = np.random.Generator(np.random.Philox(seed))
    n_cells = sim.sizes()[0]
    speed = {"coulomb": [(2.0, 1.0, 1.0)], "dsmc": [(0.0259,) * 3]}.get(kind, [(2.0,) * 3, (0.03,) * 3])
    for sp in range(cfg.n_species):
        tet, bary = cases.uniform_in_cells(rng, np.arange(n_cells), case["ppc"])
        U = rng.standard_normal((tet.size, 3))
        U *= [cases.thermal_speed(T, cfg.species[sp].mass) for T in speed[sp]]
        sim.set_particles(sp, tet, bary, U)
    sim.initialise_fields()
    return sim


def _poisson_mesh(case):
    n = (case["nx"], case["ny"], case["nz"])
    if case["sides"] == "cyclic":
        sides = _sides(False, n)
    else:
        sides = _sides(True, n)
        if case["sides"] == "mixed":   # periodic along x, insulating at -y, a biased electrode at +y
            sides[0] = sides[1] = cases.patch(abi.PATCH_CYCLIC)
            sides[2] = cases.patch(abi.PATCH_WALL, 0.0, abi.PHI_ZERO_GRADIENT)
            sides[3] = cases.patch(abi.PATCH_WALL, 50.0)
    return n, sides, _boxes(n) if case["boxes"] else ()


def _charge(case, n_cells, seed):
    """A plasma's charge density per active cell: shot noise of 50 + 50
    parcels per cell at 1e15 m^-3 over a sheath-scale imbalance."""
    rng = np.random.Generator(np.random.Philox(seed))
    noise = rng.standard_normal(n_cells) * math.sqrt(2.0 / 50.0)
    slow = np.sin(np.linspace(0.0, 3.0, n_cells) + rng.random() * 6.0)
    return cases.E_CHARGE * 1e15 * (noise + 0.05 * slow)


class State:
    net = None

    def __del__(self):
        if self.net:
            self.lib.picgpu_unet_destroy(self.net)


def prepare(case, seed):
    s = State()
    s.case = case
    kind = case["kind"]
    if kind == "unet":
        lib = native.load()
        X, Y, Z = case["nx"], case["ny"], case["nz"]
        V = X * Y * Z
        s.lib, s.net = lib, C.c_void_p()
        assert lib.picgpu_unet_create(X, Y, Z, seed, C.byref(s.net)) == abi.OK
        rng = np.random.Generator(np.random.Philox(seed))
        mask = np.ones((Z, Y, X), np.float32)
        mask[Z // 4:Z // 4 + 2, Y // 4:Y // 4 + 2, X // 4:X // 4 + 2] = 0.0
        r = rng.standard_normal((Z, Y, X), dtype=np.float32) * mask
        s.inp = np.ascontiguousarray(np.stack([r, mask], axis=-1))
        s.target = np.ascontiguousarray(rng.standard_normal((Z, Y, X), dtype=np.float32) * mask)
        s.mask = mask
        s.weights = np.zeros(lib.picgpu_unet_param_count(), np.float32)
        s.grad = np.zeros_like(s.weights)
        s.out = np.zeros(V, np.float32)
        s.loss = C.c_double()
        return s
    if kind == "ensemble":
        n_cases, n = case["cases"], (case["nx"], case["ny"], case["nz"])
        rng = np.random.Generator(np.random.Philox(seed))
        mean = case["ppc"] * n[0] * n[1] * n[2]
        counts = np.maximum(1, mean * np.exp(rng.uniform(-0.7, 0.7, n_cases))).astype(np.int64)
        one = cases.swarm_ensemble(n_cases=n_cases, n=n, size=tuple(v * 0.01 / 16 for v in n), counts=counts,
                                   EN_Td=np.logspace(1.0, 2.0, n_cases), seed=seed)
        for a in range(6):
            one.mesh.side[a] = cases.patch(abi.PATCH_CYCLIC)
        s.sim = cases.build_ensemble(one)
        return s
    if kind == "poisson":
        n, sides, boxes = _poisson_mesh(case)
        mesh = cases.block_mesh(n, tuple(0.1 * v / 128 for v in n), sides, boxes=boxes)
        cfg = cases.base_config(1e-12, [(cases.M_E, -cases.E_CHARGE, 1.0, True)], pcg_tol=case["tol"], seed=seed)
        if case["precond"] == "multigrid":
            cfg.pcg_precond = abi.PRECOND_MULTIGRID
        s.sim = Simulation(mesh, cfg)
        s.rho = _charge(case, s.sim.sizes()[0], seed)
        return s
    s.sim = _context(case, seed)
    n_cells = s.sim.sizes()[0]
    # page-locked buffers of the write interval
    s.phi, s.E, s.rho = pinned_empty(n_cells, np.float64), pinned_empty((n_cells, 3), np.float64), \
        pinned_empty(n_cells, np.float64)
    s.rows = []
    if _writes_parcels(case):
        for sp in range(s.sim.cfg.n_species):
            k = s.sim.count(sp)
            s.rows.append((pinned_empty(k, np.int32), pinned_empty((k, 3), np.float64),
                           pinned_empty((k, 3), np.float64)))
    return s


def _fields(s, which):
    def ptr(a):
        return a.ctypes.data_as(C.POINTER(C.c_double))
    f = s.sim.lib.picgpu_get_fields
    st = f(s.sim._h, ptr(s.phi) if which == "all" else None, ptr(s.E) if which == "all" else None, ptr(s.rho))
    assert st == abi.OK
    return [s.phi, s.E, s.rho] if which == "all" else [s.rho]


def _f32p(a):
    return a.ctypes.data_as(C.POINTER(C.c_float))


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "unet":
        if case["op"] == "forward":
            assert s.lib.picgpu_unet_forward(s.net, _f32p(s.inp), _f32p(s.out)) == abi.OK
            return s.out
        assert s.lib.picgpu_unet_gradients(s.net, _f32p(s.inp), _f32p(s.target), _f32p(s.mask), _f32p(s.grad),
                                           C.byref(s.loss)) == abi.OK
        return [s.grad, s.loss.value]
    if kind == "poisson":
        phi = s.sim.solve_poisson(s.rho)[0]
        # a fully periodic potential is defined up to a constant
        return phi - phi.mean() if case["sides"] == "cyclic" and not case["boxes"] else phi
    if kind == "ensemble":
        s.sim.step_graph(case["steps"], case["per_graph"])
        stats, ionisations = s.sim.case_stats(0, case["cases"])
        return [stats, ionisations, s.sim.field(abi.FIELD_RHO)]
    s.sim.step(case["steps"])
    out = _fields(s, "all" if kind == "pic" else "rho")
    for sp, rows in enumerate(s.rows):
        out.extend(s.sim.get_particles(sp, out=rows))
    if case.get("precond") == "multigrid":
        # the potential is accurate to the solver's tolerance, and up to a
        # constant in a periodic box: kept in single precision
        if not case["wall"] and not case["boxes"]:
            s.phi -= s.phi.mean()
        return [a.astype(np.float32) for a in out]
    return out


def work(case):
    kind = case["kind"]
    n_c = case["nx"] * case.get("ny", case["nx"]) * case.get("nz", case["nx"])
    if kind == "unet":
        V = n_c
        pairs = [(2, 16, 1), (16, 16, 1), (16, 32, 8), (32, 32, 8), (32, 64, 64), (64, 64, 64), (96, 32, 8),
                 (32, 32, 8), (48, 16, 1), (16, 16, 1), (16, 1, 1)]
        flops = sum(2.0 * 27 * a * b * (V // d) for a, b, d in pairs)
        weights = 4.0 * 27 * sum(a * b for a, b, _ in pairs)
        if case["op"] == "forward":
            return {"bytes": 12.0 * V + weights, "flops": flops}
        return {"bytes": 16.0 * V + 2 * weights, "flops": 3 * flops - 2.0 * 27 * 2 * 16 * V}
    if kind == "poisson":
        # charge in, potential out, a few operations per cell
        return {"bytes": 16.0 * n_c, "flops": 20.0 * n_c}
    steps = case["steps"]
    parcels = n_c * case["ppc"] * case.get("species", 1) * case.get("cases", 1)
    cells = n_c * case.get("cases", 1)
    row = 56.0 if case.get("precision", "mixed") == "mixed" else 104.0
    per_cell = 56.0 if kind == "pic" else 8.0
    return {"bytes": steps * (row * parcels + per_cell * cells), "flops": steps * 100.0 * parcels}


# -------------------------------------------------- 64-bit evaluations -----
def _exact_poisson(case, seed):
    """-laplacian(phi) = rho / eps0 on the block's cells (two-point fluxes,
    half-cell distance to a fixed potential), conjugate gradients in 64 bits."""
    n, sides, boxes = _poisson_mesh(case)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    shape = (n[2], n[1], n[0])
    h = 0.1 / 128
    active = torch.ones(shape, dtype=torch.float64, device=dev)
    wall_phi = torch.full(shape, float("nan"), dtype=torch.float64, device=dev)
    for lo, hi, p in boxes:
        sl = tuple(slice(lo[a], hi[a]) for a in (2, 1, 0))
        active[sl] = 0.0
        wall_phi[sl] = p.phi
    diag = torch.zeros_like(active)
    rhs = torch.zeros_like(active)
    links = []
    for a in range(3):
        if n[a] == 1:
            continue
        d = 2 - a
        for side in (0, 1):
            shift = 1 if side == 0 else -1
            other = torch.roll(active, shift, d)
            phi_o = torch.roll(wall_phi, shift, d)
            edge = torch.zeros(shape, dtype=torch.bool, device=dev)
            idx = [slice(None)] * 3
            idx[d] = 0 if side == 0 else n[a] - 1
            edge[tuple(idx)] = True
            p = sides[2 * a + side]
            if p.kind != abi.PATCH_CYCLIC:
                fixed = p.phi_bc == abi.PHI_FIXED_VALUE
                other = torch.where(edge, torch.zeros_like(other), other)
                phi_o = torch.where(edge, torch.full_like(phi_o, p.phi if fixed else float("nan")), phi_o)
            wall = ((other == 0) & (active > 0) & ~torch.isnan(phi_o)).double()
            diag += h * (other * active + 2.0 * wall)
            rhs += 2.0 * h * wall * torch.nan_to_num(phi_o)
            links.append((d, shift, other * active * h))
    on = active.reshape(-1) > 0
    rho = torch.from_numpy(_charge(case, int(on.sum()), seed)).to(dev)
    full = torch.zeros(on.numel(), dtype=torch.float64, device=dev)
    full[on] = rho / EPS0 * h ** 3
    rhs = rhs + full.reshape(shape)
    singular = case["sides"] == "cyclic" and not boxes
    if singular:
        rhs = rhs - rhs.mean()

    def A(x):
        y = diag * x
        for d, shift, w in links:
            y = y - w * torch.roll(x, shift, d)
        return y

    inv = torch.where(diag > 0, 1.0 / diag, torch.zeros_like(diag))
    x = torch.zeros_like(rhs)
    for _ in range(2):    # restarted once: the true residual at rounding level
        r = rhs - A(x)
        z = inv * r
        p = z.clone()
        rz = (r * z).sum()
        for it in range(4000):
            q = A(p)
            alpha = rz / (p * q).sum()
            x += alpha * p
            r -= alpha * q
            if it % 50 == 49 and float(r.norm()) <= 1e-14 * float(rhs.norm()):
                break
            z = inv * r
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
    if singular:
        x = x - x.mean()
    return x.reshape(-1)[on]


def _exact_unet(case, seed):
    """The network of picgpu_learned.h in 64 bits from the handle's weights."""
    s = prepare(case, seed)
    s.lib.picgpu_unet_get_weights(s.net, _f32p(s.weights))
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    pairs = [(2, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (32, 32), (48, 16), (16, 16),
             (16, 1)]
    w, off = [], 0
    for ci, co in pairs:
        k = 27 * ci * co
        w.append(torch.from_numpy(s.weights[off:off + k].astype(np.float64)).to(dev).requires_grad_(True))
        off += k
    inp = torch.from_numpy(s.inp).to(dev).double().permute(3, 0, 1, 2)[None]

    def conv(x, l):
        ci, co = pairs[l]
        k = w[l].reshape(27, co, ci)
        xp = torch.nn.functional.pad(x, (1,) * 6)
        out = 0.0
        for t in range(27):
            dz, dy, dx = t // 9, (t // 3) % 3, t % 3
            part = xp[:, :, dz:dz + x.shape[2], dy:dy + x.shape[3], dx:dx + x.shape[4]]
            out = out + torch.einsum("oc,bczyx->bozyx", k[t], part)
        return out

    F = torch.nn.functional
    a2 = F.relu(conv(F.relu(conv(inp, 0)), 1))
    a4 = F.relu(conv(F.relu(conv(F.avg_pool3d(a2, 2), 2)), 3))
    a6 = F.relu(conv(F.relu(conv(F.avg_pool3d(a4, 2), 4)), 5))
    up = torch.cat([F.interpolate(a6, scale_factor=2), a4], 1)
    a8 = F.relu(conv(F.relu(conv(up, 6)), 7))
    up = torch.cat([F.interpolate(a8, scale_factor=2), a2], 1)
    out = conv(F.relu(conv(F.relu(conv(up, 8)), 9)), 10)[0, 0]
    if case["op"] == "forward":
        return out.detach().reshape(-1)
    m = torch.from_numpy(s.mask).to(dev).double()
    t = torch.from_numpy(s.target).to(dev).double()
    loss = (m * (out - t) ** 2).sum() / (m * t * t).sum()
    loss.backward()
    return [torch.cat([v.grad for v in w]), float(loss)]


def exact(case, seed):
    if case["kind"] == "poisson":
        return _exact_poisson(case, seed)
    if case["kind"] == "unet":
        return _exact_unet(case, seed)
    return None
