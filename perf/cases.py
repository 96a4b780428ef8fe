"""Performance cases: the work a program has this framework do, from one step of a small network
under a user's hand to large Lennard-Jones systems, ensembles, scoring and parameter fits.

``listed()`` gives the fixed cases, ``draw(rng)`` one more of the same ranges, ``prepare`` the state
a program keeps (a set-up handle, or device tensors), ``run`` one pass through the public entry
points, ``work`` the bytes and operations a pass cannot do without, and ``exact`` the outputs of
the first pass in 64-bit arithmetic, written here from the force laws alone.

Families (``case["kind"]``):

* ``network``  -- elastic Calpha network with steric contacts and viscosity (``SpringNetwork``);
* ``lj``       -- dense beads: springs, Lennard-Jones (three forms), Coulomb (two dielectrics);
* ``membrane`` -- bead globule in the IMPALA membrane, some segments held as rigid bodies;
* ``docking``  -- mobile ligand on a static receptor: Lennard-Jones, Coulomb, hydrophobic pairs, a
  potential map and the probe;
* ``score``    -- energies and forces of a conformation handed in from outside;
* ``ensemble`` -- many independent networks in one handle;
* ``fit``      -- one training step of spring parameters (and charges) through the adjoint;
* ``direct``   -- nonbonded forces on the caller's own device buffers, without a handle.
"""

import ctypes
import math

import numpy as np
import torch

from biospring_gb300 import SpringNetwork, capi
from biospring_gb300 import workloads as W
from biospring_gb300.fit import SpringFitLoss

KCAL = 4.1840
BEAD_DENSITY = 0.0244  # beads per cubic A of the dense systems (100,000 in a cube of 160 A)


# ---------------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------------

def listed():
    return [
        # haptic steering of a small protein: every frame sends the hand's forces, advances one
        # step and draws the positions -- latency and launches are all there is
        dict(name="network_300_interactive", kind="network", n=300, steps=1, pull=1),
        # the 2,000-residue network run for a trajectory: 100 steps between two saved states
        dict(name="network_2000", kind="network", n=2000, steps=100, pull=0),
        # a solvated-bead patch of odd size with several bead types, 8-6 form, constant dielectric
        dict(name="lj_5003_types", kind="lj", n=5003, steps=20, mode=2, dielectric=0, types=7, charged=0.3, cutoff=10.0,
             skin=0.5),
        # the benchmark system: 100,000 beads, 12-6, eps = 4r, 0.1 A list skin
        dict(name="lj_100000", kind="lj", n=100000, steps=20, mode=1, dielectric=1, types=1, charged=0.2, cutoff=12.0,
             skin=0.1),
        # the largest single system: three times the benchmark's beads, ragged count
        dict(name="lj_300007", kind="lj", n=300007, steps=10, mode=1, dielectric=0, types=1, charged=0.2, cutoff=12.0,
             skin=0.5),
        # 20,000 beads in the membrane with four rigid domains of 500
        dict(name="membrane_20000_bodies", kind="membrane", n=20000, steps=50, bodies=4),
        # flexible ligand on a frozen receptor, every pair term, a potential map and the probe on
        dict(name="docking_6007", kind="docking", n=6007, steps=20, grid=33, static=0.7),
        # one conformation scored for an outside sampler: new lists, forces and energies
        dict(name="score_12000", kind="score", n=12000, mode=1, dielectric=0, types=5, charged=0.2, cutoff=12.0,
             skin=0.5),
        # 64 independent networks of 200 to 20,000 particles, launch shape picked by the autotuner
        dict(name="ensemble_64", kind="ensemble", systems=64, lo=200, hi=20000, steps=20, tune=1),
        # one training step of 10,000 particles' springs over 200 steps of dynamics
        dict(name="fit_10000", kind="fit", n=10000, steps=200, checkpoint=20, charges=0),
        # springs and charges of a smaller network fitted together, checkpoints that do not divide
        dict(name="fit_1999_charges", kind="fit", n=1999, steps=60, checkpoint=25, charges=1),
        # nonbonded forces on buffers the caller owns, inside a frame budget
        dict(name="direct_4001", kind="direct", n=4001, mode=1, dielectric=0, cutoff=12.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["network", "network", "lj", "lj", "membrane", "docking", "score", "ensemble", "fit", "direct"])
    if kind == "network":
        pull = rng.randint(0, 1)
        return dict(kind=kind, n=_log_int(rng, 300, 20000), steps=rng.randint(1, 4) if pull else _log_int(rng, 10, 200),
                    pull=pull)
    if kind == "lj":
        return dict(kind=kind, n=_log_int(rng, 2000, 250000), steps=rng.choice([1, 10, 10, 17, 20]),
                    mode=rng.choice([1, 1, 2, 3]), dielectric=rng.randint(0, 1), types=rng.choice([1, 1, 4, 9]),
                    charged=rng.choice([0.1, 0.2, 0.5]), cutoff=rng.choice([9.0, 10.0, 12.0]),
                    skin=rng.choice([0.1, 0.5, 1.0]))
    if kind == "membrane":
        return dict(kind=kind, n=_log_int(rng, 4000, 40000), steps=rng.choice([10, 25, 50]), bodies=rng.choice([0, 2, 4]))
    if kind == "docking":
        return dict(kind=kind, n=_log_int(rng, 1500, 15000), steps=rng.choice([5, 10, 20]), grid=rng.choice([17, 33, 48]),
                    static=rng.choice([0.5, 0.7, 0.9]))
    if kind == "score":
        return dict(kind=kind, n=_log_int(rng, 1000, 60000), mode=rng.choice([1, 2, 3]), dielectric=rng.randint(0, 1),
                    types=rng.choice([1, 5]), charged=0.2, cutoff=rng.choice([9.0, 12.0]), skin=0.5)
    if kind == "ensemble":
        return dict(kind=kind, systems=rng.randint(8, 64), lo=200, hi=_log_int(rng, 1000, 20000),
                    steps=rng.choice([10, 20, 25]), tune=1)
    if kind == "fit":
        charges = rng.randint(0, 1)
        return dict(kind=kind, n=_log_int(rng, 500, 3000 if charges else 10000), steps=rng.randint(20, 60 if charges else 200),
                    checkpoint=rng.choice([10, 20, 25]), charges=charges)
    return dict(kind=kind, n=_log_int(rng, 200, 16384), mode=rng.randint(0, 3), dielectric=rng.randint(0, 1),
                cutoff=rng.choice([9.0, 12.0]))


# ---------------------------------------------------------------------------------------------
# systems (host arrays, from the case and the seed alone)
# ---------------------------------------------------------------------------------------------

def _thermal(rng, n, mass):
    """Velocities at 300 K (A/fs), as a restart file holds them."""
    return (rng.standard_normal((n, 3)) * np.sqrt(2.494e-4 / mass)[:, None]).astype(np.float32)


def _beads(n, rng):
    """n beads at BEAD_DENSITY in a cube, a jittered lattice in random order (nearest distance
    about 3 A, as a relaxed bead model has it)."""
    a = BEAD_DENSITY ** (-1.0 / 3.0)
    m = int(math.ceil(n ** (1.0 / 3.0)))
    cells = np.arange(m * m * m)
    cells = cells[np.sort(rng.permutation(m * m * m)[:n])]
    x = np.stack([cells % m, cells // m % m, cells // (m * m)], axis=1) * a
    x = x + rng.uniform(-0.2, 0.2, size=(n, 3))
    return x[rng.permutation(n)].astype(np.float32)


def _springs(x, cutoff, rng):
    ij = W.pairs_within(x, cutoff)
    d = np.linalg.norm(x[ij[:, 1]].astype(np.float64) - x[ij[:, 0]], axis=1)
    r0 = (d + rng.normal(0.0, 0.05, d.shape)).astype(np.float32)
    return ij, r0


def _lj_types(s, n, types, rng):
    if types <= 1:
        s["radius"] = np.full(n, 3.5, np.float32)
        s["epsilon"] = np.full(n, 0.2 * KCAL, np.float32)
    else:
        t = rng.integers(0, types, n)
        s["radius"] = np.linspace(3.1, 3.8, types).astype(np.float32)[t]
        s["epsilon"] = (np.linspace(0.1, 0.3, types) * KCAL).astype(np.float32)[t]


def _charges(n, fraction, rng):
    """A fraction of the beads charged, two negative to one positive (an acidic assembly), so that
    the electrostatic energy is not a small difference of large sums."""
    q = np.zeros(n, np.float32)
    ids = rng.permutation(n)[: int(fraction * n)]
    q[ids] = -1.0
    q[ids[::3]] = 1.0
    return q


def _network_system(n, seed, structure=1):
    """The chain and its bonds belong to the structure; rest lengths, displacements and velocities
    to the seed."""
    rng = np.random.default_rng([seed, n, structure])
    x = W.ca_chain(n, structure)
    ij, r0 = _springs(x, 10.0, rng)
    mass = np.full(n, 110.0, np.float32)
    return dict(xyz=(x + rng.normal(0.0, 0.15, x.shape)).astype(np.float32), ij=ij, r0=r0,
                k=np.full(ij.shape[0], KCAL, np.float32), mass=mass, vel=_thermal(rng, n, mass),
                cfg=dict(timestep=0.01, spring_enable=1, steric_enable=1, steric_cutoff=8.0, steric_mode=0,
                         viscosity_enable=1, viscosity_value=1.0, rebuild_every=10, list_skin=1.0))


def _lj_system(c, seed, springs=True):
    rng = np.random.default_rng([seed, c["n"]])
    n = c["n"]
    x = _beads(n, rng)
    mass = np.full(n, 72.0, np.float32)
    s = dict(xyz=x, mass=mass, vel=_thermal(rng, n, mass), charge=_charges(n, c["charged"], rng))
    _lj_types(s, n, c["types"], rng)
    s["ij"], s["r0"] = _springs(x, 5.0, rng)
    s["k"] = np.exp(rng.uniform(math.log(0.1), math.log(10.0), s["ij"].shape[0])).astype(np.float32)
    s["cfg"] = dict(timestep=0.01, spring_enable=1, steric_enable=1, steric_cutoff=c["cutoff"], steric_mode=c["mode"],
                    coulomb_enable=1, coulomb_cutoff=c["cutoff"], coulomb_dielectric=4.0,
                    dielectric_mode=c["dielectric"], rebuild_every=10, list_skin=c["skin"])
    return s


def _membrane_system(c, seed):
    n, nb = c["n"], c["bodies"]
    rng = np.random.default_rng([seed, n])
    x = W.ca_chain(n, seed + 1, step=3.0, rg=2.2 * (n / 4) ** 0.38, min_sep=2.5)
    ij, r0 = _springs(x, 8.0, rng)
    mass = np.full(n, 50.0, np.float32)
    s = dict(xyz=x, ij=ij, r0=r0, k=np.full(ij.shape[0], KCAL, np.float32), mass=mass, vel=_thermal(rng, n, mass),
             transfer=rng.uniform(-0.05, 0.05, n).astype(np.float32), sasa=rng.uniform(0.0, 60.0, n).astype(np.float32),
             cfg=dict(timestep=0.01, spring_enable=1, impala_enable=1, viscosity_enable=1, viscosity_value=1.0,
                      rigidbody_enable=1 if nb else 0, rebuild_every=10, list_skin=1.0))
    size = min(500, n // (2 * max(nb, 1)))
    s["bodies"] = [np.arange(b * (n // max(nb, 1)), b * (n // max(nb, 1)) + size, dtype=np.int32) for b in range(nb)]
    for body in s["bodies"]:
        s["vel"][body] = 0.0  # bodies start at rest
    return s


def _docking_system(c, seed):
    n = c["n"]
    rng = np.random.default_rng([seed, n])
    x = _beads(n, rng)
    x -= x.mean(axis=0)
    static = x[:, 2] < np.quantile(x[:, 2], c["static"])
    x[~static, 2] += 2.0  # the ligand stands off the receptor's face
    mass = np.full(n, 72.0, np.float32)
    s = dict(xyz=x, mass=mass, charge=_charges(n, 0.3, rng), is_static=static.astype(np.uint8))
    s["vel"] = np.where(static[:, None], np.float32(0), _thermal(rng, n, mass)).astype(np.float32)
    s["hydrophobicity"] = np.where(rng.random(n) < 0.2, rng.uniform(0.2, 0.8, n), 0.0).astype(np.float32)
    _lj_types(s, n, 5, rng)
    s["ij"], s["r0"] = _springs(x, 5.0, rng)
    s["k"] = np.full(s["ij"].shape[0], KCAL, np.float32)
    g = c["grid"]
    lo = x.min(axis=0).astype(np.float64) - 3.0
    h = (x.max(axis=0) + 3.0 - lo) / g
    s["grid"] = (W.field_map((g, g, g), lo, h, seed + 5), lo, h)
    top = x[~static].mean(axis=0)
    s["cfg"] = dict(timestep=0.01, spring_enable=1, steric_enable=1, steric_cutoff=10.0, steric_mode=3,
                    coulomb_enable=1, coulomb_cutoff=12.0, coulomb_dielectric=4.0, hydrophobicity_enable=1,
                    hydrophobicity_cutoff=9.0, hydrophobicity_scale=1.0, viscosity_enable=1, viscosity_value=1.0,
                    potentialgrid_enable=1, potentialgrid_scale=1.0, probe_enable=1, probe_steric=1,
                    probe_electrostatic=1, probe_x=float(top[0]), probe_y=float(top[1]),
                    probe_z=float(x[:, 2].max() + 4.0), probe_mass=72.0, probe_epsilon=0.8, probe_radius=3.5,
                    probe_charge=1.0, rebuild_every=10, list_skin=1.0)
    return s


def _ensemble_system(c, seed):
    sizes = W.ensemble_sizes(c["systems"], c["lo"], c["hi"])
    parts = [_network_system(int(m), seed, 1 + b) for b, m in enumerate(sizes)]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    s = {key: np.concatenate([p[key] for p in parts]) for key in ("xyz", "r0", "k", "mass", "vel")}
    s["ij"] = np.concatenate([p["ij"] + np.int32(o) for p, o in zip(parts, off)])
    s["cfg"], s["offsets"] = parts[0]["cfg"], off
    return s


def _fit_system(c, seed):
    n = c["n"]
    s = _network_system(n, seed)
    s["xyz"] = s["xyz"].copy()
    s["cfg"] = dict(s["cfg"], precise_positions=1)
    s["target"] = (s["xyz"] + W.smooth_displacement(s["xyz"], seed + 17, 2.0)).astype(np.float32)
    if c["charges"]:
        rng = np.random.default_rng([seed, n, 3])
        s["charge"] = np.where(rng.random(n) < 0.5, rng.normal(0.0, 0.5, n), 0.0).astype(np.float32)
        s["cfg"].update(coulomb_enable=1, coulomb_cutoff=12.0, coulomb_dielectric=4.0)
    return s


def _direct_system(c, seed):
    n = c["n"]
    rng = np.random.default_rng([seed, n])
    x = _beads(n, rng)
    s = dict(xyz=x, charge=_charges(n, 0.3, rng), is_static=(rng.random(n) < 0.1).astype(np.uint8))
    s["hydrophobicity"] = np.where(rng.random(n) < 0.2, rng.uniform(0.2, 0.8, n), 0.0).astype(np.float32)
    _lj_types(s, n, 5, rng)
    if c["mode"] == 0:
        s["radius"] = (s["radius"] * np.float32(0.5)).astype(np.float32)
    s["mass"], s["vel"] = np.ones(n, np.float32), np.zeros((n, 3), np.float32)
    s["ij"], s["r0"], s["k"] = np.zeros((0, 2), np.int32), np.zeros(0, np.float32), np.zeros(0, np.float32)
    s["cfg"] = dict(spring_enable=0, steric_enable=1, steric_cutoff=c["cutoff"], steric_mode=c["mode"], coulomb_enable=1,
                    coulomb_cutoff=c["cutoff"], coulomb_dielectric=4.0, dielectric_mode=c["dielectric"],
                    hydrophobicity_enable=1, hydrophobicity_cutoff=8.0, hydrophobicity_scale=1.0)
    return s


def _system(c, seed):
    kind = c["kind"]
    if kind == "network":
        s = _network_system(c["n"], seed)
        if c["pull"]:
            rng = np.random.default_rng([seed, 11])
            s["pull"] = np.zeros((c["n"], 3), np.float32)
            ids = rng.permutation(c["n"])[:5]
            s["pull"][ids] = rng.normal(0.0, 4e-4, (5, 3))  # about 1 kcal/mol/A each
        return s
    if kind == "score":
        s = _lj_system(c, seed)
        rng = np.random.default_rng([seed, 13])
        s["pose"] = (s["xyz"] + rng.normal(0.0, 0.1, s["xyz"].shape)).astype(np.float32)
        return s
    return {"lj": _lj_system, "membrane": _membrane_system, "docking": _docking_system, "ensemble": _ensemble_system,
            "fit": _fit_system, "direct": _direct_system}[kind](c, seed)


# ---------------------------------------------------------------------------------------------
# what a program keeps, and one pass
# ---------------------------------------------------------------------------------------------

ARRAYS = ("xyz", "vel", "mass", "charge", "radius", "epsilon", "hydrophobicity", "sasa", "transfer", "is_static")


def prepare(case, seed):
    s = _system(case, seed)
    if case["kind"] == "direct":
        lib = capi.load()
        fn = lib.bs_nonbonded_forces_noalloc
        fn.restype = ctypes.c_int
        fn.argtypes = [ctypes.POINTER(capi.BsConfig), ctypes.c_int64] + [ctypes.c_void_p] * 9 + [ctypes.c_char_p,
                                                                                               ctypes.c_size_t]
        cfg = capi.default_config()
        for key, v in s["cfg"].items():
            setattr(cfg, key, v)
        keys = ("xyz", "radius", "epsilon", "charge", "hydrophobicity", "is_static")
        dev = {k: torch.from_numpy(np.ascontiguousarray(s[k])).cuda() for k in keys}
        dev["f"] = torch.zeros(case["n"], 3, device="cuda")
        dev["e"] = torch.zeros(len(capi.ENERGY_NAMES), dtype=torch.float64, device="cuda")
        return dict(case=case, fn=fn, cfg=cfg, dev=dev, args=[dev[k].data_ptr() for k in keys])
    net = SpringNetwork()
    net.addParticles(**{k: s[k] for k in ARRAYS if k in s})
    net.addSprings(s["ij"], s["r0"], s["k"])
    if s.get("bodies"):
        net.setRigidBodies(s["bodies"])
    if "grid" in s:
        net.setFieldGrid(capi.BS_GRID_POTENTIAL, *s["grid"])
    if "offsets" in s:
        net.setSystems(s["offsets"])
    net.setup(s["cfg"])
    state = dict(case=case, net=net)
    if case.get("tune"):
        net.batchAutotune()
    if "pull" in s:
        state["pull"] = s["pull"]
    if "pose" in s:
        state["pose"] = s["pose"]
    if case["kind"] == "fit":
        state["k"] = torch.from_numpy(s["k"]).cuda().requires_grad_(True)
        state["r0"] = torch.from_numpy(s["r0"]).cuda().requires_grad_(True)
        state["q"] = torch.from_numpy(s["charge"]).cuda().requires_grad_(True) if case["charges"] else None
        state["target"] = s["target"]
    return state


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "direct":
        d = state["dev"]
        stream = torch.cuda.current_stream().cuda_stream
        rc = state["fn"](ctypes.byref(state["cfg"]), c["n"], *state["args"], d["f"].data_ptr(), d["e"].data_ptr(), stream,
                         None, 0)
        if rc != capi.BS_OK:
            raise RuntimeError("bs_nonbonded_forces_noalloc: %d" % rc)
        return d["f"], d["e"].tolist()  # the energies go on the caller's display
    net = state["net"]
    if kind == "fit":
        state["k"].grad = state["r0"].grad = None
        loss = SpringFitLoss.apply(state["k"], state["r0"], net, state["target"], c["steps"], c["checkpoint"], state["q"])
        if state["q"] is not None:
            state["q"].grad = None
        loss.backward()
        out = [loss.item(), state["k"].grad, state["r0"].grad]
        return out if state["q"] is None else out + [state["q"].grad]
    if kind == "score":
        net.setPositions(state["pose"])
        net.computeForces()
        return net.getForces(), net.energies()
    if "pull" in state:
        net.setExternalForces(state["pull"])
    net.computeStep(c["steps"])
    if "pull" in state or kind == "membrane":
        return net.getPositions(), net.energies()  # a frame for the viewer
    out = [net.getPositions(), net.getVelocities(), net.energies()]  # a restart point
    if kind == "docking":
        out.append(net.getProbe())
    return out


# ---------------------------------------------------------------------------------------------
# bytes and operations of a pass
# ---------------------------------------------------------------------------------------------

def _sphere(r):
    return BEAD_DENSITY * 4.0 / 3.0 * math.pi * r ** 3


def work(case):
    """State in and out once, topology and parameters in once; operations of every step: 30 per
    Lennard-Jones pair, 20 per Coulomb or hydrophobic pair, 24 per spring, 30 per particle (pairs
    counted once, from the density). A gradient costs each step's springs about four times over."""
    kind, steps = case["kind"], case.get("steps", 1)
    if kind == "ensemble":
        n = case["systems"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
    else:
        n = case["n"]
    springs = n * {"network": 9.6, "ensemble": 9.6, "fit": 9.6, "membrane": 16.0, "direct": 0.0}.get(kind, 6.0)
    per_step = 24.0 * springs + 30.0 * n
    if kind in ("lj", "score"):
        per_step += n * _sphere(case["cutoff"]) / 2 * (30.0 + 20.0 * case["charged"] ** 2)
    elif kind == "docking":
        per_step += n * (1 - case["static"]) * (_sphere(10.0) / 2 * 30.0 + _sphere(12.0) / 2 * 0.09 * 20.0 + 30.0)
    elif kind == "direct":
        per_step += n * n / 2 * 8.0 + n * _sphere(case["cutoff"]) / 2 * (30.0 + 20.0 * 0.09)
    nbytes = n * (24.0 + 24.0 + 28.0) + springs * 16.0
    if kind == "fit":
        per_step *= 5.0
        nbytes += n * 12.0 + springs * 8.0
    return dict(bytes=nbytes, flops=per_step * steps)


# ---------------------------------------------------------------------------------------------
# the same pass in 64 bits
# ---------------------------------------------------------------------------------------------

NA, E_CHARGE, EPS0, DALTON, PI = 6.02214169E23, 1.60217653E-19, 8.854187817E-12, 1.66054E-27, 3.1415927
NEWTON = 1.0E10 / DALTON * 1.0E-30                       # N to Da A fs^-2
FORCE = 1.0E3 / NA * 1.0E10 * NEWTON                     # kJ/mol/A to Da A fs^-2
COULOMB_E = E_CHARGE ** 2 / (4.0 * PI * EPS0) / 1.0E-10 * NA * 1.0E-3
COULOMB_F = NEWTON * E_CHARGE ** 2 / (EPS0 * 1.0E-20) / (4.0 * PI)
KINETIC = (1.0E-10 * 1.0E15) ** 2 * NA * DALTON * 1.0E-3
BOLTZMANN = 1.3806504E-23


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _f64(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(_dev()).double()


def _pair_list(x, radius, shift):
    """Index pairs (i, j), each once, closer than radius: rows sorted along x, a window of columns
    for every block of rows. `shift` sets systems apart along x."""
    key = x[:, 0] + shift
    order = torch.argsort(key)
    xs = torch.cat([key[order, None], x[order, 1:]], dim=1)
    n, found, step = x.shape[0], [], 1024
    for a in range(0, n, step):
        b = min(n, a + step)
        end = int(torch.searchsorted(xs[:, 0].contiguous(), xs[b - 1, 0] + radius))
        rows, cols = xs[a:b], xs[a:end]
        d2 = torch.zeros(b - a, end - a, dtype=torch.float64, device=x.device)
        for k in range(3):
            d2 += (rows[:, k, None] - cols[None, :, k]) ** 2
        hit = torch.nonzero(torch.triu(d2 < radius * radius, diagonal=1))
        found.append(hit + a)
    p = torch.cat(found) if found else torch.zeros(0, 2, dtype=torch.long, device=x.device)
    return order[p[:, 0]], order[p[:, 1]]


class _Model:
    """Forces and energies of a system in 64 bits."""

    def __init__(self, s):
        c = capi.default_config()
        for key, v in s["cfg"].items():
            setattr(c, key, v)
        self.c, self.s, n = c, s, s["xyz"].shape[0]
        self.n, self.mass = n, _f64(s["mass"])
        get = lambda k, v: _f64(s[k]) if k in s else torch.full((n,), v, dtype=torch.float64, device=_dev())  # noqa: E731
        self.q, self.h = get("charge", 0.0), get("hydrophobicity", 0.0)
        self.sasa, self.transfer = get("sasa", 0.0), get("transfer", 0.0)
        self.radius, eps = get("radius", 1.0), get("epsilon", 0.0)
        self.dyn = 1.0 - get("is_static", 0.0)
        self.rigid = torch.zeros(n, dtype=torch.bool, device=_dev())
        self.bodies = [torch.from_numpy(b).long().to(_dev()) for b in s.get("bodies", [])]
        for b in self.bodies:
            self.rigid[b] = True
        self.P, self.F = self._lj(eps, self.radius)
        ij = torch.from_numpy(s["ij"]).long().to(_dev())
        live = ~(self.rigid[ij[:, 0]] & self.rigid[ij[:, 1]]) & (self.dyn[ij].sum(dim=1) > 0)
        self.si, self.sj = ij[live, 0], ij[live, 1]
        self.k, self.r0 = _f64(s["k"])[live], _f64(s["r0"])[live]
        x = _f64(s.get("pose", s["xyz"]))
        shift = torch.zeros(n, dtype=torch.float64, device=_dev())
        if "offsets" in s:
            of = np.repeat(np.arange(len(s["offsets"]) - 1), np.diff(s["offsets"]))
            shift = torch.from_numpy(of).to(_dev()).double() * 4000.0
        reach = max([0.0] + [r for on, r in ((c.steric_enable, c.steric_cutoff), (c.coulomb_enable, c.coulomb_cutoff),
                                             (c.hydrophobicity_enable, c.hydrophobicity_cutoff)) if on])
        self.pi = self.pj = torch.zeros(0, dtype=torch.long, device=_dev())
        if reach > 0.0:
            i, j = _pair_list(x, reach + 0.5, shift)
            keep = self.dyn[i] + self.dyn[j] > 0
            if c.spring_enable and ij.shape[0]:
                bond = torch.minimum(ij[:, 0], ij[:, 1]) * n + torch.maximum(ij[:, 0], ij[:, 1])
                keep &= ~torch.isin(torch.minimum(i, j) * n + torch.maximum(i, j), bond)
            self.pi, self.pj = i[keep], j[keep]
        ok = (self.q[self.pi] != 0) & (self.q[self.pj] != 0)
        self.ci, self.cj = (self.pi, self.pj) if s.get("all_charges") else (self.pi[ok], self.pj[ok])
        ok = (self.h[self.pi] != 0) & (self.h[self.pj] != 0)
        self.hi, self.hj = self.pi[ok], self.pj[ok]
        self.grid = self._grid(*s["grid"]) if "grid" in s else None

    def _lj(self, eps, r):
        mode = self.c.steric_mode
        if mode == 0:
            return r, r * 0
        if mode == 3:
            return eps * r ** 6, eps * r ** 8
        return eps.sqrt() * r ** 3, eps.sqrt() * r ** (6 if mode == 1 else 4)

    def _grid(self, scalar, lo, h):
        v = _f64(scalar)
        g = torch.zeros(v.shape + (4,), dtype=torch.float64, device=v.device)
        g[..., 0] = v
        scale = BOLTZMANN * 1.0E10 * NEWTON
        for a in range(3):
            m = v.shape[a]
            d = (v.narrow(a, 2, m - 2) - v.narrow(a, 0, m - 2)) / (2.0 * h[a])
            g[..., 1 + a].narrow(a, 1, m - 2).copy_(-scale * d)
        return g, torch.tensor(lo, device=v.device), torch.tensor(h, device=v.device)

    def _contact(self, r2, P, F, own):
        """Steric energy and force over distance of pairs with factor products P and F (linear
        mode: `own` is the sum of radii)."""
        mode = self.c.steric_mode
        if mode == 0:
            d = r2.sqrt()
            dv = torch.where(d < own, d - own, torch.zeros_like(d))
            return 0.5 * dv * dv, dv / d
        inv = 1.0 / r2
        t6 = P * inv ** 3
        if mode == 1:
            t = F * inv ** 6
            return t - 2.0 * t6, 12.0 * (t6 - t) * inv
        t = F * inv ** 4
        return (3.0 * t - 4.0 * t6, 24.0 * (t6 - t) * inv) if mode == 2 else (t - t6, (6.0 * t6 - 8.0 * t) * inv)

    def _charge(self, r2, qq):
        inv = r2.rsqrt()
        if self.c.dielectric_mode:
            return qq * inv * inv, -2.0 * qq * inv ** 4
        return qq * inv, -qq * inv ** 3

    def forces(self, x, v, probe=None, k=None, r0=None, q=None):
        """Force on every particle, energies (spring, steric, electrostatic, imp, hydrophobic) and
        the probe's force."""
        c, f = self.c, torch.zeros_like(x)
        e = dict(spring=0.0, steric=0.0, electrostatic=0.0, imp=0.0, hydrophobic=0.0)
        k, r0, q = self.k if k is None else k, self.r0 if r0 is None else r0, self.q if q is None else q
        kc = COULOMB_F * c.coulomb_scale / c.coulomb_dielectric
        ke = COULOMB_E * c.coulomb_scale / c.coulomb_dielectric

        def both(f, i, j, d, fod, scale):
            w = (d * fod[:, None]) * scale
            return f.index_add(0, i, w).index_add(0, j, -w)

        if c.spring_enable and self.si.numel():
            d = x[self.sj] - x[self.si]
            r = d.norm(dim=1)
            f = both(f, self.si, self.sj, d, k * (r - r0) / r, FORCE * c.spring_scale)
            e["spring"] = (0.5 * k * (r - r0) ** 2).sum() * c.spring_scale
        if c.steric_enable and self.pi.numel():
            for a in range(0, self.pi.numel(), 1 << 24):
                i, j = self.pi[a:a + (1 << 24)], self.pj[a:a + (1 << 24)]
                d = x[j] - x[i]
                r2 = (d * d).sum(dim=1)
                near = r2 < c.steric_cutoff ** 2
                i, j, d, r2 = i[near], j[near], d[near], r2[near]
                en, fod = self._contact(r2, self.P[i] * self.P[j], self.F[i] * self.F[j], self.radius[i] + self.radius[j])
                f = both(f, i, j, d, fod, FORCE * c.steric_gridscale)
                e["steric"] = e["steric"] + en.sum() * c.steric_gridscale
        if c.coulomb_enable and self.ci.numel():
            d = x[self.cj] - x[self.ci]
            r2 = (d * d).sum(dim=1)
            near = r2 < c.coulomb_cutoff ** 2
            i, j = self.ci[near], self.cj[near]
            en, fod = self._charge(r2[near], q[i] * q[j])
            f = both(f, i, j, d[near], fod, kc)
            e["electrostatic"] = en.sum() * ke
        if c.hydrophobicity_enable and self.hi.numel():
            d = x[self.hj] - x[self.hi]
            r = d.norm(dim=1)
            near = r < c.hydrophobicity_cutoff
            i, j, d, r = self.hi[near], self.hj[near], d[near], r[near]
            t = self.h[i] * self.h[j] * torch.exp(-r)
            f = both(f, i, j, d, t / r, FORCE * c.hydrophobicity_scale)
            e["hydrophobic"] = -t.sum() * NA * 1.0E-3 * c.hydrophobicity_scale
        if self.grid is not None:
            g, lo, h = self.grid
            at = ((x - lo) / h).long()
            inside = ((at >= 0) & (at < torch.tensor(g.shape[:3], device=x.device))).all(dim=1) & (self.dyn > 0)
            cell = g[tuple(at[inside].T)]
            add = torch.zeros_like(x)
            add[inside] = cell[:, 1:] * q[inside, None] * c.potentialgrid_scale
            f = f + add
            e["electrostatic"] = e["electrostatic"] + (cell[:, 0] * q[inside]).sum() * BOLTZMANN * 1.0E-3 * NA
        if c.viscosity_enable:
            f = f - v * c.viscosity_value
        if c.impala_enable:
            u = x[:, 2]
            ex = torch.exp(c.impala_alpha * (u.abs() - c.impala_z0))
            g = -self.sasa * self.transfer + np.float32(-0.018) * self.sasa
            e["imp"] = (self.dyn * c.impala_scale * g * (0.5 - 1.0 / (1.0 + ex))).sum()
            dc = c.impala_alpha * torch.sign(u) / (ex + 2.0 + 1.0 / ex)
            f = f - torch.stack([u * 0, u * 0, c.impala_scale * g * dc * FORCE], dim=1)
        fp = None
        if probe is not None:
            d = probe - x
            r2 = (d * d).sum(dim=1)
            one = torch.ones(1, dtype=torch.float64, device=x.device)
            pr = c.probe_radius * one
            P, F = self._lj(c.probe_epsilon * one, pr)
            en, fod = self._contact(r2, P * self.P, F * self.F, pr + self.radius)
            en2, fod2 = self._charge(r2, c.probe_charge * q)
            w = d * (fod * FORCE * c.steric_gridscale + fod2 * kc)[:, None] * self.dyn[:, None]
            f, fp = f + w, -w.sum(dim=0)
            e["steric"] = e["steric"] + (en * self.dyn).sum() * c.steric_gridscale
            e["electrostatic"] = e["electrostatic"] + (en2 * self.dyn).sum() * ke
        return f * self.dyn[:, None], e, fp


def _turn(p, w, half):
    """p rotated by the normalised quaternion (w sin(half), cos(half))."""
    v, s = w * math.sin(half), math.cos(half)
    m = (float((v * v).sum()) + s * s) ** 0.5
    return v / m, s / m


def _qmul(a, b):
    return (b[0] * a[1] + a[0] * b[1] + torch.linalg.cross(a[0], b[0]), a[1] * b[1] - (a[0] * b[0]).sum(-1))


def _advance(m, steps, ext=None):
    """`steps` semi-implicit Euler steps; the external force acts on the first."""
    c, dt = m.c, float(np.float32(m.c.timestep))
    x, v = _f64(m.s["xyz"]), _f64(m.s["vel"])
    probe = torch.tensor([c.probe_x, c.probe_y, c.probe_z], dtype=torch.float64, device=x.device) if c.probe_enable else None
    pv = torch.zeros(3, dtype=torch.float64, device=x.device)
    body = []
    for ids in m.bodies:
        M = float(m.mass[ids].sum())
        X = (x[ids] * m.mass[ids, None]).sum(dim=0) / M
        zero = torch.zeros(3, dtype=torch.float64, device=x.device)
        body.append(dict(ids=ids, M=M, X=X, V=zero, L=zero, q=(zero, 1.0), p0=x[ids] - X))
    free = (~m.rigid).double()
    for step in range(steps):
        f, e, fp = m.forces(x, v, probe)
        if ext is not None and step == 0:
            f = f + ext * m.dyn[:, None]
        v = v + f / m.mass[:, None] * dt * free[:, None]
        e["kinetic"] = (0.5 * m.mass * (v * v).sum(dim=1) * m.dyn * free).sum() * KINETIC
        nx = x + v * dt * (m.dyn * free)[:, None]
        for b in body:
            ids = b["ids"]
            a = f[ids].sum(dim=0) / b["M"]
            torque = torch.linalg.cross(x[ids] - b["X"], f[ids]).sum(dim=0)
            b["V"] = b["V"] + a * dt
            b["X"] = b["X"] + b["V"] * dt + a * 0.5 * dt * dt
            b["L"] = b["L"] + torque * dt
            w = b["L"] / (0.4 * b["M"])
            dq = _turn(None, w, float(w.norm()) * dt / 2.0)
            q = _qmul(dq, b["q"])
            size = (float((q[0] * q[0]).sum()) + float(q[1]) ** 2) ** 0.5
            b["q"] = (q[0] / size, float(q[1]) / size)
            qv = b["q"][0].expand_as(b["p0"])
            zero = torch.zeros(len(ids), dtype=torch.float64, device=x.device)
            qs = zero + b["q"][1]
            mid = (b["p0"] * qs[:, None] + torch.linalg.cross(qv, b["p0"]), -(qv * b["p0"]).sum(-1))
            r = -qv * mid[1][:, None] + mid[0] * qs[:, None] + torch.linalg.cross(mid[0], -qv)
            nx[ids] = b["X"] + r
            v[ids] = (nx[ids] - x[ids]) / dt
        x = nx
        if probe is not None:
            fp = fp - (pv * c.viscosity_value if c.viscosity_enable else 0.0)
            pv = pv + fp / c.probe_mass * dt
            e["kinetic"] = e["kinetic"] + 0.5 * c.probe_mass * float((pv * pv).sum()) * KINETIC
            probe = probe + pv * dt
    return x, v, e, probe, pv


def _np(t):
    return t.detach().cpu().numpy()


def _energies(e):
    return {k: float(e.get(k, 0.0)) for k in capi.ENERGY_NAMES}


def _exact_fit(case, s):
    s["all_charges"] = bool(case["charges"])
    m = _Model(s)
    dt = float(np.float32(m.c.timestep))
    k, r0, q = m.k.clone().requires_grad_(True), m.r0.clone().requires_grad_(True), m.q.clone().requires_grad_(True)
    x, v = _f64(s["xyz"]), _f64(s["vel"])
    for _ in range(case["steps"]):
        f, _, _ = m.forces(x, v, k=k, r0=r0, q=q)
        v = v + f / m.mass[:, None] * dt
        x = x + v * dt
    loss = ((x - _f64(s["target"])) ** 2).sum() / m.n
    loss.backward()
    out = [float(loss), _np(k.grad), _np(r0.grad)]
    return out + [_np(q.grad)] if case["charges"] else out


def exact(case, seed):
    s, kind = _system(case, seed), case["kind"]
    if kind == "fit":
        return _exact_fit(case, s)
    m = _Model(s)
    if kind in ("score", "direct"):
        x = _f64(s.get("pose", s["xyz"]))
        f, e, _ = m.forces(x, torch.zeros_like(x))
        e = _energies(e)
        return [_np(f), e] if kind == "score" else [_np(f), [e[k] for k in capi.ENERGY_NAMES]]
    x, v, e, probe, pv = _advance(m, case["steps"], _f64(s["pull"]) if "pull" in s else None)
    e = _energies(e)
    if "pull" in s or kind == "membrane":
        return [_np(x), e]
    out = [_np(x), _np(v), e]
    if kind == "docking":
        out.append(_np(torch.cat([probe, pv])))
    return out
