"""The forms of the kernel of several steps, and of the steps without energy sums, against the same steps one kernel at
a time with their energies: positions, velocities, energies and the step count bit for bit. Every steric form, with
the lanes and held rows of each range of sizes (16 lanes with rows held at two and three blocks an SM and not held,
8 lanes held and not, 4 lanes), with and without the pairwise hydrophobic term; both sides of the largest resident
grid (38,912), beyond which a step's energies are summed only where they can be read."""

from __future__ import annotations

import numpy as np
import pytest

from biospring_gb300 import workloads as W
from helpers import gpu_network
from test_gpu_run import _phases, _same

pytestmark = pytest.mark.gpu


def _beads(n, mode, hydrophobic=False):
    rng = np.random.default_rng(n + mode)
    m = int(np.ceil(n ** (1 / 3)))
    x = np.stack(np.unravel_index(np.arange(n), (m, m, m)), axis=1) * 3.4 + rng.uniform(-0.2, 0.2, (n, 3))
    ij = np.stack([np.arange(n - 1), np.arange(1, n)], axis=1).astype(np.int32)
    r0 = np.linalg.norm(x[1:] - x[:-1], axis=1).astype(np.float32) + np.float32(0.05)
    s = W.System("beads", x.astype(np.float32), ij, r0, np.full(n - 1, 4.0, np.float32), {})
    s.radius, s.epsilon = rng.uniform(1.7, 1.8, n).astype(np.float32), rng.uniform(0.5, 0.8, n).astype(np.float32)
    if mode:
        s.radius = s.radius + np.float32(1.6)
    s.charge = rng.choice([-1.0, 0.0, 0.0, 1.0], n).astype(np.float32)
    s.hydrophobicity = np.where(rng.random(n) < 0.3, 0.5, 0.0).astype(np.float32)
    s.is_static = (rng.random(n) < 0.1).astype(np.uint8)
    s.config.update(steric_enable=1, steric_mode=mode, steric_cutoff=6.0, coulomb_enable=1, coulomb_cutoff=7.0,
                    hydrophobicity_enable=int(hydrophobic), hydrophobicity_cutoff=6.0, spring_enable=1, timestep=0.05,
                    rebuild_every=10, list_skin=0.5)
    return s


def _compare(s, steps=23):
    a, b = gpu_network(s), gpu_network(s)
    a.computeStep(steps)  # two periods and a remainder
    _phases(b, steps, 10)
    _same(a, b, steps)


@pytest.mark.parametrize("hydrophobic", [False, True])
@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [300, 5000, 7500, 10000, 16000, 20000])
def test_steric_forms(n, mode, hydrophobic):
    _compare(_beads(n, mode, hydrophobic))


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [38912, 38913])
def test_end_of_the_range(n, mode):
    _compare(_beads(n, mode))


@pytest.mark.parametrize("extra", ["hydrophobic", "precise", "bodies", "probe"])
def test_steps_without_energy_sums(extra):
    s = _beads(38913, 3, extra == "hydrophobic")
    if extra == "precise":
        s.config.update(precise_positions=1)
    if extra == "bodies":
        free = np.flatnonzero(s.is_static == 0)
        s.bodies = [free[k:k + 300].astype(np.int32) for k in (0, 9000)]
        s.config.update(rigidbody_enable=1, timestep=0.002)
    if extra == "probe":
        s.config.update(probe_enable=1, probe_steric=1, probe_electrostatic=1, probe_x=-4.0, probe_y=20.0, probe_z=20.0,
                        probe_mass=70.0, probe_epsilon=0.5, probe_radius=3.0, probe_charge=1.0)
    _compare(s)


def test_list_goes_stale_within_a_period():
    s = W.ca_network(n=400, seed=400)
    s.vel = np.random.default_rng(3).normal(0.0, 0.05, (400, 3)).astype(np.float32)
    s.config.update(timestep=1.0, list_skin=0.6, rebuild_every=10, viscosity_enable=0)
    a, b = gpu_network(s), gpu_network(s)
    a.computeStep(37)
    for k in range(37):
        b.computeStep(1)
        if k == 4:  # half a period: the list was stale before its rebuild was due
            assert np.linalg.norm(b.getPositions() - s.xyz, axis=1).max() > 0.3
    _same(a, b, 37)


@pytest.mark.parametrize("extra", ["none", "hydrophobic", "bodies", "probe"])
@pytest.mark.parametrize("n", [300, 5000, 10000, 20000])
def test_one_step_a_call(n, extra):
    """A call of one step takes the single-step kernel, with bodies or the probe the kernel of several."""
    s = _beads(n, 1, extra == "hydrophobic")
    if extra == "bodies":
        free = np.flatnonzero(s.is_static == 0)
        s.bodies = [free[k:k + 50].astype(np.int32) for k in (0, 150)]
        s.config.update(rigidbody_enable=1, timestep=0.002)
    if extra == "probe":
        s.config.update(probe_enable=1, probe_steric=1, probe_electrostatic=1, probe_x=-4.0, probe_y=10.0, probe_z=10.0,
                        probe_mass=70.0, probe_epsilon=0.5, probe_radius=3.0, probe_charge=1.0)
    a, b = gpu_network(s), gpu_network(s)
    a.computeStep(14)
    for _ in range(14):
        b.computeStep(1)
    assert np.array_equal(a.getProbe(), b.getProbe())
    _same(a, b, 14)
