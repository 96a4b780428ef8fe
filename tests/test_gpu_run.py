"""The kernel of several steps (one cooperative launch between two list rebuilds) against the same steps
launched one kernel at a time: positions, velocities, energies and the step count bit for bit, at the
edges of its blocks and of its range (16 lanes a particle below 8,000, 8 up to 19,456, 4 up to the 38,912
that 608 resident blocks hold; rows held in registers up to 4,864 and 7,296 with 16 lanes, 14,592 with 8), across stale lists and with bodies. With the probe, whose reaction is summed
in another order (float-float, then rounded once), positions agree to 1e-6 A."""

from __future__ import annotations

import numpy as np
import pytest

from biospring_gb300 import BsError
from biospring_gb300 import workloads as W
from helpers import gpu_network, load_golden, system_from_golden

pytestmark = pytest.mark.gpu


def _state(net):
    return net.getPositions(), net.getVelocities(), np.array(list(net.energies().values())), net.stepCount()


def _phases(net, steps, every):
    for k in range(steps):
        if k % every == 0:
            net.launchPhase(0)
        net.launchPhase(1)
    net.synchronize()


def _same(a, b, steps):
    for x, y in zip(_state(a), _state(b)):
        assert np.array_equal(x, y)
    assert a.stepCount() == steps
    a.close()
    b.close()


def _system(n):
    if n > 4096:
        rng = np.random.default_rng(n)
        m = int(np.ceil(n ** (1 / 3)))
        x = np.stack(np.unravel_index(np.arange(n), (m, m, m)), axis=1) * 3.4 + rng.uniform(-0.2, 0.2, (n, 3))
        ij = np.stack([np.arange(n - 1), np.arange(1, n)], axis=1).astype(np.int32)
        r0 = np.linalg.norm(x[1:] - x[:-1], axis=1).astype(np.float32) + np.float32(0.05)
        s = W.System("beads", x.astype(np.float32), ij, r0, np.full(n - 1, 4.0, np.float32), {})
        s.radius, s.epsilon = np.full(n, 3.4, np.float32), np.full(n, 0.8, np.float32)
        s.charge = rng.choice([-1.0, 0.0, 0.0, 1.0], n).astype(np.float32)
        s.config.update(steric_enable=1, steric_mode=1, steric_cutoff=6.0, coulomb_enable=1, coulomb_cutoff=7.0)
    else:
        s = W.ca_network(n=n, seed=n) if n > 2 else W.membrane_globule(n=n, seed=5)
    s.config.update(timestep=0.05, rebuild_every=10, list_skin=0.5)
    return s


@pytest.mark.parametrize("n", [1, 16, 17, 300, 4864, 4865, 7296, 7297, 7999, 8001, 14592, 14593, 19456, 19457, 20000, 38912,
                               38913])
def test_same_bits_as_single_steps(n):
    s = _system(n)
    a, b = gpu_network(s), gpu_network(s)
    a.computeStep(23)  # two periods and a remainder
    _phases(b, 23, 10)
    _same(a, b, 23)


def test_stale_list_stops_and_resumes():
    s = _system(400)
    s.vel = np.random.default_rng(3).normal(0.0, 0.05, (400, 3)).astype(np.float32)
    s.config.update(timestep=1.0, list_skin=0.6)
    a, b = gpu_network(s), gpu_network(s)
    a.computeStep(37)
    for _ in range(37):
        b.computeStep(1)
    _same(a, b, 37)


@pytest.mark.parametrize("axes", [(0,), (0, 1, 2)])
def test_no_coordinates_are_reported(axes):
    s = _system(300)
    net = gpu_network(s)
    x = s.xyz.copy()
    x[:, list(axes)] = np.nan
    net.setPositions(x)
    with pytest.raises(BsError):
        net.computeStep(2)
    net.close()


def test_external_force_acts_on_the_first_step():
    s = _system(300)
    f = np.random.default_rng(4).normal(0.0, 1e-3, (300, 3)).astype(np.float32)
    a, b = gpu_network(s), gpu_network(s)
    for net in (a, b):
        net.setExternalForces(f)
    a.computeStep(10)
    _phases(b, 10, 10)
    _same(a, b, 10)


@pytest.mark.parametrize("n", [2100, 20000])
def test_bodies(n):
    s = W.membrane_globule(n=n, seed=3, nbodies=4, body_size=500)
    s.config.update(timestep=0.2, rigidbody_enable=1, rebuild_every=10)
    a, b = gpu_network(s), gpu_network(s)
    a.computeStep(20)
    _phases(b, 20, 10)
    _same(a, b, 20)


def test_probe():
    s = system_from_golden(load_golden("probe.npz"))
    s.config.update(timestep=0.2, rebuild_every=10)
    a, b = gpu_network(s), gpu_network(s)
    a.computeStep(15)
    _phases(b, 15, 10)
    assert np.abs(a.getPositions().astype(np.float64) - b.getPositions()).max() < 1e-6
    assert np.abs(a.getProbe().astype(np.float64) - b.getProbe()).max() < 1e-6
    a.close()
    b.close()
