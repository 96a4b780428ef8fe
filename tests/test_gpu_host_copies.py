"""The caller's arrays on their way in and out: a pageable source may be overwritten as soon as the call
returns, page-locked ones too where the call waits; results on both sides of the size (21,845 particles) up to
which the kernel writes them to the host itself; spring parameters one at a time; energies that stay current
across a getter. All bit for bit."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from biospring_gb300 import workloads as W
from helpers import gpu_network

pytestmark = pytest.mark.gpu


def _free(n):
    x = np.random.default_rng(n).uniform(0.0, 3.0 * n ** (1 / 3), (n, 3)).astype(np.float32)
    return W.System("free", x, np.zeros((0, 2), np.int32), np.zeros(0, np.float32), np.zeros(0, np.float32),
                    dict(spring_enable=0, timestep=0.5))


def _pinned(a):
    return torch.from_numpy(a.copy()).pin_memory().numpy()


@pytest.mark.parametrize("n", [1, 21845, 21846])
@pytest.mark.parametrize("pinned", [False, True])
def test_arrays_in_and_out(n, pinned):
    s = _free(n)
    net = gpu_network(s)
    rng = np.random.default_rng(7)
    x, v, f = (rng.normal(0.0, 1.0, (n, 3)).astype(np.float32) for _ in range(3))
    a, b, c = (_pinned(q) if pinned else q.copy() for q in (x, v, f))
    net.setPositions(a)
    a[:] = np.nan
    net.setVelocities(b)
    b[:] = np.nan
    assert np.array_equal(net.getPositions(), x) and np.array_equal(net.getVelocities(), v)
    net.setExternalForces(c)
    c[:] = np.nan
    net.setExternalForces(f.copy())  # replaces them, through the same buffer
    net.computeStep(1)
    want = v + f * np.float32(0.5)  # mass 1, no other force
    assert np.array_equal(net.getVelocities(), want)
    assert np.array_equal(net.getPositions(), x + want * np.float32(0.5))
    net.close()


def test_spring_parameters_one_at_a_time():
    s = W.ca_network(300, seed=3)
    rng = np.random.default_rng(4)
    k, r0 = (s.k * rng.uniform(0.5, 2.0, s.k.shape)).astype(np.float32), (s.r0 + 0.2).astype(np.float32)
    a, b = gpu_network(s), gpu_network(W.System("b", s.xyz, s.ij, r0, k, s.config))
    a.setSpringParameters(equilibrium=r0)
    a.setSpringParameters(stiffness=k)
    a.computeStep(12)
    b.computeStep(12)
    assert np.array_equal(a.getPositions(), b.getPositions())
    a.close()
    b.close()


def test_energies_around_getters():
    s = W.ca_network(300, seed=5)
    net = gpu_network(s)
    net.computeForces()
    e = net.energies()
    net.getForces()
    assert net.energies() == e
    net.computeStep(3)
    net.getPositions()
    e3 = net.energies()
    assert e3 != e and e3["kinetic"] > 0.0
    ref = gpu_network(s)
    ref.computeStep(3)
    assert ref.energies() == e3
    net.setPositions(s.xyz)  # the next evaluation rebuilds the lists and evaluates in one go
    net.computeForces()
    assert abs(net.energies()["spring"] - e["spring"]) <= 1e-6 * e["spring"]
    net.close()
    ref.close()
