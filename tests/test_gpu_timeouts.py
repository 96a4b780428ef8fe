"""Waits between the blocks of a kernel that run out (BS_BARRIER_POLLS=1: a block that does not find the others at its
first look gives up): list rebuild, kernel of several steps, backward steps, ensemble steps. The call returns
BS_E_TIMEOUT, so do the following ones, and the same handle set up again gives the bits of a new one."""

from __future__ import annotations

import numpy as np
import pytest

from biospring_gb300 import BsError, SpringNetwork, capi
from biospring_gb300 import workloads as W
from helpers import gpu_network

pytestmark = pytest.mark.gpu


def _charged(n):
    """n beads, of which a block of 16 takes more work than the rest."""
    x = (np.stack(np.unravel_index(np.arange(n), (4, 4, 4)), axis=1) * 3.0).astype(np.float32)
    s = W.System("beads", x, np.zeros((0, 2), np.int32), np.zeros(0, np.float32), np.zeros(0, np.float32),
                 dict(spring_enable=0, coulomb_enable=1, coulomb_cutoff=30.0, timestep=0.01, rebuild_every=50, list_skin=1.0))
    s.charge, s.mass = np.ones(n, np.float32), np.full(n, 100.0, np.float32)
    return s


def _times_out(call, n=2):
    for _ in range(n):
        with pytest.raises(BsError) as e:
            call()
        assert e.value.code == capi.BS_E_TIMEOUT


def _fresh(net, s, steps):
    """net, set up again, against a new handle."""
    net.setup(s.bs_config())
    ref = gpu_network(s)
    net.computeStep(steps)
    ref.computeStep(steps)
    assert np.array_equal(net.getPositions(), ref.getPositions()) and net.energies() == ref.energies()
    net.close()
    ref.close()


def test_rebuild(monkeypatch):
    s = W.ca_network(2000, seed=1)
    net = SpringNetwork()
    net.addParticles(**{k: v for k, v in s.arrays().items() if v is not None})
    net.addSprings(s.ij, s.r0, s.k)
    monkeypatch.setenv("BS_BARRIER_POLLS", "1")
    _times_out(lambda: net.setup(s.bs_config()))
    monkeypatch.delenv("BS_BARRIER_POLLS")
    _fresh(net, s, 20)


def test_steps(monkeypatch):
    s = _charged(17)  # one block rebuilds, two step
    monkeypatch.setenv("BS_BARRIER_POLLS", "1")
    net = gpu_network(s)
    monkeypatch.delenv("BS_BARRIER_POLLS")
    _times_out(lambda: net.computeStep(1000))
    _times_out(net.getPositions)
    _fresh(net, s, 60)


def test_backward_steps(monkeypatch):
    s = W.ca_network(3, seed=1)  # one block rebuilds and steps, two take the backward steps
    monkeypatch.setenv("BS_BARRIER_POLLS", "1")
    net = gpu_network(s)
    monkeypatch.delenv("BS_BARRIER_POLLS")
    _times_out(lambda: net.adjoint(40, s.xyz + np.float32(0.5), checkpoint=40))
    net.setup(s.bs_config())
    ref = gpu_network(s)
    for a, b in zip(net.adjoint(40, s.xyz + np.float32(0.5), checkpoint=40), ref.adjoint(40, s.xyz + np.float32(0.5), checkpoint=40)):
        assert np.array_equal(a, b)
    net.close()
    ref.close()


def test_ensemble(monkeypatch):
    s = _charged(17)
    monkeypatch.setenv("BS_BARRIER_POLLS", "1")
    net = SpringNetwork()
    net.addParticles(**{k: v for k, v in s.arrays().items() if v is not None})
    net.setSystems([0, 17])
    net.setBatchShape(128, 8, 1)  # one block rebuilds, two step
    net.setup(s.bs_config())
    monkeypatch.delenv("BS_BARRIER_POLLS")
    _times_out(lambda: net.computeStep(1000))
    net.setup(s.bs_config())
    net.computeStep(60)
    assert net.stepCount() == 60
    net.close()
