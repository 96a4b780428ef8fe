"""Results on both sides of the 48 KB (4,096 particles) up to which the kernel writes them to the host itself, and
states on both sides of the 384 KB (32,768 particles) up to which they go in through the handle's own buffer, one after
the other. All bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

from biospring_gb300 import workloads as W
from helpers import gpu_network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2048, 2049, 4096, 4097, 32768, 32769])
def test_states_in_and_results_out(n):
    rng = np.random.default_rng(n)
    a, b, v = (rng.uniform(0.0, 3.0 * n ** (1 / 3), (n, 3)).astype(np.float32) for _ in range(3))
    net = gpu_network(W.System("free", a, np.zeros((0, 2), np.int32), np.zeros(0, np.float32), np.zeros(0, np.float32),
                               dict(spring_enable=0, timestep=0.5)))
    for x in (b, a, b):
        mine = x.copy()
        net.setPositions(mine)
        mine[:] = np.nan
        force = v.copy()
        net.setExternalForces(force)  # through the same buffer
        force[:] = np.nan
        mine = v.copy()
        net.setVelocities(mine)
        mine[:] = np.nan
        assert np.array_equal(net.getPositions(), x) and np.array_equal(net.getVelocities(), v)
        net.computeStep(1)
        want = v + v * np.float32(0.5)  # mass 1, no force but the external one
        assert np.array_equal(net.getVelocities(), want)
        assert np.array_equal(net.getPositions(), x + want * np.float32(0.5))
    net.close()
