"""Block groups of the ensemble kernel, sized by their systems' work: an ensemble of unequal systems gives
the same bits whatever the groups (one block each, several systems to a group of many blocks, more
systems than blocks), also where systems stop on stale lists inside a group and go on; energies, summed over a
group's blocks in float-float, agree to 1e-6 relative."""

from __future__ import annotations

import numpy as np
import pytest

from biospring_gb300 import SpringNetwork
from biospring_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _run(system, offsets, shape, cfg, steps):
    net = SpringNetwork()
    net.addParticles(**{k: v for k, v in system.arrays().items() if v is not None})
    net.addSprings(system.ij, system.r0, system.k)
    net.setSystems(offsets)
    net.setBatchShape(*shape)
    net.setup(cfg)
    for n in steps:
        net.computeStep(n)
    out = net.getPositions(), net.getVelocities(), net.getSystemEnergies(), net.stepCount()
    net.close()
    return out


@pytest.mark.parametrize("sizes", [np.geomspace(50, 20000, 24).astype(int), np.tile([3, 40, 17, 600], 350)],
                         ids=["unequal", "many"])
@pytest.mark.parametrize("stale", [False, True])
def test_groups_give_the_same_bits(sizes, stale):
    s = W.ensemble([int(n) for n in sizes], seed=5)
    cfg = dict(s.config)
    if stale:
        cfg.update(timestep=0.5, list_skin=0.05, viscosity_value=0.5)
        s.k = s.k * np.float32(50.0)
    off = s.meta["offsets"]
    a = _run(s, off, (512, 4, 1), cfg, (23,))
    assert a[3] == 23
    for shape in ((128, 4, 8), (256, 4, 2)):
        b = _run(s, off, shape, cfg, (23,))
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and b[3] == 23
        np.testing.assert_allclose(b[2], a[2], rtol=1e-6, atol=1e-9)
