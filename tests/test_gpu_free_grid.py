"""Systems without a nonbonded term: the grid that only orders the particles picks its own edge and
widens for a system that has spread. Steps and springs against the oracle; positions within 1e-5 A
after 5 steps (FP32 sums in another order at 0.01 fs)."""

from __future__ import annotations

import numpy as np
import pytest

from biospring_gb300 import SpringNetwork
from biospring_gb300 import workloads as W
from helpers import gpu_network
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _system(n, far):
    s = W.membrane_globule(n=n, seed=5)
    if far:
        s.xyz = s.xyz.copy()
        s.xyz[-1] += np.float32(far)  # one bead far away: the first edge gives too many cells
        s.ij, s.r0, s.k = (a[np.all(s.ij != n - 1, axis=1)] for a in (s.ij, s.r0, s.k))
    return s


@pytest.mark.parametrize("n,far", [(1, 0.0), (2, 0.0), (33, 0.0), (4097, 0.0), (4097, 1.0e5), (300, 1.0e9)])
def test_single_system(n, far):
    s = _system(n, far)
    net = gpu_network(s)
    orc = po.Oracle(s)
    net.computeStep(5)
    orc.step(5)
    assert np.abs(net.getPositions().astype(np.float64) - orc.positions()).max() <= max(1e-5, far * 1e-7)
    net.close()
    orc.close()


def test_batch_of_systems():
    parts = [_system(700, 0.0), _system(300, 1.0e5), _system(1, 0.0)]
    off = np.concatenate([[0], np.cumsum([p.n for p in parts])]).astype(np.int64)
    net = SpringNetwork()
    net.addParticles(np.concatenate([p.xyz for p in parts]), sasa=np.concatenate([p.sasa for p in parts]),
                     transfer=np.concatenate([p.transfer for p in parts]))
    net.addSprings(np.concatenate([p.ij + np.int32(o) for p, o in zip(parts, off)]),
                   np.concatenate([p.r0 for p in parts]), np.concatenate([p.k for p in parts]))
    net.setSystems(off)
    net.setup(parts[0].bs_config())
    net.computeStep(15)
    x = net.getPositions()
    for p, a, b in zip(parts, off, off[1:]):
        orc = po.Oracle(p)
        orc.step(15)
        assert np.abs(x[a:b].astype(np.float64) - orc.positions()).max() < (0.02 if p is parts[1] else 1e-5)
        orc.close()
    net.close()
