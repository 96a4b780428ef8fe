"""Pair lists of a dense system that has spread out since its set-up, against the oracle's pair sets (equal index for
index): groups of cells split over several blocks and taken whole, and more groups than the launch has blocks, up
to 32,768 particles and above."""

from __future__ import annotations

import copy

import numpy as np
import pytest

from helpers import gpu_network
from oracle import pyoracle as po
from test_gpu_lists import _beads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,apart", [(12000, 1.2), (12000, 1.5), (12000, 6.0), (20000, 1.5), (20000, 4.0), (40000, 4.0)])
def test_pair_sets_after_spreading(n, apart):
    s = _beads(n, 0.0244, n)
    s.config.update(spring_enable=1, steric_enable=1, steric_mode=1, steric_cutoff=12.0, coulomb_enable=1, coulomb_cutoff=11.0,
                    list_skin=0.5)
    t = copy.copy(s)
    # a tenth of the particles in pairs of neighbours, so that every list keeps partners however far the rest are apart
    t.xyz = s.xyz * np.float32(apart)
    t.xyz[1:n // 5:2] = t.xyz[0:n // 5 - 1:2] + np.float32(3.0)
    net, orc = gpu_network(s), po.Oracle(t)
    net.setPositions(t.xyz)
    for term in (0, 1):
        ref = orc.pairs(term).astype(np.int64)
        assert ref.shape[0] > 0
        np.testing.assert_array_equal(net.getPairs(term), ref)
    net.close()
    orc.close()
