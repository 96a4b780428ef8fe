"""Backward steps in one kernel between two rebuilds: gradients against the FP64 adjoint, within the 1e-4
relative L2 of the other gradient checks, on both sides of the sizes where the lanes per particle change
(6,080, 12,160) and where the steps get a kernel each (36,480), and with more springs per particle
than a lane holds (3 each: more than 48 with 16 lanes, more than 12 with 4)."""

from __future__ import annotations

import numpy as np
import pytest

from biospring_gb300 import workloads as W
from helpers import gpu_network
from oracle import pyoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cutoff,steps,checkpoint", [(1, 10.0, 3, 2), (21, 10.0, 5, 1), (500, 18.0, 9, 4),
                                                       (6080, 10.0, 6, 4), (6081, 10.0, 6, 6), (12161, 10.0, 6, 4),
                                                       (36481, 8.0, 4, 3)])
def test_gradients_at_the_edges(n, cutoff, steps, checkpoint):
    s = W.ca_network(max(n, 3), seed=6, spring_cutoff=cutoff)
    if n < 3:  # one particle: no spring, the loss alone
        s = W.System("one", s.xyz[:n], s.ij[:0], s.r0[:0], s.k[:0], s.config)
    s.config.update(precise_positions=1, rebuild_every=checkpoint)
    target = (s.xyz + W.smooth_displacement(s.xyz, 3, 2.0)).astype(np.float32)
    net = gpu_network(s)
    loss, gk, gr = net.adjoint(steps, target, checkpoint=checkpoint)
    ref_loss, rk, rr = pyoracle.adjoint_fp64(s, steps, target)
    assert abs(loss - ref_loss) <= 1e-6 * abs(ref_loss)
    if s.ij.shape[0]:
        if n == 500:
            assert np.bincount(s.ij.ravel(), minlength=n).max() > 48
        assert np.linalg.norm(gk - rk) < 1e-4 * np.linalg.norm(rk)
        assert np.linalg.norm(gr - rr) < 1e-4 * np.linalg.norm(rr)
    net.close()
