"""The adjoint where a list rebuild inside its run is blocked: a grid with more cells than there is room for, and
slot offsets that leave the 16-bit list. The host then grows what was too small and runs again, and the
gradients are those of the FP64 adjoint within the 1e-4 relative L2 of the other gradient checks. On both sides of the
36,480 particles up to which the backward steps run in one kernel; always the handle's first adjoint, for which
the spring ids have never been sorted."""

from __future__ import annotations

import numpy as np
import pytest

from biospring_gb300 import workloads as W
from helpers import gpu_network
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _lattice(n, m, a):
    c = np.arange(n)
    return np.stack([c % m[0], c // m[0] % m[1], c // (m[0] * m[1])], axis=1) * a


def _system(x, seed):
    """Overlapping beads with springs along the index, at rest up to 0.05 A at x."""
    n = x.shape[0]
    rng = np.random.default_rng(seed)
    ij = np.stack([np.arange(n - 1), np.arange(1, n)], axis=1).astype(np.int32)
    d = np.linalg.norm(x[1:].astype(np.float64) - x[:-1], axis=1)
    s = W.System("beads", x, ij, (d + rng.normal(0.0, 0.05, n - 1)).astype(np.float32), np.full(n - 1, 4.0, np.float32), {})
    s.radius = np.full(n, 2.2, np.float32)
    s.config.update(spring_enable=1, steric_enable=1, steric_mode=0, steric_cutoff=8.0, list_skin=1.0, viscosity_enable=1,
                    viscosity_value=1.0, timestep=0.01, precise_positions=1, rebuild_every=10)
    return s


def _first_adjoint(s, before):
    """Gradients at s by a handle that was set up with the particles at `before` and moved to s."""
    target = (s.xyz + W.smooth_displacement(s.xyz, 3, 2.0)).astype(np.float32)
    there = s.xyz
    s.xyz = before
    net = gpu_network(s)
    s.xyz = there
    net.setPositions(there)
    loss, gk, gr = net.adjoint(4, target, checkpoint=2)
    ref_loss, rk, rr = pyoracle.adjoint_fp64(s, 4, target)
    assert abs(loss - ref_loss) <= 1e-6 * abs(ref_loss)
    assert np.linalg.norm(gk - rk) < 1e-4 * np.linalg.norm(rk)
    assert np.linalg.norm(gr - rr) < 1e-4 * np.linalg.norm(rr)
    assert np.array_equal(net.getPositions(), there)
    net.close()


@pytest.mark.parametrize("n", [500, 36600])
def test_more_cells_than_room(n):
    m = int(np.ceil(n ** (1 / 3)))
    rng = np.random.default_rng(n)
    x = _lattice(n, (m, m, m), 4.0) + rng.uniform(-0.2, 0.2, (n, 3))
    # the same structure in eight parts 150 A from each other: 21^3 and 33^3 cells of 9 A, where the handle has room for
    # 2 x 7^3 + 1,024 and 2 x 18^3 + 1,024
    far = x + 150.0 * (x > x.mean(axis=0))
    _first_adjoint(_system(far.astype(np.float32), n), x.astype(np.float32))


@pytest.mark.parametrize("side", [183, 190])
def test_offsets_beyond_16_bits(side):
    # a plate of two sheets in one layer of cells, and a strip of 14 rows in the layer above it, over its last rows
    # at set-up (offsets below 16 bits) and then over its first rows
    rng = np.random.default_rng(side)
    plate = _lattice(side * side, (side, side, 1), 4.0)
    plate[:, 2] = 4.0 * (rng.random(side * side) < 0.5)
    strip = _lattice(14 * side, (side, 14, 1), 4.0)
    strip[:, 2] = 9.5
    high = strip + np.array([0.0, 4.0 * (side - 14), 0.0])
    jitter = rng.uniform(-0.2, 0.2, ((side + 14) * side, 3)) * [1.0, 1.0, 0.0]
    x0, x1 = (np.concatenate([plate, q]) + jitter for q in (high, strip))
    _first_adjoint(_system(x1.astype(np.float32), side), x0.astype(np.float32))
