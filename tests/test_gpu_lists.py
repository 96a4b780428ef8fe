"""Pair lists of dense systems against the oracle's pair sets (equal index for index): on both sides of the
sizes where a group's homes are split over 4, 2 or 1 blocks (16,384 and 32,768 particles), with more
candidates than the 1,536 a block stages and more homes than a batch, with one, two and three distinct
list radii, static particles, more spring partners than the threads of a home hold, a crowded corner (rows
longer than their first capacity) and slot offsets that leave 16 bits."""

from __future__ import annotations

import numpy as np
import pytest

from biospring_gb300 import workloads as W
from helpers import gpu_network, rel_l2
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _beads(n, density, seed, flat=False):
    rng = np.random.default_rng(seed)
    a = density ** (-1.0 / 3.0)
    m = np.array([int(np.ceil(np.sqrt(n / 4)))] * 2 + [4]) if flat else np.array([int(np.ceil(n ** (1 / 3)))] * 3)
    cells = np.sort(rng.permutation(int(m.prod()))[:n])
    x = np.stack([cells % m[0], cells // m[0] % m[1], cells // (m[0] * m[1])], axis=1) * a
    x = (x + rng.uniform(-0.3, 0.3, (n, 3)))[rng.permutation(n)].astype(np.float32)
    ij = W.pairs_within(x, 1.3 * a)
    s = W.System("beads", x, ij, np.full(ij.shape[0], a, np.float32), np.ones(ij.shape[0], np.float32), {})
    s.radius, s.epsilon = np.full(n, 1.0, np.float32), np.full(n, 0.1, np.float32)
    s.charge = rng.choice([-1.0, 0.0, 0.0, 1.0], n).astype(np.float32)
    s.hydrophobicity = np.where(rng.random(n) < 0.3, 0.5, 0.0).astype(np.float32)
    s.is_static = (rng.random(n) < 0.2).astype(np.uint8)
    return s


def _check(s, terms):
    net, orc = gpu_network(s), po.Oracle(s)
    found = 0
    for term in terms:
        got, ref = net.getPairs(term), orc.pairs(term).astype(np.int64)
        found += ref.shape[0]
        np.testing.assert_array_equal(got, ref)
    assert found > 0
    net.close()
    orc.close()


@pytest.mark.parametrize("n,density,cuts", [
    (700, 0.03, (9.0, 9.0, 9.0)),       # a few groups, most blocks without homes
    (5000, 0.12, (12.0, 12.0, 12.0)),   # some 4,700 candidates and 170 homes a group
    (6007, 0.0244, (10.0, 12.0, 9.0)),  # three radii
    (16384, 0.03, (10.0, 10.0, 8.0)),
    (16385, 0.03, (10.0, 10.0, 8.0)),
    (32768, 0.03, (9.0, 9.0, 9.0)),
    (32769, 0.03, (9.0, 9.0, 9.0)),
])
def test_pair_sets(n, density, cuts):
    s = _beads(n, density, n)
    s.config.update(spring_enable=1, steric_enable=1, steric_mode=1, steric_cutoff=cuts[0], coulomb_enable=1,
                    coulomb_cutoff=cuts[1], hydrophobicity_enable=1, hydrophobicity_cutoff=cuts[2], list_skin=0.5)
    _check(s, (0, 1, 2))


def test_many_partners():
    s = _beads(3000, 0.0244, 4)
    s.ij = W.pairs_within(s.xyz, 10.0)  # 100 partners a particle: more than 8, 32 and 64
    s.r0 = np.full(s.ij.shape[0], 6.0, np.float32)
    s.k = np.ones(s.ij.shape[0], np.float32)
    assert np.bincount(s.ij.ravel()).max() > 64
    s.config.update(spring_enable=1, steric_enable=1, steric_mode=1, steric_cutoff=12.0)
    _check(s, (0,))


def test_crowded_corner():
    s = _beads(20000, 0.0244, 5)
    s.xyz = s.xyz.copy()
    near = np.argsort(np.linalg.norm(s.xyz, axis=1))[:4000]
    s.xyz[near] *= np.float32(0.5)  # eight times the density: rows past their first capacity
    s.config.update(steric_enable=1, steric_mode=1, steric_cutoff=10.0, coulomb_enable=1, coulomb_cutoff=10.0)
    _check(s, (0, 1))


@pytest.mark.parametrize("n", [63999, 64000, 64161])
def test_sparse(n):
    """Few particles a cell: a warp a home below 64,000 particles, a thread a home from there on."""
    s = _beads(n, 0.004, n)
    s.config.update(spring_enable=1, steric_enable=1, steric_mode=1, steric_cutoff=9.0, coulomb_enable=1,
                    coulomb_cutoff=8.0, hydrophobicity_enable=1, hydrophobicity_cutoff=9.0, list_skin=0.5)
    _check(s, (0, 1, 2))


@pytest.mark.parametrize("n,density", [(8000, 0.0005), (8000, 0.0008), (65535, 0.02), (65536, 0.02)])
def test_cell_order(n, density):
    """The cell order by placed keys and by bins: more and fewer than the 4,096 cells of the short way, and
    65,535 and 65,536 particles. The forces hang on the spring table of the new order (1e-5 relative, as the
    other force checks)."""
    s = _beads(n, density, n + 1)
    s.config.update(spring_enable=1, steric_enable=1, steric_mode=1, steric_cutoff=9.0 if density > 0.01 else 17.0)
    net, orc = gpu_network(s), po.Oracle(s)
    np.testing.assert_array_equal(net.getPairs(0), orc.pairs(0).astype(np.int64))
    net.computeForces()
    orc.compute_forces()
    assert rel_l2(net.getForces(), orc.forces(), s.is_static == 0) < 1e-5  # a static particle gets none
    net.close()
    orc.close()


def test_full_bins():
    """More than the 64 particles of a bin in one cell."""
    rng = np.random.default_rng(12)
    x = rng.uniform(0.0, 6.0, (600, 3)).astype(np.float32)
    x[300:] += np.float32(100.0)
    s = W.System("clumps", x, np.zeros((0, 2), np.int32), np.zeros(0, np.float32), np.zeros(0, np.float32), {})
    s.radius, s.epsilon = np.full(600, 0.5, np.float32), np.full(600, 0.1, np.float32)
    s.config.update(spring_enable=0, steric_enable=1, steric_mode=1, steric_cutoff=9.0)
    _check(s, (0,))


def test_sparse_wide_offsets():
    s = _beads(120000, 0.004, 8, flat=True)
    s.config.update(spring_enable=1, steric_enable=1, steric_mode=1, steric_cutoff=9.0)
    _check(s, (0,))


def test_wide_offsets():
    s = _beads(120000, 0.03, 6, flat=True)
    s.config.update(steric_enable=1, steric_mode=1, steric_cutoff=9.0)
    _check(s, (0,))
