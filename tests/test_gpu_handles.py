"""Several handles at work at once, from one thread on their own streams and from a thread each: kernels that need all
their blocks resident take turns with other handles', and every handle's results are those it gives alone, bit for
bit."""

from __future__ import annotations

import threading

import numpy as np
import pytest

from biospring_gb300 import workloads as W
from helpers import gpu_network
from test_gpu_run_forms import _beads

pytestmark = pytest.mark.gpu


def _systems():
    out = [W.ca_network(2000, seed=1), W.ca_network(6000, seed=2), _beads(9000, 1), _beads(18000, 2), _beads(24000, 1)]
    for s in out:
        s.config.update(rebuild_every=10, list_skin=0.5)
    return out


def _result(net):
    return net.getPositions(), net.getVelocities(), np.array(list(net.energies().values()))


def _alone():
    out = []
    for s in _systems():
        net = gpu_network(s)
        net.computeStep(45)
        out.append(_result(net))
        net.close()
    return out


def test_on_streams():
    nets = [gpu_network(s) for s in _systems()]
    for steps in (20, 3, 22):
        for net in nets:
            net.computeStepAsync(steps)
    for net, want in zip(nets, _alone()):
        for a, b in zip(_result(net), want):
            assert np.array_equal(a, b)
        net.close()


def test_on_threads():
    systems, got = _systems(), {}
    target = systems[0].xyz + np.float32(0.1)
    fit = W.ca_network(2000, seed=1)
    fit.config.update(precise_positions=1)

    def step(k):
        net = gpu_network(systems[k])
        for steps in (20, 3, 22):
            net.computeStep(steps)
        got[k] = _result(net)
        net.close()

    def adjoint(k):
        net = gpu_network(fit)
        got[k] = [net.adjoint(40, target, checkpoint=10) for _ in range(3)]
        net.close()

    threads = [threading.Thread(target=step, args=(k,)) for k in range(len(systems))]
    threads += [threading.Thread(target=adjoint, args=("fit",))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k, want in enumerate(_alone()):
        for a, b in zip(got[k], want):
            assert np.array_equal(a, b)
    net = gpu_network(fit)
    want = net.adjoint(40, target, checkpoint=10)
    for run in got["fit"]:
        for a, b in zip(run, want):
            assert np.array_equal(a, b)
    net.close()
