"""bs_nonbonded_forces_noalloc at the edges of its work split: the warps that share a group of homes
change at 5,000 and 10,000 particles, a group holds 4 homes, a window 32 partners. Against
the oracle, forces 1e-5 relative L2, energies 1e-5 relative plus the oracle's own distance to FP64."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from biospring_gb300 import capi
from biospring_gb300 import workloads as W
from helpers import rel_l2
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _call(s, cfg):
    torch = pytest.importorskip("torch")
    fn = capi.load().bs_nonbonded_forces_noalloc
    fn.restype = C.c_int
    fn.argtypes = [C.POINTER(capi.BsConfig), C.c_int64] + [C.c_void_p] * 9 + [C.c_char_p, C.c_size_t]
    d = [torch.from_numpy(np.ascontiguousarray(a).reshape(-1).copy()).cuda()
         for a in (s.xyz, s.radius, s.epsilon, s.charge, s.hydrophobicity, s.is_static)]
    f = torch.full((s.n, 3), float("nan"), device="cuda")
    e = torch.full((6,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert fn(C.byref(cfg), s.n, *[t.data_ptr() for t in d], f.data_ptr(), e.data_ptr(), None, None, 0) == capi.BS_OK
    torch.cuda.synchronize()
    return f.cpu().numpy(), e.cpu().numpy()


@pytest.mark.parametrize("n,mode,dense", [(2, 1, 0), (5, 0, 1), (31, 2, 1), (33, 1, 1), (260, 3, 1), (2500, 1, 0),
                                          (2501, 0, 0), (4999, 2, 0), (5001, 3, 0), (10001, 1, 0)])
def test_split_edges(n, mode, dense):
    """dense: all particles inside one cutoff, so that every queue fills and empties."""
    cfg = dict(spring_enable=0, steric_enable=1, steric_mode=mode, steric_cutoff=60.0 if dense else 9.0, coulomb_enable=1,
               coulomb_cutoff=60.0 if dense else 12.0, coulomb_dielectric=4.0, hydrophobicity_enable=1,
               hydrophobicity_cutoff=8.0)
    rng = np.random.default_rng(n)
    xyz = W.rsa_fill(n, max(9.0, (n / 0.02) ** (1.0 / 3.0) + 3.0), 3.0, 50 + n)
    s = W.System("direct", xyz, np.zeros((0, 2), np.int32), np.zeros(0, np.float32), np.zeros(0, np.float32), cfg,
                 radius=rng.uniform(1.5, 2.0, n).astype(np.float32),
                 epsilon=rng.uniform(0.1, 0.3, n).astype(np.float32),
                 charge=np.where(rng.random(n) < 0.5, 1.0, 0.0).astype(np.float32),
                 hydrophobicity=np.where(rng.random(n) < 0.5, 0.5, 0.0).astype(np.float32),
                 is_static=(rng.random(n) < 0.1).astype(np.uint8))
    s.is_static[0] = 0
    f, e = _call(s, po.oracle_config(s))
    orc = po.Oracle(s)
    orc.compute_forces()
    fr, er = orc.forces(), orc.energies()
    _, e64 = orc.eval_fp64()
    orc.close()
    dyn = s.is_static == 0
    assert rel_l2(f, fr, dyn) < 1e-5 and np.all(f[~dyn] == 0.0)
    for k in range(6):
        assert abs(e[k] - er[k]) <= 1e-5 * abs(er[k]) + abs(er[k] - e64[k]), (k, e[k], er[k], e64[k])
