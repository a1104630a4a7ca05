"""Readback into host arrays, device arrays and a mix of both, some fields left out, and into
device arrays that are not aligned for their values: the same values everywhere."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from hidem_b200 import abi, workloads
from hidem_b200.hidemlib import HiDEMLib

pytestmark = pytest.mark.gpu

LINK_OUT = ["state", "initialLen", "globalKeyEndA", "globalKeyEndB"] + abi.SIDE_FIELDS


@pytest.mark.parametrize("precision", [abi.PREC_MIXED, abi.PREC_FP64])
@pytest.mark.parametrize("cells", [(1, 1, 1), (5, 3, 3)])
def test_destinations(gpu, precision, cells):
    import torch
    P, p, l = workloads.ice_block(cells=cells, precision=precision, seed=4)
    lib = HiDEMLib(P)
    lib.set_particles(p)
    lib.set_links(l)
    lib.step(12)
    host_p, host_l = lib.get_particles(), lib.get_links()
    dev_p, dev_l = lib.get_particles_device(), lib.get_links_device()
    for k in abi.PARTICLE_FIELDS:
        assert np.array_equal(dev_p[k].cpu().numpy(), host_p[k]), k
    for k in LINK_OUT:
        assert np.array_equal(dev_l[k].cpu().numpy(), host_l[k]), k
    dev = torch.device("cuda", 0)
    mix_p, mix_l = abi.empty_particles_torch(lib.n, precision, dev), abi.empty_links_torch(lib.L, precision, dev)
    for k in ("yCord", "wDiff", "type"):
        mix_p[k] = np.zeros_like(host_p[k])
    for k in ("xTheta", "radius"):
        del mix_p[k]
    for k in ("CT1", "CT4", "state"):
        mix_l[k] = np.zeros_like(host_l[k])
    del mix_l["CT0"]
    lib.get_particles(mix_p)
    lib.get_links(mix_l)
    value = lambda v: v.cpu().numpy() if hasattr(v, "cpu") else v  # noqa: E731
    for k, v in mix_p.items():
        assert np.array_equal(value(v), host_p[k]), k
    for k, v in mix_l.items():
        if k in LINK_OUT:
            assert np.array_equal(value(v), host_l[k]), k
    # two bytes past an aligned address
    lp = np.dtype(abi.lp_dtype(precision))
    raw = torch.zeros(lib.L * 2 * lp.itemsize + 64, dtype=torch.uint8, device=dev)
    raw_x = torch.zeros(lib.n * 8 + 64, dtype=torch.uint8, device=dev)
    psoa, lsoa = abi.HidemParticleSoA(), abi.HidemLinkSoA()
    psoa.xCord = raw_x.data_ptr() + 2
    lsoa.CT[3] = raw.data_ptr() + 2
    lib._check(lib._lib.hidem_get_particles(lib._ctx, C.byref(psoa)))
    lib._check(lib._lib.hidem_get_links(lib._ctx, C.byref(lsoa)))
    got_x = raw_x[2:2 + lib.n * 8].cpu().numpy().tobytes()
    got_ct = raw[2:2 + lib.L * 2 * lp.itemsize].cpu().numpy().tobytes()
    assert got_x == host_p["xCord"].tobytes() and got_ct == host_l["CT3"].tobytes()
    lib.close()
