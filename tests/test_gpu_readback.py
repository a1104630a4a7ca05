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


# arrays that overlap (a buffer for fields that are not looked at, views into one allocation): the
# later field's values stand where two meet, whether the first lies there whole, in part or in
# another type
@pytest.mark.parametrize("precision", [abi.PREC_MIXED, abi.PREC_FP64])
@pytest.mark.parametrize("cells", [(5, 3, 3), (23, 11, 9)])
def test_overlapping_destinations(gpu, precision, cells):
    import torch
    P, p, l = workloads.ice_block(cells=cells, precision=precision, seed=4)
    lib = HiDEMLib(P)
    lib.set_particles(p)
    lib.set_links(l)
    lib.step(12)
    host_p, host_l = lib.get_particles(), lib.get_links()
    n, L, lp = lib.n, lib.L, np.dtype(abi.lp_dtype(precision)).itemsize
    # fields in the order of the reads, each with the byte its array starts at
    fields = [("xCord", 0), ("yCord", 8 * (n // 3)), ("uDiff", 8 * (n // 2)), ("xTheta", 8 * (n // 2) + lp * (n // 4)),
              ("type", 16 * (n // 5))]
    ends = [("CT0", 0), ("CT1", lp * (L // 3)), ("CT4", lp * L), ("state", lp * (L // 2))]
    psoa, lsoa = abi.HidemParticleSoA(), abi.HidemLinkSoA()
    for soa, read, order, host in ((psoa, lib._lib.hidem_get_particles, fields, host_p),
                                   (lsoa, lib._lib.hidem_get_links, ends, host_l)):
        room = max(at + host[k].nbytes for k, at in order)
        dev = torch.zeros(room, dtype=torch.uint8, device="cuda")
        want = np.zeros(room, np.uint8)
        torch.cuda.synchronize()
        for k, at in order:
            want[at:at + host[k].nbytes] = host[k].view(np.uint8)
            if k.startswith("CT"):
                soa.CT[int(k[2])] = dev.data_ptr() + at
            else:
                setattr(soa, k, dev.data_ptr() + at)
        for _ in range(3):
            lib._check(read(lib._ctx, C.byref(soa)))
            assert np.array_equal(dev.cpu().numpy(), want)
    lib.close()
