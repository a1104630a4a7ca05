"""The device pool keeps what one context gives back for the next one, up to a stated share of the
device's memory: a job after another maps nothing anew, and no more than that share is held."""
from __future__ import annotations

import ctypes as C

import pytest

from hidem_b200 import abi, workloads
from hidem_b200.hidemlib import HiDEMLib

pytestmark = pytest.mark.gpu

RELEASE_THRESHOLD, RESERVED_CURRENT, RESERVED_HIGH = 4, 5, 6  # CUmemPool_attribute


def pool_attribute(which, value=None):
    cuda = C.CDLL("libcuda.so.1")
    pool, out = C.c_void_p(), C.c_uint64(0 if value is None else value)
    assert cuda.cuDeviceGetDefaultMemPool(C.byref(pool), C.c_int(0)) == 0
    call = cuda.cuMemPoolGetAttribute if value is None else cuda.cuMemPoolSetAttribute
    assert call(pool, C.c_int(which), C.byref(out)) == 0
    return out.value


def test_jobs_after_the_first_map_nothing(gpu):
    import torch
    P, p, l = workloads.ice_block(cells=(40, 40, 30), precision=abi.PREC_FP64, seed=2)
    total = torch.cuda.mem_get_info()[1]

    def job():
        with HiDEMLib(P) as lib:
            for _ in range(2):  # a second set of the same size in the same context
                lib.set_timestep(0)
                lib.set_particles(p)
                lib.set_links(l)
                lib.step(12)
                lib.get_links()
    job()
    assert pool_attribute(RELEASE_THRESHOLD) >= max(8 << 30, total // 8)
    held = pool_attribute(RESERVED_CURRENT)
    pool_attribute(RESERVED_HIGH, 0)  # from here on
    job()
    assert pool_attribute(RESERVED_CURRENT) == held == pool_attribute(RESERVED_HIGH)


def test_a_threshold_the_caller_raised_stays(gpu):
    before = pool_attribute(RELEASE_THRESHOLD)
    more = 3 * (before // 2)
    try:
        pool_attribute(RELEASE_THRESHOLD, more)
        HiDEMLib(abi.default_params()).close()
        assert pool_attribute(RELEASE_THRESHOLD) == more
    finally:
        pool_attribute(RELEASE_THRESHOLD, before)
