"""AUTO's step kernel belongs to the particle set it was chosen for: a context that is given a
set of another size times its kernels again, and a batch does not take over what a small first
context timed on itself."""
from __future__ import annotations

import pytest

from hidem_b200 import abi, workloads
from hidem_b200.hidemlib import HiDEMBatch, HiDEMLib

pytestmark = pytest.mark.gpu

TIMED = (abi.STEP_KERNEL_ITEMS, abi.STEP_KERNEL_TWO_PASS)


def block(cells):
    return workloads.ice_block(cells=cells, precision=abi.PREC_MIXED, seed=3)


# 65,536 and 65,600 particles: the largest timed set and one above it
def test_choice_follows_the_particle_set(gpu):
    small, other, border, large = block((4, 4, 4)), block((5, 4, 4)), block((32, 32, 16)), block((41, 20, 20))
    assert border[1]["xCord"].shape[0] == 65536 and large[1]["xCord"].shape[0] == 65600
    with HiDEMLib(small[0]) as lib:
        for _, p, l in (small, large, small, other, border):
            lib.set_particles(p)
            lib.set_links(l)
            if p["xCord"].shape[0] > 65536:
                assert lib.step_kernel() == abi.STEP_KERNEL_TWO_PASS
                lib.step(1)
                assert lib.step_kernel() == abi.STEP_KERNEL_TWO_PASS
                continue
            assert lib.step_kernel() == abi.STEP_KERNEL_AUTO
            lib.step(9)
            assert lib.step_kernel() == abi.STEP_KERNEL_AUTO
            lib.step(1)
            assert lib.step_kernel() in TIMED
        # the same size again keeps the choice
        kept = lib.step_kernel()
        lib.set_particles(border[1])
        lib.set_links(border[2])
        assert lib.step_kernel() == kept


# one small block that has timed itself beside a large one: the two-pass step, three launches a
# step; alone, the batch takes the block's own choice
def test_batch_decides_by_its_total(gpu):
    small, large = block((4, 4, 4)), block((41, 20, 20))
    libs = []
    for P, p, l in (small, large):
        lib = HiDEMLib(P)
        lib.set_particles(p)
        lib.set_links(l)
        libs.append(lib)
    libs[0].step(10)
    kernel = libs[0].step_kernel()
    assert kernel in TIMED
    for members, per_step in ((libs, 3), (libs[:1], 3 if kernel == abi.STEP_KERNEL_TWO_PASS else 1)):
        with HiDEMBatch(members) as batch:
            batch.step(5)
            assert batch.counts()["launches"] == 5 * per_step
    for lib in libs:
        lib.close()
