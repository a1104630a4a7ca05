"""Rebuilds that move the link ends from one slot layout to the next: after particles have
changed cells, at sizes around the blocks of 32, and after a rebuild that failed midway."""
from __future__ import annotations

import numpy as np
import pytest

from hidem_b200 import abi, workloads
from hidem_b200.hidemlib import HiDEMBatch, HiDEMLib
from oracle import oracle
from test_gpu_parity import L_OUT, P_OUT, PRECS, assert_same, gpu_run

pytestmark = pytest.mark.gpu


# an unsupported, spinning-up block whose particles change cells (and slots) between rebuilds
@pytest.mark.parametrize("precision", PRECS)
@pytest.mark.parametrize("cells", [(1, 1, 1), (2, 2, 2), (3, 3, 1), (5, 4, 3)])
def test_moving_particles(gpu, precision, cells):
    P, p, l = workloads.ice_block(cells=cells, precision=precision, seed=6, fixed_bottom=False, g=-2e6,
                                  gridRegenInterval=3)
    ref = oracle.port().run(P, p, l, 25)
    for kernel in (abi.STEP_KERNEL_TWO_PASS, abi.STEP_KERNEL_ITEMS):
        assert_same(gpu_run(P, p, l, 25, kernel=kernel), ref[0], ref[1], ref[3])


@pytest.mark.parametrize("precision", PRECS)
def test_rebuild_after_a_failed_one(gpu, precision):
    P, p, l = workloads.ice_block(cells=(12, 12, 12), precision=precision, seed=5, g=-1e5)
    out = []
    for fail in (True, False):
        lib = HiDEMLib(P)
        lib.set_particles(p)
        lib.set_links(l)
        lib.step(8)
        if fail:
            wide = abi.HidemParams.from_buffer_copy(P)
            wide.searchDistanceScale = 20.0  # every particle in one cell: refused after the sort
            lib.set_params(wide)
            with pytest.raises(abi.HidemError) as e:
                lib.regenerate()
            assert e.value.status == abi.HIDEM_ERR_CAPACITY
            lib.set_params(P)
        lib.regenerate()
        lib.step(8)
        out.append((lib.get_particles(), lib.get_links(), lib.get_neighbours()[0]))
        lib.close()
    for k in P_OUT:
        assert np.array_equal(out[0][0][k], out[1][0][k]), k
    for k in L_OUT:
        assert np.array_equal(out[0][1][k], out[1][1][k]), k
    assert np.array_equal(out[0][2], out[1][2])


# a run that ends in a refused rebuild leaves the state of the steps before it, their link
# updates included
@pytest.mark.parametrize("precision", PRECS)
@pytest.mark.parametrize("kernel", [abi.STEP_KERNEL_TWO_PASS, abi.STEP_KERNEL_ITEMS])
def test_run_that_ends_in_a_refused_rebuild(gpu, precision, kernel):
    P, p, l = workloads.ice_block(cells=(4, 4, 4), precision=precision, seed=7, g=-2e6, gridRegenInterval=8)
    p["zDiff"][-1] = 60.0  # leaves the block: the grid of step 8 has far more cells
    out = []
    for steps in (16, 8):
        lib = HiDEMLib(P)
        lib.set_step_kernel(kernel)
        lib.set_checks(abi.CHECK_GRID_GROWTH)
        lib.set_particles(p)
        lib.set_links(l)
        if steps == 16:
            with pytest.raises(abi.HidemError) as e:
                lib.step(16)
            assert e.value.status == abi.HIDEM_ERR_DEVICE
        else:
            lib.step(8)
        li, st = lib.get_break_events()
        out.append((lib.get_particles(), lib.get_links(), sorted(zip(li.tolist(), st.tolist()))))
        lib.close()
    for k in P_OUT:
        assert np.array_equal(out[0][0][k], out[1][0][k], equal_nan=True), k
    for k in L_OUT:
        assert np.array_equal(out[0][1][k], out[1][1][k], equal_nan=True), k
    assert out[0][2] == out[1][2] and len(out[0][2]) > 0


# what follows a rebuild that failed midway starts with a rebuild of its own: the lists of the
# layout before it are not read in the new slot order
@pytest.mark.parametrize("precision", PRECS)
@pytest.mark.parametrize("batched", [False, True])
def test_steps_after_a_failed_rebuild(gpu, precision, batched):
    P, p, l = workloads.ice_block(cells=(12, 12, 12), precision=precision, seed=5, g=-1e5)
    out = []
    for fail in (True, False):
        lib = HiDEMLib(P)
        lib.set_particles(p)
        lib.set_links(l)
        lib.step(8)
        if fail:
            wide = abi.HidemParams.from_buffer_copy(P)
            wide.searchDistanceScale = 20.0
            lib.set_params(wide)
            with pytest.raises(abi.HidemError):
                lib.regenerate()
            with pytest.raises(abi.HidemError):  # refused again, not answered from the old lists
                lib.computePartForce()
            with pytest.raises(abi.HidemError):
                lib.get_neighbours()
            lib.set_params(P)
        else:
            lib.regenerate()
        if batched:
            with HiDEMBatch([lib]) as batch:
                batch.step(9)
        else:
            lib.step(9)
        out.append((lib.get_particles(), lib.get_links(), lib.get_neighbours()[0]))
        lib.close()
    for k in P_OUT:
        assert np.array_equal(out[0][0][k], out[1][0][k]), k
    for k in L_OUT:
        assert np.array_equal(out[0][1][k], out[1][1][k]), k
    assert np.array_equal(out[0][2], out[1][2])
