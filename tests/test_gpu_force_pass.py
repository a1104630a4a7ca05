"""The two-pass step's force pass: sizes at the edges of its blocks of 32 slots, CTAs of 128
and the rule between its two variants, its folded link update against the break pass of the
split calls, and the geometries its shared-root evaluation hands to the plain IEEE operations.
Bit-exact against the oracle (or the split calls at sizes the oracle is slow at)."""
from __future__ import annotations

import numpy as np
import pytest

from hidem_b200 import abi, workloads
from hidem_b200.hidemlib import HiDEMBatch, HiDEMLib
from oracle import oracle
from test_gpu_parity import L_OUT, P_OUT, PRECS, assert_same, gpu_run

pytestmark = pytest.mark.gpu


# 4, 32, 36, 128, 132 and 1,500 particles: part of a block, whole blocks, part of a CTA
@pytest.mark.parametrize("precision", PRECS)
@pytest.mark.parametrize("cells", [(1, 1, 1), (2, 2, 2), (3, 3, 1), (2, 4, 4), (3, 11, 1), (15, 5, 5)])
def test_two_pass_sizes(gpu, precision, cells):
    P, p, l = workloads.ice_block(cells=cells, precision=precision, seed=8, gridRegenInterval=9)
    ref = oracle.port().run(P, p, l, 24)
    res = gpu_run(P, p, l, 24, kernel=abi.STEP_KERNEL_TWO_PASS)
    assert_same(res, ref[0], ref[1], ref[3])


# below and above the sizes where the variants change (75,776 particles mixed, 37,888 FP64)
@pytest.mark.parametrize("precision,cells", [(abi.PREC_MIXED, (29, 29, 22)), (abi.PREC_MIXED, (29, 29, 23)),
                                             (abi.PREC_FP64, (21, 21, 21)), (abi.PREC_FP64, (22, 21, 21))])
def test_two_pass_against_split_calls(gpu, precision, cells):
    P, p, l = workloads.ice_block(cells=cells, precision=precision, seed=9)
    fused = gpu_run(P, p, l, 14, kernel=abi.STEP_KERNEL_TWO_PASS)
    items = gpu_run(P, p, l, 14, kernel=abi.STEP_KERNEL_ITEMS)
    assert_same(fused, items[0], items[1], items[3])
    split = gpu_run(P, p, l, 14, mode="split")
    assert_same(fused, split[0], split[1], split[3])
    assert len(fused[3]) > 0


def _pair(precision, sep, **over):
    """Two bonded particles `sep` apart at a random attitude, spinning and drifting."""
    lp = abi.lp_dtype(precision)
    p = abi.empty_particles(2, precision)
    for k, f in enumerate(("xCord", "yCord", "zCord")):
        p[f][:] = [0.25, 0.25 + sep[k]]
    rng = np.random.default_rng(3)
    for f in P_OUT[3:]:
        p[f][:] = rng.uniform(-1e-6, 1e-6, 2).astype(lp)
    p["radius"][:] = 0.5
    p["globalKeys"][:] = [0, 1]
    l = abi.empty_links(1, precision)
    l["globalKeyEndA"][0], l["globalKeyEndB"][0] = 0, 1
    l["state"][0] = 1
    l["initialLen"][0] = np.float32(np.sqrt(np.sum(np.square(sep))))
    return workloads.block_params(precision, breakTime=1e9, **over), p, l


# vertical (no xy part), nearly vertical (its square outside the shared-root range), near
# coincidence, next to a length whose root rounds to all ones (the lengths themselves:
# test_lengths_the_shared_root_leaves_out), E W4 outside the admitted range
@pytest.mark.parametrize("precision", PRECS)
@pytest.mark.parametrize("sep,over", [((0.0, 0.0, 1.0), {}), ((1e-7, 0.0, 0.97), {}), ((1e-9, -1e-9, 0.9), {}),
                                      ((3e-7, 2e-7, 1e-7), {}), ((0.9999999, 0.0, 0.0), {}),
                                      ((0.0, 1.9999999, 0.0), {}), ((0.6, 0.5, 0.4), dict(E=1e-14)),
                                      ((0.6, 0.5, 0.4), dict(E=1e21))])
def test_geometries_outside_the_shared_root_range(gpu, precision, sep, over):
    P, p, l = _pair(precision, sep, **over)
    check_one_step(P, p, l)


def check_one_step(P, p, l):
    ref = oracle.port().run(P, p, l, 1)
    for kernel in (abi.STEP_KERNEL_TWO_PASS, abi.STEP_KERNEL_ITEMS, abi.STEP_KERNEL_THREAD):
        lib = HiDEMLib(P)
        lib.set_step_kernel(kernel)
        lib.set_particles(p)
        lib.set_links(l)
        lib.step(1)
        out, links = lib.get_particles(), lib.get_links()
        lib.close()
        for k in P_OUT:
            assert np.array_equal(out[k], ref[0][k], equal_nan=True), (k, kernel)
        for k in L_OUT:
            assert np.array_equal(links[k], ref[1][k], equal_nan=True), (k, kernel)


# The lengths at which the shared-root evaluation hands over to the IEEE operations, each shown to
# be one here: a squared length whose root rounds to all ones (the two largest floats below an even
# power of two), in contact and beyond it, as the whole length and as its part in the xy plane; and
# a length whose square rounds to all ones (every squared length of 2 or 1/2: 1 / sqrt(2) * 2 is one
# unit below sqrt(2)). No length's cube does: checked over every significand.
@pytest.mark.parametrize("sep,where", [((1 - 2.0 ** -24, 0.0, 0.0), "root"), ((0.0, 0.0, 1 - 2.0 ** -24), "length only"),
                                       ((0.0, 1 - 2.0 ** -24, 0.25), "plane only"), ((2 - 2.0 ** -23, 0.0, 0.0), "root"),
                                       ((0.5 - 2.0 ** -25, 0.0, 0.0), "root"), ((1.0, 1.0, 0.0), "square"),
                                       ((0.5, 0.0, 0.5), "square"), ((0.5, 0.25, 0.4330127018922193), "square")])
def test_lengths_the_shared_root_leaves_out(gpu, sep, where):
    f = np.float32
    x, y, z = (f(v) for v in sep)
    ones = lambda v: int(v.view(np.uint32)) & 0x7fffff == 0x7fffff  # noqa: E731
    xy = x * x + y * y
    D = xy + z * z
    length = (f(1) / np.sqrt(D)) * D
    root = ones(np.sqrt(D)), ones(np.sqrt(xy))
    assert root == {"root": (True, True), "length only": (True, False), "plane only": (False, True),
                    "square": (False, False)}[where]
    assert ones(length * length) or where != "square"
    check_one_step(*_pair(abi.PREC_MIXED, sep))


def test_no_length_has_a_cube_of_all_ones():
    m = np.arange(0x3f800000, 0x40000000, dtype=np.uint32).view(np.float32)  # the pattern repeats in every binade
    cube = (m * m) * m
    assert not np.any((cube.view(np.uint32) & 0x7fffff) == 0x7fffff)


# Initial lengths the quick test for an unbroken link must leave to the functor: negative with a
# bend beyond the threshold (the functor breaks where (S - L0) / L0 turns its sign), zero, so small
# that the squares lose digits, infinite; and ordinary ones on both sides of the threshold.
@pytest.mark.parametrize("precision", PRECS)
@pytest.mark.parametrize("bend", [0.0, 0.4, 5.0])
@pytest.mark.parametrize("length", [-1.0, -0.2, -5.0, 0.0, 1e-20, 1e-30, np.inf, 0.9995, 0.8, 2.0])
def test_break_decision_for_any_initial_length(gpu, precision, bend, length):
    P, p, l = _pair(precision, (0.6, 0.5, 0.62))
    P.breakTime, P.bendBreak, P.maxLoad = -1.0, 1.0, 0.5
    p["yTheta"][1] = bend
    l["initialLen"][0] = length
    ref = oracle.port().run(P, p, l, 3)
    for kernel in (abi.STEP_KERNEL_TWO_PASS, abi.STEP_KERNEL_ITEMS, abi.STEP_KERNEL_THREAD):
        out_p, out_l, _, events, _ = gpu_run(P, p, l, 3, kernel=kernel)
        assert np.array_equal(events.reshape(-1, 2), np.asarray(ref[3]).reshape(-1, 2)), kernel
        for k in P_OUT:
            assert np.array_equal(out_p[k], ref[0][k], equal_nan=True), (k, kernel)
        for k in L_OUT:
            assert np.array_equal(out_l[k], ref[1][k], equal_nan=True), (k, kernel)
    # the batch's break pass
    lib = HiDEMLib(P)
    lib.set_particles(p)
    lib.set_links(l)
    with HiDEMBatch([lib]) as batch:
        batch.step(3)
    li, st = lib.get_break_events()
    assert np.array_equal(np.stack([li, st], axis=1).reshape(-1, 2), np.asarray(ref[3]).reshape(-1, 2))
    lib.close()
