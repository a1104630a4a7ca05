"""The per-particle lists of link ends (ascending link index) for particles of fewer than, exactly
and more than the sixteen ends one pass sorts, and for none: the link states, the link-end history
and the forces they give against the oracle, links in shuffled order."""
from __future__ import annotations

import numpy as np
import pytest

from hidem_b200 import abi, workloads
from oracle import oracle
from test_gpu_parity import PRECS, assert_same, gpu_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", PRECS)
@pytest.mark.parametrize("spokes", [1, 15, 16, 17, 40])
def test_star(gpu, precision, spokes):
    rng = np.random.default_rng(spokes)
    lp = abi.lp_dtype(precision)
    n = spokes + 2  # the hub, its spokes, and one particle without links
    p = abi.empty_particles(n, precision)
    d = rng.normal(size=(n, 3))
    d *= (0.9 + 0.2 * rng.random((n, 1))) / np.linalg.norm(d, axis=1, keepdims=True)
    d[0], d[-1] = 0.0, (5.0, 5.0, 5.0)
    for k, f in enumerate(("xCord", "yCord", "zCord")):
        p[f][:] = d[:, k]
    for f in ("xDiff", "yDiff", "zDiff", "uDiff", "vDiff", "wDiff", "xTheta", "yTheta", "zTheta"):
        p[f][:] = rng.uniform(-1e-6, 1e-6, n).astype(lp)
    p["radius"][:] = 0.3
    p["globalKeys"][:] = np.arange(n)
    order = rng.permutation(spokes) + 1
    l = abi.empty_links(spokes, precision)
    hub_is_a = rng.random(spokes) < 0.5
    l["globalKeyEndA"][:] = np.where(hub_is_a, 0, order)
    l["globalKeyEndB"][:] = np.where(hub_is_a, order, 0)
    l["state"][:] = 1
    l["initialLen"][:] = np.linalg.norm(d[order], axis=1).astype(lp)
    P = workloads.block_params(precision, maxRadius=0.3, searchDistanceScale=4.0, maxLoad=1e-4)
    ref = oracle.port().run(P, p, l, 9)
    for kernel in (abi.STEP_KERNEL_TWO_PASS, abi.STEP_KERNEL_ITEMS):
        assert_same(gpu_run(P, p, l, 9, kernel=kernel), ref[0], ref[1], ref[3])
