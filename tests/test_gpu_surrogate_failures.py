"""A training step that fails on the host (a tensor map the driver refuses, at each one a step
encodes) leaves no work behind on the streams the backward pass forks onto, and the next step
gives what it would have given without the failures."""
from __future__ import annotations

import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from hidem_b200 import abi
from hidem_b200 import surrogate as sg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def harness(tmp_path_factory, gpu):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = tmp_path_factory.mktemp("surrogate") / "libsurrogate.so"
    here = Path(__file__).resolve().parent
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2", "-shared", "-Xcompiler",
                    "-fPIC", f"-I{here.parent / 'include'}", "-o", str(out),
                    str(here / "surrogate_failure_harness.cu")], check=True)
    h = C.CDLL(str(out))
    for name in ("hidem_surrogate_create", "hidem_surrogate_destroy", "hidem_surrogate_get_params",
                 "hidem_surrogate_set_data", "hidem_surrogate_num_params"):
        declared = getattr(abi.load(), name)
        getattr(h, name).argtypes, getattr(h, name).restype = declared.argtypes, declared.restype
    h.step_encodings.argtypes = [C.c_void_p]
    h.failed_step.argtypes = [C.c_void_p, C.c_int]
    return h


def open_net(h, cfg, u, t):
    s = C.c_void_p()
    assert h.hidem_surrogate_create(C.byref(cfg), 0, C.byref(s)) == 0
    assert h.hidem_surrogate_set_data(s, u.ctypes.data, t.ctypes.data, u.shape[0]) == 0
    return s


def params(h, s):
    out = np.empty(h.hidem_surrogate_num_params(s), np.float32)
    assert h.hidem_surrogate_get_params(s, out.ctypes.data) == 0
    return out


# a batch whose side streams have milliseconds of work when the failure comes
def test_failed_step_joins_its_streams(harness):
    h = harness
    cfg = sg.default_config(batch=1 << 17, inputs=82, fourier_bands=4, seed=4)
    rng = np.random.default_rng(1)
    u = rng.uniform(-1, 1, (4096, 82)).astype(np.float32)
    t = np.tanh(u[:, :3] + u[:, 3:6])
    a, b = open_net(h, cfg, u, t), open_net(h, cfg, u, t)
    count = h.step_encodings(a)
    assert count > 20  # the forward pass's, and two or three for each GEMM of the backward pass
    assert h.step_encodings(b) == count
    assert [h.failed_step(a, k) for k in range(count)] == [0] * count
    assert h.step_encodings(a) == h.step_encodings(b) == count
    pa, pb = params(h, a), params(h, b)
    assert np.array_equal(pa, pb) and np.isfinite(pa).all()
    for s in (a, b):
        h.hidem_surrogate_destroy(s)
