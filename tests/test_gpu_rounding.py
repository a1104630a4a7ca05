"""The mixed build's roots, reciprocals and quotients from one shared approximate reciprocal
root (physics.cuh) against the IEEE operations they stand for: every significand, both
exponent parities, at exponents across the admitted range; no mismatch is allowed."""
from __future__ import annotations

import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest


@pytest.fixture(scope="module")
def harness(tmp_path_factory, gpu):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = tmp_path_factory.mktemp("rounding") / "librounding.so"
    here = Path(__file__).resolve().parent
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-fmad=false",
                    "-prec-div=true", "-prec-sqrt=true", "-ftz=false", "-shared", "-Xcompiler", "-fPIC",
                    f"-I{here.parent / 'include'}", "-o", str(out), str(here / "rounding_harness.cu")], check=True)
    h = C.CDLL(str(out))
    h.rounding_mismatches.argtypes = [C.c_uint, C.c_uint, C.POINTER(C.c_ulonglong)]
    return h


# two binades from 2^e: the ends of the root range (2^-90 .. 2^90 for the contact's cube,
# 2^-40 .. 2^40 for lengths, whose powers the quotients divide by) and lengths near 1
@pytest.mark.gpu
@pytest.mark.parametrize("exponent", [-90, -60, -40, -1, 0, 38, 58, 88])
def test_every_significand(harness, exponent):
    bad = (C.c_ulonglong * 4)()
    assert harness.rounding_mismatches((127 + exponent) << 23, 12345 + exponent, bad) == 0
    # the reciprocals and quotients are used for arguments in [2^-60, 2^60]
    n = 4 if -60 <= exponent <= 58 else 1
    assert list(bad)[:n] == [0] * n, list(bad)
