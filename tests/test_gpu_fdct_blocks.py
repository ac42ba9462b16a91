"""The encoder's forward DCT with its one error bound per block (fdct_core.h kFdctBound,
fdct_round) under volume and adversarial input: the blocks of test_gpu_transform_stress.py,
which drives the bound per coefficient, through tests/cuda/fdct_harness.cu. Every quantised
coefficient equals the oracle's; every one within 2^-20 of a half-integer is left to the
binary64 order."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

import adversarial
import oracle
from helpers import report

pytestmark = [pytest.mark.gpu, pytest.mark.slow]

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_blocks_with_the_bound_of_the_whole_block(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = tmp_path / "libfdct_harness.so"
    p = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                        "-fPIC", "-I", os.path.join(ROOT, "mmrecode_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cuda", "fdct_harness.cu"), "-o", str(out)], capture_output=True, text=True)
    assert p.returncode == 0, p.stderr
    lib = ctypes.CDLL(str(out))
    lib.harness_fdct_block_bound.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_uint64] + [ctypes.c_void_p] * 2
    s, q, kinds, near = adversarial.fdct_blocks(20261213, n=600_000)
    rq = (1.0 / q.astype(np.float32)).astype(np.float32)  # as the encoder's host plan computes them
    gpu, exact = np.empty((len(s), 64), np.int32), ctypes.c_ulonglong(0)
    assert lib.harness_fdct_block_bound(s.ctypes.data, q.ctypes.data, rq.ctypes.data, len(s), gpu.ctypes.data,
                                        ctypes.byref(exact)) == 0
    bad = np.nonzero((gpu != oracle.fdct_quantize_many(s, q)).any(axis=1))[0]
    report("fdct_blocks_block_bound", blocks=len(s), near_ties_2e20=near, exact_coefficients=exact.value, kinds=kinds)
    assert len(bad) == 0, f"{len(bad)} of {len(s)} blocks differ, first {bad[:3]}"
    assert exact.value >= near
