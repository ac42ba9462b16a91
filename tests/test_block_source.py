"""The encoder reads a block's samples from its plane's storage alone, whatever the plane's
address, stride and size are (mmrecode_gb300/csrc/block_source.h)."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    so = tmp_path_factory.mktemp("rows") / "block_source_harness.so"
    subprocess.run([gxx, "-O1", "-shared", "-fPIC", "-std=c++17", f"-I{ROOT / 'mmrecode_gb300' / 'csrc'}",
                    "-o", str(so), str(ROOT / "tests" / "cuda" / "block_source_harness.cpp")], check=True)
    lib = ctypes.CDLL(str(so))
    lib.mmr_test_source_row.restype = ctypes.c_uint64
    lib.mmr_test_source_row.argtypes = [ctypes.c_void_p, ctypes.c_size_t] + [ctypes.c_uint32] * 5 + [ctypes.c_void_p]
    return lib


@pytest.mark.parametrize("offset", range(8))
@pytest.mark.parametrize("pw,ph,extra", [(8, 8, 0), (8, 1, 0), (9, 3, 0), (16, 9, 0), (17, 8, 5), (20, 3, 3), (24, 2, 0), (24, 2, 8), (31, 2, 0), (40, 9, 1), (1, 1, 0), (7, 7, 1)])
def test_rows_are_read_inside_the_plane(lib, offset, pw, ph, extra):
    stride = pw + extra
    store = np.random.default_rng(offset).integers(0, 256, stride * ph + 64, dtype=np.uint8)
    first = (-store.ctypes.data) % 8 + 8 + offset
    plane = store[first:first + stride * ph].reshape(ph, stride)
    outside = ctypes.c_uint32()
    for y0 in range(0, ph + 8, 8):
        for x0 in range(0, pw + 8, 8):
            for r in range(8):
                v = lib.mmr_test_source_row(plane.ctypes.data, stride, pw, ph, x0, y0, r, ctypes.byref(outside))
                row = plane[min(y0 + r, ph - 1)]
                assert v == sum(int(row[min(x0 + x, pw - 1)]) << (8 * x) for x in range(8)), (x0, y0, r)
                assert outside.value == 0, (x0, y0, r)
