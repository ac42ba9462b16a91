"""Host planes of an encode batch that touch in memory go up as one copy, except across
pinned buffers of different owners (mmrecode_gb300/csrc/plane_uploads.h)."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def copies(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    so = tmp_path_factory.mktemp("uploads") / "plane_uploads_harness.so"
    subprocess.run([gxx, "-O1", "-shared", "-fPIC", "-std=c++17", f"-I{ROOT / 'mmrecode_gb300' / 'csrc'}",
                    "-o", str(so), str(ROOT / "tests" / "cuda" / "plane_uploads_harness.cpp")], check=True)
    lib = ctypes.CDLL(str(so))
    lib.mmr_test_plane_uploads.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t] * 2 + [ctypes.c_void_p]

    def run(planes, ranges):
        at, size = (np.array([p[k] for p in planes], np.uint64) for k in (0, 1))
        lo, hi = (np.array([r[k] for r in ranges] or [0], np.uint64) for k in (0, 1))
        out = np.zeros(len(planes), np.uint32)
        lib.mmr_test_plane_uploads(at.ctypes.data, size.ctypes.data, len(planes), lo.ctypes.data, hi.ctypes.data,
                                   len(ranges), out.ctypes.data)
        return out.tolist()
    return run


P = 0x10000  # planes of one page, at pages 0, 1, 2, ...


def page(i, n=1):
    return (P + 4096 * i, 4096 * n)


@pytest.mark.parametrize("ranges,expect", [
    ([], [0, 0, 0, 0]),                                              # ordinary memory
    ([(0, 4)], [0, 0, 0, 0]),                                        # one pinned buffer
    ([(0, 2), (2, 4)], [0, 0, 1, 1]),                                # two
    ([(0, 1), (1, 2), (2, 3), (3, 4)], [0, 1, 2, 3]),
    ([(0, 2)], [0, 0, 1, 1]),                                        # pinned, then ordinary
    ([(2, 4)], [0, 0, 1, 1]),                                        # ordinary, then pinned
    ([(1, 2)], [0, 1, 2, 2]),
])
def test_no_copy_spans_two_owners(copies, ranges, expect):
    pinned = [(P + 4096 * a, P + 4096 * b) for a, b in ranges]
    assert copies([page(i) for i in range(4)], pinned) == expect
    # planes that do not follow one another never share a copy
    assert copies([page(0), page(2), page(1), page(3)], pinned) == [0, 1, 2, 3]


def test_a_plane_that_ends_past_its_buffer_is_not_joined(copies):
    assert copies([page(0), page(1, 2)], [(P, P + 2 * 4096)]) == [0, 1]
    assert copies([page(0), page(1, 1), page(2, 1)], [(P, P + 2 * 4096 + 100)]) == [0, 0, 1]
