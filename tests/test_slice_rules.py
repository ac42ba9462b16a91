"""Rules of the chunked entropy decoder (mmrecode_gb300/csrc/plan.h) that hold for any
state a damaged scan may leave behind, checked on the host."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    so = tmp_path_factory.mktemp("slice") / "slice_harness.so"
    subprocess.run([gxx, "-O1", "-shared", "-fPIC", "-std=c++17", f"-I{ROOT / 'mmrecode_gb300' / 'csrc'}",
                    "-o", str(so), str(ROOT / "tests" / "cuda" / "slice_harness.cpp")], check=True)
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("sched_len", [1, 3, 6, 10, 64])
def test_no_slice_decodes_past_its_intervals_last_mcu(lib, sched_len):
    """The final decode starts at MCU base / sched_len, block si, and takes one block after
    the other: whatever si and base are, the last one lies in the interval; where they
    agree (every slice of a valid scan) no block is left out."""
    share = lib.mmr_test_slice_share
    for mcus in (1, 2, 5):
        blocks = mcus * sched_len
        for base in list(range(blocks + 2)) + [0xFFFFFFFF]:
            for si in range(sched_len):
                for n in (0, 1, sched_len, blocks - 1, blocks, 0xFFFFFFFF):
                    got = share(n, base, blocks, si, sched_len) & 0xFFFFFFFF
                    if got:
                        assert base // sched_len * sched_len + si + got <= blocks, (base, si, n, got)
                    if base < blocks and si == base % sched_len:
                        assert got == min(n, blocks - base), (base, si, n, got)
