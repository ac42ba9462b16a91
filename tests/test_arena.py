"""Device memory of decode batches (mmrecode_gb300/csrc/arena.h): a server's batch stays
within what it reserved for its requests, whatever their size, rate and restart interval;
requests are reserved what they always were where that is enough."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


class Frame(ctypes.Structure):
    _fields_ = [(k, ctypes.c_uint64) for k in ("len", "planar", "blocks", "intervals", "planes", "host_out")]


@pytest.fixture(scope="module")
def arena(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    so = tmp_path_factory.mktemp("arena") / "arena_harness.so"
    subprocess.run([gxx, "-O1", "-shared", "-fPIC", "-std=c++17", f"-I{ROOT / 'mmrecode_gb300' / 'csrc'}",
                    "-o", str(so), str(ROOT / "tests" / "cuda" / "arena_harness.cpp")], check=True)
    lib = ctypes.CDLL(str(so))

    def run(frames, limited):
        a, out = (Frame * len(frames))(*frames), (ctypes.c_uint64 * 4)()
        lib.mmr_test_arena(a, ctypes.c_size_t(len(frames)), int(limited), out)
        return list(out)
    return run


FACTORS = {"gray": [(1, 1)], "420": [(2, 2), (1, 1), (1, 1)], "422": [(2, 1), (1, 1), (1, 1)], "444": [(1, 1)] * 3,
           "444 as 2x2": [(2, 2)] * 3}


def frame(w, h, sub, bits_per_sample, ri, rgb=False):
    fs = FACTORS[sub]
    hm, vm = (max(f[k] for f in fs) for k in (0, 1))
    mcu = (8, 8) if sub == "gray" else (8 * hm, 8 * vm)
    cols, rows = -(-w // mcu[0]), -(-h // mcu[1])
    planar = sum(-(-w * a // hm) * -(-h * b // vm) for a, b in fs)
    blocks = cols * rows * (1 if sub == "gray" else sum(a * b for a, b in fs))
    ri = {"none": cols * rows, "row": cols}.get(ri, ri)
    return Frame(int(planar * bits_per_sample / 8) + 600, planar, blocks, -(-cols * rows // ri), int(rgb and sub != "420"),
                 3 * w * h if rgb else planar)


SIZES = [(16, 16), (64, 48), (320, 240), (719, 405), (1920, 1080), (4096, 2160), (1, 4000), (4000, 1)]


@pytest.mark.parametrize("sub", FACTORS)
@pytest.mark.parametrize("ri", ["none", "row", 1, 2])
def test_batches_stay_within_what_was_reserved(arena, sub, ri):
    for w, h in SIZES:
        for rate in (0.1, 1.0, 4.0, 8.0):
            for rgb in (False, True):
                for n in (1, 2, 16):
                    reserved, taken, _, _ = arena([frame(w, h, sub, rate, ri, rgb)] * n, True)
                    assert taken <= reserved, (w, h, rate, rgb, n)


def test_unlike_frames_together(arena):
    frames = [frame(w, h, sub, rate, ri) for (w, h), sub, rate, ri in
              zip(SIZES * 3, list(FACTORS) * 5, (0.3, 6.0, 2.0, 1.0, 8.0) * 5, ("none", 1, "row", 2) * 6)]
    for n in (2, 5, 24):
        reserved, taken, _, _ = arena(frames[:n], True)
        assert taken <= reserved, n


@pytest.mark.parametrize("w,h,sub,rate,ri", [(1920, 1080, "420", 4.0, "none"), (320, 240, "420", 1.0, "none"), (640, 480, "420", 1.2, 1)])
def test_several_guesses_only_where_they_fit(arena, w, h, sub, rate, ri):
    f = frame(w, h, sub, rate, ri)
    reserved, taken, unlimited, paths = arena([f], True)
    assert unlimited > reserved >= taken and paths == 1
    assert arena([f], False)[1:] == [unlimited, unlimited, 6]  # without a budget they are taken
    roomy = frame(1920, 1080, "422", 0.2, "row")
    assert arena([roomy], True)[3] == 6


def test_ordinary_requests_are_reserved_what_they_were(arena):
    for f in (frame(1920, 1080, "422", 2.2, "row", True), frame(320, 240, "420", 1.0, "none"), frame(4096, 2160, "444", 3.0, 4)):
        assert arena([f], True)[0] == 8 * f.len + f.planar * 9 // 2 + f.planar + 65536 + f.host_out
