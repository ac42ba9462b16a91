"""GPU encoder, the sizes its prefix sums change form at: up to and past 4096 tiles of 128
blocks, segments, and sums of stuffing counts, frames and restart intervals ending inside a
tile. Every byte equals the CPU encoder's."""
import numpy as np
import pytest

import mmrecode_gb300 as m
from mmrecode_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,sub,n,ri", [
    (1920, 1080, "422", 9, 0),    # more than 4096 tiles
    (1920, 1080, "422", 9, 120),
    (1024, 1032, "444", 1, 1),    # more than 4096 segments
    (1024, 1032, "444", 1, 4),
    (1000, 520, "420", 2, 7),
    (40, 24, "420", 3, 1),
    (8, 8, "444", 1, 0),
])
def test_every_byte_equals_the_cpu_encoder(w, h, sub, n, ri):
    frame = synth.mjpeg_frame(3, 0, w, h, sub)
    noise = np.random.default_rng(3).integers(0, 256, w * min(h, 64), dtype=np.uint8).tobytes()
    frame.planes[0].data = noise + bytes(frame.planes[0].data)[len(noise):]  # (more 0xFF bytes)
    ref = m.encode_jpeg(frame, 92, True, ri)
    with m.Context() as ctx:
        for status, message, data in ctx.encode_jpeg_batch([frame] * n, 92, True, ri):
            assert status == 0, message
            assert data == ref
