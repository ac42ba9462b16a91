"""Chunked entropy decode at grid sizes where its threads are spread over more warps: one
thread in four, one in two, or every thread takes a slice (a small frame fills one CTA of
slices). Every status and sample equals the oracle decoder's."""
import pytest

import mmrecode_gb300 as m
import oracle
from helpers import assert_same_decode, frame_planes_gpu
from mmrecode_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def packets():
    return [synth.encode_jpeg(synth.mjpeg_frame(5, i, w, h, sub), q, True, ri)
            for i, (w, h, sub, q, ri) in enumerate([(48, 32, "420", 60, 0), (64, 64, "444", 95, 0), (33, 17, "422", 80, 1),
                                                    (80, 48, "422", 90, 5), (16, 16, "420", 30, 0)])]


# (one engine takes a batch whole: 76 CTAs of slices are the most for one thread in four,
# 152 for one in two)
@pytest.mark.parametrize("n", [1, 5, 76, 77, 152, 153, 305])
def test_every_spread_equals_the_oracle(packets, n):
    refs = [oracle.jpeg_decode(p) for p in packets]
    with m.Context(engines=1) as ctx:
        for i, (r, payload) in enumerate(ctx.decode_batch([packets[k % 5] for k in range(n)], m.CODEC_MJPEG)):
            assert r.status == refs[i % 5].status == 0, r.message
            assert_same_decode(0, "", frame_planes_gpu(m.frame_from_batch(r, payload)), refs[i % 5], f"{n}: {i}")
