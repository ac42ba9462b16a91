"""Damaged packets between good ones in a batch: what a damaged scan decodes to stays in
its own frame. Layouts whose last component has a block among the first of an MCU (a scan
that lists the components in another order than the frame, several blocks of every
component per MCU): slices past an error start in states that do not fit the block counts
before them. Every status, message and sample equals the oracle decoder's."""
import random

import numpy as np
import pytest

import mmrecode_gb300 as m
import oracle
from helpers import assert_same_decode, encode_blocks, frame_planes_gpu, jpeg, prefixed, stuff

pytestmark = pytest.mark.gpu


def packet(seed, comps, scan, width=320, height=240):
    """Random sparse blocks, whose DC differences pull towards the middle, in scan order."""
    rng = np.random.default_rng(seed)
    factors = {c[0]: c[1] * c[2] for c in comps}
    hmax, vmax = max(c[1] for c in comps), max(c[2] for c in comps)
    mcus = -(-width // (8 * hmax)) * -(-height // (8 * vmax))
    level, blocks = {c[0]: 0 for c in comps}, []
    for _ in range(mcus):
        for sel, _, _ in scan:
            for _ in range(factors[sel]):
                diff = int(rng.integers(-60, 61)) - level[sel] // 4
                level[sel] += diff
                acs, k = [], 1
                while k < 60 and rng.random() < 0.8:
                    run = int(rng.integers(0, 4))
                    acs.append((run, int(rng.choice([-9, -3, -2, -1, 1, 2, 3, 9]))))
                    k += run + 1
                blocks.append((diff, acs, True))
    return jpeg(width, height, comps, scan=scan, entropy=stuff(encode_blocks(blocks).raw_bytes()))


def damaged(data, rnd):
    sos = data.index(b"\xff\xda")
    first = sos + 2 + (data[sos + 2] << 8 | data[sos + 3])
    d = bytearray(data)
    at = rnd.randrange(first, len(d) - 20)
    if rnd.random() < 0.5:
        d[at] ^= 1 << rnd.randrange(8)
    else:
        del d[at:at + rnd.randint(1, 9)]
    return bytes(d)


@pytest.mark.parametrize("comps,order", [
    ([(1, 2, 2, 0), (2, 1, 1, 1), (3, 1, 1, 1)], (3, 1, 2)),
    ([(1, 2, 2, 0), (2, 1, 1, 1), (3, 1, 1, 1)], (2, 3, 1)),
    ([(1, 1, 1, 0), (2, 1, 1, 1), (3, 1, 1, 1)], (3, 2, 1)),
    ([(1, 2, 2, 0), (2, 2, 2, 1), (3, 2, 2, 1)], (1, 2, 3)),
    ([(1, 2, 2, 0), (2, 1, 2, 1), (3, 1, 2, 1)], (1, 2, 3)),
])
@pytest.mark.parametrize("rgb", [False, True])
def test_good_frames_beside_damaged_ones(comps, order, rgb):
    rnd = random.Random(sum(order[0] * c[1] for c in comps))
    good = [packet(s, comps, [(i, 0, 0) for i in order]) for s in range(3)]
    packets = []
    for k in range(30):
        packets += [damaged(good[k % 3], rnd), good[(k + 1) % 3]]
    refs = {p: oracle.jpeg_decode(p) for p in packets}
    assert all(refs[p].status == 0 for p in good) and sum(refs[p].status != 0 for p in packets) > 10
    with m.Context(engines=1) as ctx:
        out = m.OUTPUT_RGB24 if rgb else m.OUTPUT_PLANAR
        for i, ((r, payload), p) in enumerate(zip(ctx.decode_batch(packets, m.CODEC_MJPEG, out), packets)):
            ref = refs[p]
            assert r.status == ref.status, f"{i}: {r.message} vs {ref.message}"
            if ref.status:
                assert r.message == prefixed(ref.status, ref.message), i
            elif rgb:
                assert payload == oracle.rgb24(ref.frame), i
            else:
                assert_same_decode(0, "", frame_planes_gpu(m.frame_from_batch(r, payload)), ref, str(i))
