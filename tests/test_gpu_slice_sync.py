"""Slice synchronisation over several CTAs of slices: valid scans built so that a CTA's last
slice still has no start when the last pass begins, and then takes the exit that most of its
guesses had, which is not the stored one that the next CTA has read.

The scan (auto slices of 256 bits, six guesses each, 128 slices to a CTA) is flat, two zero
bits a block, so guesses meet only each other: all of them, and the chain of wrong exits
that the second CTA starts with, are a bit off. The last block of slice 254 ends them: its
first amplitude bits are no code to a decode that is a bit off, at the slice's very end, so
no guess of that slice has an exit. Slice 255, the CTA's last, therefore stays without a
start; in it blocks whose codes differ between luma and chroma bring most guesses, but not
the first, to the true state. Every sample equals the oracle decoder's."""
import random

import pytest

import mmrecode_gb300 as m
import oracle
from helpers import assert_same_decode, frame_planes_gpu, jpeg, stuff

pytestmark = pytest.mark.gpu

SLICE, MCUS_X, MCUS_Y = 256, 64, 90
DC = ([1, 1] + [0] * 14, [0, 1])
# (EOB; a level of 8 bits; one of 1 bit in luma, no symbol in chroma; the other way round)
AC_LUMA = ([1, 0, 3] + [0] * 13, [0x00, 0x08, 0x01, 0x10])
AC_CHROMA = ([1, 0, 3] + [0] * 13, [0x00, 0x08, 0x10, 0x01])


def packet(seed):
    rnd = random.Random(seed)
    last = (255 * SLICE - 4) // 2  # this block begins four bits before the end of slice 254
    special = {last: "100" + "111" + format(rnd.randrange(32), "05b")}
    for _ in range(rnd.randrange(1, 8)):
        special[last + 1 + rnd.randrange(90)] = None
    for _ in range(200):
        special.setdefault(last + 400 + rnd.randrange(1200), None)
    bits = []
    for i in range(6 * MCUS_X * MCUS_Y):
        own = "110" if i % 6 >= 4 else "101"
        bits.append("00" if i not in special else "0" + (special[i] or own + rnd.choice("01")) + "0")
    s = "".join(bits)
    s += "1" * (-len(s) % 8)
    return jpeg(16 * MCUS_X, 16 * MCUS_Y, [(1, 2, 2, 0), (2, 1, 1, 1), (3, 1, 1, 1)],
                scan=[(1, 0, 0), (2, 0, 1), (3, 0, 1)], quant={0: [9] * 64, 1: [7] * 64},
                dht=[(0, 0, *DC), (1, 0, *AC_LUMA), (1, 1, *AC_CHROMA)],
                entropy=stuff(int(s, 2).to_bytes(len(s) // 8, "big")))


@pytest.mark.parametrize("seed", range(12))
def test_a_ctas_last_slice_without_a_start_before_the_last_pass(seed):
    p = packet(seed)
    ref = oracle.jpeg_decode(p)
    assert ref.status == 0, ref.message
    with m.Context(engines=1) as ctx:
        (r, payload), = ctx.decode_batch([p], m.CODEC_MJPEG)
    assert r.status == 0, r.message
    assert_same_decode(0, "", frame_planes_gpu(m.frame_from_batch(r, payload)), ref, str(seed))
