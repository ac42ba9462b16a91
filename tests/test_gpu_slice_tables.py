"""Chunked entropy decode, the forms its kernels choose between: tables in shared memory
or not (more than two AC or DC tables, codes over many 16-bit patterns, windows clamped
to an incomplete code), one or several speculative decodes per slice, one or many CTAs of
slices per interval, intervals shorter than a slice. Every status, message and sample
equals the oracle decoder's, on valid streams and on copies damaged in the entropy data."""
import random

import numpy as np
import pytest

import mmrecode_gb300 as m
import oracle
from helpers import assert_same_decode, frame_planes_gpu, prefixed
from mmrecode_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with m.Context() as c:
        yield c


def check(ctx, packets, label):
    refs = [oracle.jpeg_decode(p) for p in packets]
    for bits in (0, 128, 1024, 1 << 20):
        ctx.set_slice_bits(bits)
        for batch in ([[p] for p in packets], [packets]) if bits == 0 else ([packets],):
            results = [r for b in batch for r in ctx.decode_batch(b, m.CODEC_MJPEG)]
            for i, ((r, payload), ref) in enumerate(zip(results, refs)):
                tag = f"{label}[{i}] slice_bits={bits} batches={len(batch)}"
                assert r.status == ref.status, f"{tag}: {r.message} vs {ref.message}"
                if ref.status:
                    assert r.message == prefixed(ref.status, ref.message), tag
                else:
                    assert_same_decode(0, "", frame_planes_gpu(m.frame_from_batch(r, payload)), ref, tag)
    ctx.set_slice_bits(0)


def damaged(packet, seed, n):
    rnd = random.Random(seed)
    sos = packet.index(b"\xff\xda")
    ds = sos + 2 + (packet[sos + 2] << 8 | packet[sos + 3])
    out = []
    for k in range(n):
        d = bytearray(packet)
        p = rnd.randrange(ds, len(d) - 2)
        if k % 3 == 0:
            d[p] ^= 1 << rnd.randrange(8)
        elif k % 3 == 1:
            del d[p:p + rnd.randint(1, 9)]
        else:
            d = d[:p] + d[-2:]
        out.append(bytes(d))
    return out


def segment(code, payload):
    return bytes([0xFF, code]) + (len(payload) + 2).to_bytes(2, "big") + payload


def canonical(counts, symbols):
    codes, code, k = {}, 0, 0
    for length in range(1, 17):
        for _ in range(counts.get(length, 0)):
            codes[symbols[k]] = (code, length)
            code, k = code + 1, k + 1
        code <<= 1
    return codes


def gray_jpeg(seed, blocks_x, blocks_y, dc_counts, ac_counts, ac_symbols):
    """A gray baseline JPEG of random levels coded with the given canonical tables."""
    rng = np.random.default_rng(seed)
    dc = canonical(dc_counts, list(range(12)))
    ac = canonical(ac_counts, ac_symbols)
    bits, prev = [], 0

    def put(code, length):
        bits.append(format(code, f"0{length}b") if length else "")

    def amplitude(v):
        size = abs(v).bit_length()
        put(v if v > 0 else v + (1 << size) - 1, size)

    for _ in range(blocks_x * blocks_y):
        level = int(rng.integers(-200, 201))
        put(*dc[abs(level - prev).bit_length()])
        amplitude(level - prev)
        prev, run = level, 0
        density = rng.uniform(0, 0.5)
        for _ in range(63):
            v = int(rng.integers(-7, 8)) if rng.random() < density else 0
            if v == 0 or (min(run, 15) << 4 | abs(v).bit_length()) not in ac:
                run += 1
                continue
            while run >= 16:
                put(*ac[0xF0])
                run -= 16
            put(*ac[run << 4 | abs(v).bit_length()])
            amplitude(v)
            run = 0
        if run:
            put(*ac[0x00])
    s = "".join(bits)
    s += "1" * (-len(s) % 8)
    data = int(s, 2).to_bytes(len(s) // 8, "big").replace(b"\xff", b"\xff\x00")
    table = lambda tc, counts, syms: segment(0xC4, bytes([tc << 4]) + bytes(counts.get(i, 0) for i in range(1, 17)) + bytes(syms))  # noqa: E731
    return (b"\xff\xd8" + segment(0xDB, b"\0" + bytes([4] * 64)) +
            segment(0xC0, b"\x08" + (8 * blocks_y).to_bytes(2, "big") + (8 * blocks_x).to_bytes(2, "big") + b"\x01\x01\x11\x00") +
            table(0, dc_counts, list(range(12))) + table(1, ac_counts, ac_symbols) +
            segment(0xDA, b"\x01\x01\x00\x00\x3f\x00") + data + b"\xff\xd9")


AC = [0x00, 0xF0] + [(r << 4) | s for r in range(16) for s in range(1, 4)]


@pytest.mark.parametrize("dc_counts,ac_counts", [
    ({4: 12}, {6: 50}),                        # no code longer than 11 bits
    ({12: 12}, {12: 50}),                      # only longer ones, many patterns, clamped windows
    ({2: 1, 16: 11}, {1: 1, 16: 49}),          # one short code, few patterns of half the space
    ({3: 6, 16: 6}, {3: 6, 11: 10, 12: 10, 13: 10, 16: 14}),
])
def test_tables_of_every_shape(ctx, dc_counts, ac_counts):
    packets = [gray_jpeg(s, w, h, dc_counts, ac_counts, AC) for s, (w, h) in enumerate([(1, 1), (9, 7), (40, 33)])]
    check(ctx, packets + damaged(packets[2], 5, 9), "shapes")


def more_tables(packet):
    """The packet with the chroma components on tables of their own: Cr on a copy of
    Cb's with one more (rejected) symbol, so that three DC and three AC tables differ."""
    i, tables = 2, {}
    while packet[i + 1] != 0xDA:
        length = packet[i + 2] << 8 | packet[i + 3]
        if packet[i + 1] == 0xC4:
            p, seg = 0, packet[i + 4:i + 2 + length]
            while p < len(seg):
                n = sum(seg[p + 1:p + 17])
                tables[seg[p]] = seg[p + 1:p + 17 + n]
                p += 17 + n
        i += 2 + length
    extra = b""
    for key in (0x01, 0x11):
        t = tables[key]
        extra += segment(0xC4, bytes([key + 1]) + t[:15] + bytes([t[15] + 1]) + t[16:] + b"\x0c")
    d = bytearray(packet[:i] + extra + packet[i:])
    sos = i + len(extra)
    assert d[sos + 4] == 3
    d[sos + 10] = 0x22  # Cr: DC table 2, AC table 2
    return bytes(d)


@pytest.mark.parametrize("sub,ri", [("420", 0), ("422", 30), ("444", 0), ("444", 1)])
def test_three_tables_of_each_class(ctx, sub, ri):
    packets = [more_tables(p) for p in synth.mjpeg_stream(701, 2, 480, 272, sub, 85, ri)]
    check(ctx, packets + damaged(packets[0], 6, 6), f"three {sub}")


@pytest.mark.parametrize("w,h,sub,q,ri", [(2048, 1024, "420", 60, 0),   # thousands of slices in one interval
                                          (1920, 1080, "420", 92, 0), (720, 480, "420", 40, 2), (640, 64, "422", 75, 1)])
def test_intervals_over_many_and_few_slices(ctx, w, h, sub, q, ri):
    packets = synth.mjpeg_stream(702, 1, w, h, sub, q, ri)
    check(ctx, packets + damaged(packets[0], 7, 3), f"{w}x{h}")
