"""Marker scan and byte-unstuffing: packets at every address modulo 16 on the device and
with entropy data starting at every offset, runs of 0xFF of every length before stuffed
zeros and restart markers (within a 16-byte group, a 512-byte row, a tile, and across
them), packets cut inside a run, more tiles than one group of sums. Every status, message
and sample equals the oracle decoder's."""
import ctypes
import random

import numpy as np
import pytest

import mmrecode_gb300 as m
import oracle
from helpers import prefixed
from mmrecode_gb300 import _lib

pytestmark = pytest.mark.gpu


def noise_jpeg(seed, w, h, quality, ri):
    px = np.random.default_rng(seed).integers(0, 256, (3, h, w), dtype=np.uint8)
    return m.encode_jpeg(m.VideoFrame(m.YUV444P8, w, h, [m.Plane(p.tobytes(), w, w, h) for p in px]), quality, True, ri)


def altered(jpg, rnd, comment, runs, rate):
    """A comment segment of the given length, and fill bytes before some 0xFF of the scan."""
    sos = jpg.index(b"\xff\xda")
    ds = sos + 2 + (jpg[sos + 2] << 8 | jpg[sos + 3])
    body = bytearray()
    for b in jpg[ds:]:
        if b == 0xFF and rnd.random() < rate:
            body += b"\xff" * rnd.choice(runs)
        body.append(b)
    com = b"\xff\xfe" + (comment + 2).to_bytes(2, "big") + bytes(comment)
    return jpg[:2] + com + jpg[2:ds] + bytes(body)


def packets(kind):
    rnd = random.Random(kind)
    if kind == "groups":  # more than 64 and more than 128 tiles
        return [altered(noise_jpeg(i, 512, 256, 100, ri), rnd, i, [1], 0.01) for i, ri in enumerate((0, 16, 1))]
    out = []
    for i in range(32):
        w, h = rnd.choice([(8, 8), (48, 24), (96, 64), (160, 96)])
        runs = {"plain": [1], "short": [1, 2, 13, 14, 15, 16, 17], "long": [31, 500, 511, 512, 513, 4095, 4096, 9000]}[kind]
        p = altered(noise_jpeg(i, w, h, rnd.choice([50, 95, 100]), rnd.choice([0, 1, 2, 7])), rnd, i % 16, runs,
                    {"plain": 0, "short": 0.3, "long": 0.02}[kind])
        if i % 8 == 7:
            p = p[:-2] + b"\xff" * rnd.choice([1, 2, 20])  # ends inside a marker
        elif i % 8 == 6:
            p = p[:-2 - rnd.randrange(1, 40)] + b"\xff\xfe\x00\x02"
        out.append(p)
    return out


@pytest.mark.parametrize("kind", ["plain", "short", "long", "groups"])
def test_scan_equals_oracle_at_every_alignment(kind):
    torch = pytest.importorskip("torch")
    pk = packets(kind)
    refs = [oracle.jpeg_decode(p) for p in pk]
    assert any(r.status == 0 for r in refs)
    with m.Context() as ctx:
        for shift in (0, 1, 8, 13):
            offs, at = [], 0
            for i, p in enumerate(pk):
                offs.append((at + 15) // 16 * 16 + (i + shift) % 16)
                at = offs[-1] + len(p)
            host = torch.full((at,), 0xFF, dtype=torch.uint8)  # (0xFF between the packets)
            for p, o in zip(pk, offs):
                host.numpy()[o:o + len(p)] = memoryview(p)
            dev = host.cuda()
            cap = [m.probe(m.CODEC_MJPEG, p).planar_bytes for p in pk]
            outs = [torch.zeros(max(c, 1), dtype=torch.uint8, device="cuda") for c in cap]
            torch.cuda.synchronize()
            arr = (_lib.GpuItem * len(pk))()
            for i, p in enumerate(pk):
                it = arr[i]
                it.struct_size = ctypes.sizeof(_lib.GpuItem)
                it.data, it.device_data, it.len = host.data_ptr() + offs[i], dev.data_ptr() + offs[i], len(p)
                it.codec, it.output, it.flags = m.CODEC_MJPEG, m.OUTPUT_PLANAR, m.ITEM_OUT_DEVICE
                it.out, it.out_capacity = outs[i].data_ptr(), cap[i]
            try:
                ctx.decode_raw(arr)
            except m.MmrError:
                assert any(r.status for r in refs)
            for i, ref in enumerate(refs):
                tag = f"{kind}[{i}] at {offs[i]}"
                assert arr[i].status == ref.status, (tag, arr[i].message, ref.message)
                if ref.status:
                    assert arr[i].message.decode() == prefixed(ref.status, ref.message), tag
                else:
                    assert outs[i][:arr[i].out_bytes].cpu().numpy().tobytes() == b"".join(d for _, _, d in ref.frame.planes), tag
