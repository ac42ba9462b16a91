"""Forward DCT of integer content: quotients exactly half-way between two integers are
listed per CTA and recomputed packed in binary64 (fdct_kernel). Every byte equals the CPU
encoder's, at block counts around one CTA step (32 blocks), with every block a tie (a
CTA's list fills within one step) and with more steps than CTAs."""
import numpy as np
import pytest

import mmrecode_gb300 as m

pytestmark = pytest.mark.gpu


def _frame(w, h, kind, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    if kind == "ties":  # per block a sum of 8 * 12 (mod 8 * 24): S / 8 / 3 is half-way at q90's DC quantiser 3
        y = np.full((h, w), 128, np.int64)
        for by in range(0, h, 8):
            for bx in range(0, w, 8):
                if (bx // 8 + by // 8) % 2:
                    y[by, bx] += 12
                else:
                    y[by:by + 8, bx:bx + 8] += rng.integers(-2, 3, y[by:by + 8, bx:bx + 8].shape)
    else:  # small integer noise: every class of tie, now and then
        y = 128 + rng.integers(-6, 7, (h, w))
    y = np.clip(y, 0, 255).astype(np.uint8)
    return m.VideoFrame(m.GRAY8, w, h, [m.Plane(y.tobytes(), w, w, h)], m.RANGE_FULL)


@pytest.mark.parametrize("w,h,kind", [(8, 8, "ties"), (8 * 31, 8, "ties"), (8 * 32, 8, "ties"), (8 * 33, 8, "noise"),
                                      (8 * 40 - 3, 8 * 30 - 5, "ties"), (1600, 1200, "noise"), (1608, 1208, "ties")])
@pytest.mark.parametrize("quality", [90, 100])
def test_ties_equal_the_cpu_encoder(w, h, kind, quality):
    frames = [_frame(w, h, kind, s) for s in range(2)]
    with m.Context() as ctx:
        got = ctx.encode_jpeg_batch(frames, quality, annex_k=True)
        assert ctx.encode_stats()["exact_coefficients"] > 0 or w * h < 512
    for f, (status, message, data) in zip(frames, got):
        assert status == 0, message
        assert data == m.encode_jpeg(f, quality, annex_k=True)


def _random_frame(rng, fmt, w, h, flat):
    """A frame with padded strides; flat ones have few symbols, the others dense blocks."""
    sx, sy = {m.YUV420P8: (2, 2), m.YUV422P8: (2, 1)}.get(fmt, (1, 1))
    planes = []
    for i in range(1 if fmt == m.GRAY8 else 3):
        pw, ph = (w, h) if i == 0 else ((w + sx - 1) // sx, (h + sy - 1) // sy)
        stride = pw + int(rng.integers(0, 3))
        y = np.full((ph, stride), int(rng.integers(0, 256))) if flat else rng.integers(0, 256, (ph, stride))
        planes.append(m.Plane(y.astype(np.uint8).tobytes(), stride, pw, ph))
    return m.VideoFrame(fmt, w, h, planes, m.RANGE_FULL)


@pytest.mark.parametrize("annex_k,ri", [(True, 0), (False, 0), (True, 1), (True, 7), (False, 2)])
def test_batches_of_every_layout_equal_the_cpu_encoder(annex_k, ri):
    """Frames of one to many chunks and segments in one batch (a CTA of chunks within a
    frame, over two, over many), gray frames first (their plan lacks the second tables),
    host frames packed one behind the other or not, device buffers at odd addresses and
    ones that are one byte too small."""
    import ctypes

    import torch

    from mmrecode_gb300 import _lib
    rng = np.random.Generator(np.random.PCG64(5))
    formats = [m.GRAY8, m.YUV420P8, m.YUV422P8, m.YUV444P8]
    frames = [_random_frame(rng, formats[i % 4], int(rng.integers(1, 90)), int(rng.integers(1, 70)), i % 3 == 0)
              for i in range(24)]
    frames += [_random_frame(rng, f, 411, 305, flat) for f in formats for flat in (False, True)]
    want = [m.encode_jpeg(f, 88, annex_k, ri) for f in frames]
    with m.Context() as ctx:
        for (status, message, data), ref in zip(ctx.encode_jpeg_batch(frames, 88, annex_k, ri), want):
            assert status == 0, message
            assert data == ref
        # into device buffers: each frame at an odd address, every fifth one a byte short
        at, spots = 0, []
        for ref in want:
            spots.append(at + 1 + int(rng.integers(0, 16)))
            at = spots[-1] + len(ref) + 16
        out = torch.full((at + 64,), 0xEE, dtype=torch.uint8, device="cuda")
        items, keep = (_lib.EncodeItem * len(frames))(), []
        for i, f in enumerate(frames):
            items[i].struct_size = ctypes.sizeof(_lib.EncodeItem)
            items[i].frame = m._view(f, keep)
            items[i].flags = m.ITEM_OUT_DEVICE
            items[i].out = out.data_ptr() + spots[i]
            items[i].out_capacity = len(want[i]) - (1 if i % 5 == 4 else 0)
        torch.cuda.synchronize()
        ctx.encode_raw(items, 88, annex_k, ri)
        got = out.cpu().numpy()
        expect = np.full_like(got, 0xEE)
        for i, ref in enumerate(want):
            if i % 5 == 4:
                assert items[i].status == m.INVALID_ARGUMENT
            else:
                assert items[i].status == 0 and items[i].out_len == len(ref)
                expect[spots[i]:spots[i] + len(ref)] = np.frombuffer(ref, np.uint8)
        assert (got == expect).all()  # nothing outside the frames' bytes is written
