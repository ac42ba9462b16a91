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
