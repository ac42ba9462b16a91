"""Frames in host buffers that touch but were pinned separately, or not at all, in one
encode batch: every stream equals the CPU encoder's."""
import ctypes
import mmap

import numpy as np
import pytest

import mmrecode_gb300 as m
from mmrecode_gb300 import _lib

pytestmark = pytest.mark.gpu

W = H = 64  # a gray frame is one 4 KiB page on most systems


@pytest.mark.parametrize("pinned", [[], [(0, 6)], [(0, 3), (3, 6)], [(i, i + 1) for i in range(6)], [(0, 3)], [(2, 6)]])
def test_neighbouring_buffers(pinned):
    import torch

    cudart = torch.cuda.cudart()
    torch.zeros(1, device="cuda")
    rows = max(H, mmap.PAGESIZE // W)  # whole pages per frame
    size, n = rows * W, 6
    area = mmap.mmap(-1, n * size)
    samples = np.frombuffer(area, np.uint8).reshape(n, rows, W)
    samples[:] = np.random.default_rng(9).integers(90, 160, samples.shape)
    base = samples.ctypes.data
    done = []
    try:
        for a, b in pinned:
            assert int(cudart.cudaHostRegister(base + a * size, (b - a) * size, 0)) == 0
            done.append(base + a * size)
        items, outs = (_lib.EncodeItem * n)(), []
        keep = []
        for i in range(n):
            frame = m.VideoFrame(m.GRAY8, W, rows, [m.Plane(samples[i].tobytes(), W, W, rows)], m.RANGE_FULL)
            items[i].struct_size = ctypes.sizeof(_lib.EncodeItem)
            items[i].frame = m._view(frame, keep)
            items[i].frame.planes[0].data = ctypes.cast(base + i * size, type(items[i].frame.planes[0].data))
            outs.append((ctypes.c_uint8 * (size * 8 + 4096))())
            items[i].out = ctypes.addressof(outs[i])
            items[i].out_capacity = len(outs[i])
        with m.Context() as ctx:
            ctx.encode_raw(items, 85, True, 0)
        for i in range(n):
            frame = m.VideoFrame(m.GRAY8, W, rows, [m.Plane(samples[i].tobytes(), W, W, rows)], m.RANGE_FULL)
            assert items[i].status == 0
            assert bytes(outs[i][:items[i].out_len]) == m.encode_jpeg(frame, 85, True, 0)
    finally:
        for p in done:
            cudart.cudaHostUnregister(p)
