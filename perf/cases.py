"""Performance cases: what programs built on this library have it do, call by call.

Every case goes through the public Python entry points (``decode_jpeg``, ``decode_dv``,
``Context.decode_raw``, ``Context.encode_raw``, ``Context.open_stream``), with packets and
frames where such a program has them (device memory, pinned host memory, plain bytes).
Pictures are synthetic in the manner of ``mmrecode_gb300.synth``: a gradient, uniform
rectangles and Gaussian noise per plane, made on the GPU from the seed.

All outputs are bytes (samples, streams) and statuses: they are whole numbers, so there is
no ``exact``.
"""

import concurrent.futures
import ctypes
import os

import numpy as np
import torch

import mmrecode_gb300 as m
from mmrecode_gb300 import _lib

DEVICE = "cuda"
SUBSAMPLING = {"gray": (m.GRAY8, 0, 0), "420": (m.YUV420P8, 2, 2), "422": (m.YUV422P8, 2, 1), "444": (m.YUV444P8, 1, 1)}
DV_PICTURES = 64  # distinct DV pictures per batch: the DV encoder runs on the CPU

_context = None


def context():
    """The one context a program keeps for its lifetime."""
    global _context
    if _context is None:
        _context = m.Context()
    return _context


# ---------------------------------------------------------------- cases ---


def listed():
    return [
        # A thumbnail or preview: one small packet, decoded by itself. The smallest call.
        {"name": "jpeg 320x240 alone", "kind": "one_jpeg", "width": 320, "height": 240, "sub": "420", "quality": 75,
         "ri": "none", "noise": 6.0},
        # Scrubbing a DV tape capture: one NTSC frame per call.
        {"name": "dv ntsc alone", "kind": "one_dv", "pal": False},
        # A player's frame: one 1080p packet in host memory to RGB in host memory.
        {"name": "1080p 422 rgb alone", "kind": "decode", "frames": 1, "width": 1920, "height": 1080, "sub": "422",
         "quality": 90, "ri": "row", "noise": 8.0, "rgb": True, "device": False},
        # A second of VGA webcam video (30 frames, no restart markers) to planes on the device.
        {"name": "vga 420 x30", "kind": "decode", "frames": 30, "width": 640, "height": 480, "sub": "420", "quality": 75,
         "ri": "none", "noise": 8.0, "rgb": False, "device": True},
        # Bulk transcoding or training input: 300 frames of 1080p to RGB on the device. The largest.
        {"name": "1080p 422 rgb x300", "kind": "decode", "frames": 300, "width": 1920, "height": 1080, "sub": "422",
         "quality": 90, "ri": "row", "noise": 8.0, "rgb": True, "device": True},
        # The same from and to pinned host memory.
        {"name": "1080p 422 rgb host x64", "kind": "decode", "frames": 64, "width": 1920, "height": 1080, "sub": "422",
         "quality": 90, "ri": "row", "noise": 8.0, "rgb": True, "device": False},
        # A batch of pictures of every size, layout, quality and restart interval.
        {"name": "mixed rgb x64", "kind": "mixed", "frames": 64, "layout": 1, "noise": 8.0, "rgb": True},
        # A DV tape archive: 1000 NTSC frames to planes on the device.
        {"name": "dv ntsc x1000", "kind": "dv", "frames": 1000, "pal": False, "rgb": False, "damaged": False},
        # A damaged PAL tape, concealed, to RGB.
        {"name": "dv pal conceal rgb x50", "kind": "dv", "frames": 50, "pal": True, "rgb": True, "damaged": True},
        # Encoding a device-resident clip to Motion JPEG with restart markers.
        {"name": "encode 1080p 422 x60", "kind": "encode", "frames": 60, "width": 1920, "height": 1080, "sub": "422",
         "quality": 90, "ri": "row", "noise": 8.0, "annex_k": True, "device": True},
        # Encoding a short clip of an odd size from and to host memory, with the reference's settings.
        {"name": "encode 719x405 420 host x12", "kind": "encode", "frames": 12, "width": 719, "height": 405, "sub": "420",
         "quality": 75, "ri": "none", "noise": 6.0, "annex_k": False, "device": False},
        # A whole 720p Motion JPEG file to Y4M.
        {"name": "stream 720p 422 x60", "kind": "stream", "frames": 60, "width": 1280, "height": 720, "sub": "422",
         "quality": 85, "ri": "row", "noise": 8.0},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    """One case of the ranges above. Sizes are any whole number of samples (odd ones too),
    64x48 to 3840x2160, batches 1 to 300 frames of MJPEG and 1 to 1000 of DV, bounded so
    that a case stays below the largest listed one."""
    kind = rng.choice(["one_jpeg", "one_dv", "decode", "decode", "decode", "mixed", "dv", "dv", "encode", "encode", "stream"])
    noise = round(rng.uniform(1.0, 10.0), 2)
    if kind == "one_dv":
        return {"kind": kind, "pal": rng.random() < 0.5, "variant": rng.randrange(1 << 16)}
    if kind == "dv":
        return {"kind": kind, "frames": _log_int(rng, 1, 1000), "pal": rng.random() < 0.5, "rgb": rng.random() < 0.5,
                "damaged": rng.random() < 0.3}
    if kind == "mixed":
        return {"kind": kind, "frames": _log_int(rng, 2, 64), "layout": rng.randrange(1 << 16), "noise": noise, "rgb": rng.random() < 0.7}
    w = _log_int(rng, 64, 3840)
    h = max(48, min(2160, int(w * rng.uniform(0.45, 0.9))))
    c = {"kind": kind, "width": w, "height": h, "sub": rng.choice(["420", "420", "422", "422", "444", "gray"]),
         "quality": rng.randint(50, 95), "ri": rng.choice(["none", "row", 4]), "noise": noise}
    most = max(1, min(300, int(200e6 / (2 * w * h))))
    if kind == "decode":
        c |= {"frames": _log_int(rng, 1, most), "rgb": rng.random() < 0.5, "device": rng.random() < 0.6}
    elif kind == "encode":
        c |= {"frames": _log_int(rng, 1, min(most, 60)), "annex_k": rng.random() < 0.5, "device": rng.random() < 0.6}
    elif kind == "stream":
        c |= {"frames": _log_int(rng, 1, min(most, 120))}
    return c


# --------------------------------------------------------------- pictures ---


def _plane_sizes(w, h, sub):
    _, sx, sy = SUBSAMPLING[sub]
    if sub == "gray":
        return [(w, h)]
    cw, ch = (w + sx - 1) // sx, (h + sy - 1) // sy
    return [(w, h), (cw, ch), (cw, ch)]


def _picture(gen, rng, sizes, noise, n_rect):
    """One picture's planes, packed one after another (uint8, device)."""
    colours = rng.uniform(16, 240, (n_rect, 3))
    rects = np.concatenate([rng.uniform(0, 0.9, (n_rect, 2)), rng.uniform(0.05, 0.4, (n_rect, 2))], axis=1)
    out = []
    for p, (pw, ph) in enumerate(sizes):
        a, b = rng.uniform(0.2, 1.0, 2)
        phase = rng.uniform(0, 255)
        x = torch.arange(pw, device=DEVICE, dtype=torch.float32) * (a / pw * 200.0 / (a + b))
        y = torch.arange(ph, device=DEVICE, dtype=torch.float32) * (b / ph * 200.0 / (a + b))
        f = y[:, None] + x[None, :] + phase * 0.2
        if p:
            f = 128.0 + (f - 100.0) * 0.5
        for k in range(n_rect):
            x0, y0, rw, rh = rects[k]
            f[int(y0 * ph):int(min(1.0, y0 + rh) * ph), int(x0 * pw):int(min(1.0, x0 + rw) * pw)] = float(colours[k, p])
        f = f + torch.randn((ph, pw), device=DEVICE, generator=gen) * noise
        out.append(f.round_().clamp_(0, 255).to(torch.uint8).reshape(-1))
    return torch.cat(out)


def _generators(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed), np.random.Generator(np.random.PCG64(seed))


def _interval(ri, w, sub):
    if ri == "row":
        return (w + 8 * max(1, SUBSAMPLING[sub][1]) - 1) // (8 * max(1, SUBSAMPLING[sub][1]))
    return 0 if ri == "none" else int(ri)


def _encode_items(frames, w, h, sub, base_in, pitch, base_out, cap, flags):
    """An EncodeItem array over packed frames `pitch` bytes apart, outputs `cap` apart."""
    fmt = SUBSAMPLING[sub][0]
    sizes = _plane_sizes(w, h, sub)
    items = (_lib.EncodeItem * frames)()
    for i in range(frames):
        it = items[i]
        it.struct_size = ctypes.sizeof(_lib.EncodeItem)
        v = it.frame
        v.struct_size = ctypes.sizeof(_lib.VideoFrameView)
        v.format, v.range, v.width, v.height, v.plane_count = fmt, m.RANGE_FULL, w, h, len(sizes)
        at = base_in + i * pitch
        for c, (pw, ph) in enumerate(sizes):
            v.planes[c].data = ctypes.cast(at, _lib.u8p)
            v.planes[c].data_len, v.planes[c].stride, v.planes[c].width, v.planes[c].height = pw * ph, pw, pw, ph
            at += pw * ph
        it.flags = flags
        it.out = base_out + i * cap
        it.out_capacity = cap
    return items


def _encode_capacity(w, h, sub, ri):
    """A JPEG buffer's size: two bytes a sample hold any picture here, and never over the library's bound."""
    bound = _lib.load().mmr_gpu_jpeg_encode_bound(SUBSAMPLING[sub][0], w, h, ri)
    return (min(bound, 2 * _planar_bytes(w, h, sub) + 8192) + 255) // 256 * 256


def _jpeg_packets(gen, rng, frames, w, h, sub, quality, ri, noise):
    """Encoded pictures as numpy byte arrays (encoded by the library's own GPU encoder)."""
    sizes = _plane_sizes(w, h, sub)
    pitch = sum(a * b for a, b in sizes)
    ri = _interval(ri, w, sub)
    cap = _encode_capacity(w, h, sub, ri)
    packets = []
    step = max(1, min(frames, int(64e6 / pitch)))
    for at in range(0, frames, step):
        n = min(step, frames - at)
        raw = torch.cat([_picture(gen, rng, sizes, noise, 20) for _ in range(n)])
        out = torch.empty(n * cap, dtype=torch.uint8, device=DEVICE)
        torch.cuda.synchronize()
        items = _encode_items(n, w, h, sub, raw.data_ptr(), pitch, out.data_ptr(), cap, m.ITEM_IN_DEVICE | m.ITEM_OUT_DEVICE)
        context().encode_raw(items, quality, True, ri)
        for i in range(n):
            assert items[i].status == 0, items[i].message
            packets.append(out[i * cap:i * cap + items[i].out_len].cpu().numpy())
    return packets


def _dv_packets(gen, rng, frames, pal, damaged):
    sizes = [(720, 576), (360, 288), (360, 288)] if pal else [(720, 480), (180, 480), (180, 480)]
    n = min(frames, DV_PICTURES)
    pictures = [_picture(gen, rng, sizes, 6.0, 1).cpu().numpy() for _ in range(n)]

    def one(px):
        planes, at = [], 0
        for w, h in sizes:
            planes.append(m.Plane(px[at:at + w * h].tobytes(), w, w, h))
            at += w * h
        f = m.VideoFrame(m.YUV420P8 if pal else m.YUV411P8, 720, sizes[0][1], planes, m.RANGE_LIMITED)
        return np.frombuffer(m.encode_dv(f, m.DV_MODE_ACTIVITY), np.uint8)

    with concurrent.futures.ThreadPoolExecutor(max_workers=min(16, os.cpu_count() or 4)) as ex:
        encoded = list(ex.map(one, pictures))
    packets = [encoded[i % n] for i in range(frames)]
    if damaged:  # a tape drop-out: a few video DIF blocks with a damaged identifier in every third frame
        sequences = 12 if pal else 10
        for i in range(0, frames, 3):
            packets[i] = packets[i].copy()
            for _ in range(int(rng.integers(1, 6))):
                dif = int(rng.integers(0, sequences)) * 150 + 7 + int(rng.integers(0, 9)) * 16 + int(rng.integers(0, 15))
                packets[i][dif * 80 + 2] ^= 0xff
    return packets


def _mixed_parameters(layout, frames):
    """The batch's pictures: sizes in steps of 16 over 320x240..3840x2160 (every fourth picture any size, odd ones
    too), every layout, quality 50..95, restart interval none, one MCU row or 4 MCUs."""
    rng = np.random.Generator(np.random.PCG64(layout))
    out = []
    for i in range(frames):
        w, h = int(rng.integers(20, 241)) * 16, int(rng.integers(15, 136)) * 16
        if i % 4 == 3:
            w, h = w - int(rng.integers(0, 16)), h - int(rng.integers(0, 16))
        out.append((w, h, ["420", "422", "444"][int(rng.integers(0, 3))], int(rng.integers(50, 96)),
                    ["none", "row", 4][int(rng.integers(0, 3))]))
    return out


# ----------------------------------------------------------------- states ---


def _decode_state(packets, codec, needs, rgb, device, flags):
    """An item array over one slab of packets and one slab of outputs (256-byte aligned)."""
    n = len(packets)
    ends = np.cumsum([0] + [(len(p) + 255) // 256 * 256 for p in packets])
    outs = np.cumsum([0] + [(k + 255) // 256 * 256 for k in needs])
    host = torch.empty(int(ends[-1]) + 256, dtype=torch.uint8, pin_memory=True)
    hv = host.numpy()
    for i, p in enumerate(packets):
        hv[ends[i]:ends[i] + len(p)] = p
    dev = host.to(DEVICE) if device else None
    out = torch.zeros(int(outs[-1]), dtype=torch.uint8, device=DEVICE) if device else \
        torch.zeros(int(outs[-1]), dtype=torch.uint8, pin_memory=True)
    items = (_lib.GpuItem * n)()
    for i, p in enumerate(packets):
        it = items[i]
        it.struct_size = ctypes.sizeof(_lib.GpuItem)
        it.data = host.data_ptr() + int(ends[i])
        it.len = len(p)
        if device:
            it.device_data = dev.data_ptr() + int(ends[i])
        it.codec = codec
        it.output = m.OUTPUT_RGB24 if rgb else m.OUTPUT_PLANAR
        it.flags = flags | ((m.ITEM_IN_DEVICE | m.ITEM_OUT_DEVICE) if device else 0)
        it.out = out.data_ptr() + int(outs[i])
        it.out_capacity = int(needs[i])
    records = np.frombuffer(items, np.uint8).reshape(n, ctypes.sizeof(_lib.GpuItem))
    at, seg = _lib.GpuItem.status.offset, _lib.GpuItem.concealed_segments.offset
    return {"kind": "decode", "items": items, "out": out, "status": records[:, at:at + 4], "concealed": records[:, seg:seg + 4],
            "keep": (host, dev)}


def _planar_bytes(w, h, sub):
    return sum(a * b for a, b in _plane_sizes(w, h, sub))


def prepare(case, seed):
    kind = case["kind"]
    gen, rng = _generators(seed)
    if kind in ("one_jpeg", "decode", "stream"):
        w, h, sub = case["width"], case["height"], case["sub"]
        packets = _jpeg_packets(gen, rng, case.get("frames", 1), w, h, sub, case["quality"], case["ri"], case["noise"])
        if kind == "one_jpeg":
            return {"kind": kind, "data": packets[0].tobytes()}
        if kind == "stream":
            data = torch.from_numpy(np.concatenate(packets)).pin_memory()
            out = torch.zeros(256 + len(packets) * (_planar_bytes(w, h, sub) + 6), dtype=torch.uint8, pin_memory=True)
            return {"kind": kind, "data": data, "out": out}
        need = 3 * w * h if case["rgb"] else _planar_bytes(w, h, sub)
        return _decode_state(packets, m.CODEC_MJPEG, [need] * len(packets), case["rgb"], case["device"], 0)
    if kind == "mixed":
        packets, needs = [], []
        for w, h, sub, quality, ri in _mixed_parameters(case["layout"], case["frames"]):
            packets += _jpeg_packets(gen, rng, 1, w, h, sub, quality, ri, case["noise"])
            needs.append(3 * w * h if case["rgb"] else _planar_bytes(w, h, sub))
        return _decode_state(packets, m.CODEC_MJPEG, needs, case["rgb"], True, 0)
    if kind == "one_dv":
        return {"kind": kind, "data": _dv_packets(gen, rng, 1, case["pal"], False)[0].tobytes()}
    if kind == "dv":
        packets = _dv_packets(gen, rng, case["frames"], case["pal"], case["damaged"])
        rows = 576 if case["pal"] else 480
        need = 720 * rows * 3 if case["rgb"] else 720 * rows * 3 // 2
        return _decode_state(packets, m.CODEC_DV, [need] * len(packets), case["rgb"], True,
                             m.ITEM_CONCEAL if case["damaged"] else 0)
    if kind == "encode":
        n, w, h, sub, device = case["frames"], case["width"], case["height"], case["sub"], case["device"]
        sizes = _plane_sizes(w, h, sub)
        raw = torch.cat([_picture(gen, rng, sizes, case["noise"], 20) for _ in range(n)])
        ri = _interval(case["ri"], w, sub)
        cap = _encode_capacity(w, h, sub, ri)
        if not device:
            raw = raw.cpu().pin_memory()
        out = torch.zeros(n * cap, dtype=torch.uint8, device=DEVICE) if device else \
            torch.zeros(n * cap, dtype=torch.uint8, pin_memory=True)
        torch.cuda.synchronize()
        items = _encode_items(n, w, h, sub, raw.data_ptr(), _planar_bytes(w, h, sub), out.data_ptr(), cap,
                              (m.ITEM_IN_DEVICE | m.ITEM_OUT_DEVICE) if device else 0)
        records = np.frombuffer(items, np.uint8).reshape(n, ctypes.sizeof(_lib.EncodeItem))
        at, size = _lib.EncodeItem.status.offset, _lib.EncodeItem.out_len.offset
        return {"kind": kind, "items": items, "raw": raw, "out": out, "status": records[:, at:at + 4],
                "lengths": records[:, size:size + 8], "options": (case["quality"], case["annex_k"], ri)}
    raise ValueError(kind)


def run(state):
    kind = state["kind"]
    if kind == "decode":
        context().decode_raw(state["items"])
        return [state["out"], state["status"], state["concealed"]]
    if kind == "one_jpeg":
        return [np.frombuffer(p.data, np.uint8) for p in m.decode_jpeg(state["data"]).planes]
    if kind == "one_dv":
        return [np.frombuffer(p.data, np.uint8) for p in m.decode_dv(state["data"]).planes]
    if kind == "encode":
        context().encode_raw(state["items"], *state["options"])
        return [state["out"], state["status"], state["lengths"]]
    with context().open_stream((state["data"].data_ptr(), state["data"].numel())) as stream:
        outcome = stream.decode_into(state["out"].data_ptr(), state["out"].numel())
    return [state["out"][:outcome.bytes_written], outcome.status, outcome.frames_written]


# ------------------------------------------------------------------- work ---

_densities = {}


def _bytes_per_sample(sub, quality, noise):
    """Compressed bytes per sample of such a picture, from a 256x256 one (CPU encoder)."""
    key = (sub, quality, noise)
    if key not in _densities:
        rng = np.random.Generator(np.random.PCG64(1))
        planes = [m.Plane(np.clip(np.rint(128 + np.add.outer(np.arange(h), np.arange(w)) * 0.05 + rng.normal(0, noise, (h, w))),
                                  0, 255).astype(np.uint8).tobytes(), w, w, h) for w, h in _plane_sizes(256, 256, sub)]
        fmt = SUBSAMPLING[sub][0]
        data = m.encode_jpeg(m.VideoFrame(fmt, 256, 256, planes, m.RANGE_FULL), quality, True, 0)
        _densities[key] = (len(data) - 600) / _planar_bytes(256, 256, sub)
    return _densities[key]


def work(case):
    """Compressed bytes once, samples (or pixels) once. Operations: a fast 8x8 transform
    (about 10 a sample) and the colour conversion (about 9 a pixel)."""
    kind = case["kind"]
    if kind in ("one_dv", "dv"):
        n, rows = case.get("frames", 1), 576 if case["pal"] else 480
        rgb = case.get("rgb", False)
        return {"bytes": n * ((144000 if case["pal"] else 120000) + 720 * rows * (3 if rgb else 1.5)),
                "flops": n * 720 * rows * (15 + (9 if rgb else 0))}
    if kind == "mixed":
        total = {"bytes": 0.0, "flops": 0.0}
        for w, h, sub, quality, _ in _mixed_parameters(case["layout"], case["frames"]):
            samples = _planar_bytes(w, h, sub)
            total["bytes"] += samples * _bytes_per_sample(sub, quality, case["noise"]) + (3 * w * h if case["rgb"] else samples)
            total["flops"] += 10 * samples + (9 * w * h if case["rgb"] else 0)
        return total
    w, h, sub, n = case["width"], case["height"], case["sub"], case.get("frames", 1)
    samples = _planar_bytes(w, h, sub)
    packed = samples * _bytes_per_sample(sub, case["quality"], case["noise"])
    rgb = case.get("rgb", False)
    return {"bytes": n * (packed + (3 * w * h if rgb else samples)), "flops": n * (10 * samples + (9 * w * h if rgb else 0))}
