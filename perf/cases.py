"""The work that users of this library have it do, as cases that can be timed.

A case codes video frames through the public entry points (pyrowave_b200.capi,
the binding of include/pyrowave.h and include/pyrowave_cuda.h):

  encode     device planes -> device bitstream
  decode     device bitstream (block table + words) -> device planes
  roundtrip  both, back to back on one stream
  packets    a frame as received, in packets of at most 8 KiB in device memory
             -> device planes
  host       host planes -> packetized bytes on the host -> host planes
  batch      encode and decode of many frames of mixed sizes in one call

Frame sizes, chroma formats and budgets are those of bench.py and the tests, and
of the same ranges. Every output is whole numbers (bitstream words, samples), so
there is no 64-bit value to be near to: exact() has none to give.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from pyrowave_b200 import capi

PACKET_BYTES = 8192
MIXED_SIZES = [(1280, 720), (1366, 768), (1920, 1080), (2560, 1080), (2560, 1440), (3840, 2160)]


def _case(kind, width, height, chroma444, budget, bits=8, precision="default", name=None, frames=1):
    case = {"kind": kind, "width": width, "height": height, "chroma444": chroma444, "budget": budget, "bits": bits,
            "precision": precision, "frames": frames}
    return dict(case, name=name) if name else case


def listed():
    return [
        # A thumbnail or preview stream: nothing but launches and latency.
        _case("roundtrip", 256, 144, False, 16000, name="roundtrip_144p"),
        # The sender of a 720p game stream.
        _case("encode", 1280, 720, False, 150000, name="encode_720p"),
        # Sender and receiver of the ordinary 1080p stream, each on a machine of its own.
        _case("encode", 1920, 1080, False, 400000, name="encode_1080p"),
        _case("decode", 1920, 1080, False, 400000, name="decode_1080p"),
        # The same frame as it comes from a network card into device memory.
        _case("packets", 1920, 1080, False, 400000, name="packets_1080p"),
        # The same frame for programs that keep their planes and packets on the host.
        _case("host", 1920, 1080, False, 400000, name="host_1080p"),
        # The reference's default precision (FP16 staging and storage of levels 0-1).
        _case("roundtrip", 1920, 1080, False, 400000, precision="reference", name="roundtrip_1080p_fp16"),
        # High bit depth, 4:4:4, an odd size that fills no tile: a cropped capture window.
        _case("roundtrip", 1365, 767, True, 600000, bits=16, name="roundtrip_odd_444_16bit"),
        # A 4K stream, both ends on one GPU.
        _case("roundtrip", 3840, 2160, False, 1200000, name="roundtrip_4k"),
        # Sender and receiver of a 4K 4:4:4 desktop.
        _case("encode", 3840, 2160, True, 1200000, name="encode_4k_444"),
        _case("decode", 3840, 2160, True, 1200000, name="decode_4k_444"),
        # A transcoding server: every size and both chroma formats in one call.
        _case("batch", 3840, 2160, True, 416000, name="batch_12_mixed", frames=12),
    ]


def draw(rng):
    kind = rng.choice(["encode", "decode", "roundtrip", "roundtrip", "packets", "host", "batch"])
    if kind == "batch":
        return _case(kind, 3840, 2160, True, rng.randrange(300000, 520000) & ~3, frames=rng.randint(4, 12))
    chroma444 = rng.random() < 0.4
    width = int(round(math.exp(rng.uniform(math.log(160), math.log(3840)))))
    height = max(64, min(2160, int(round(width * rng.choice([9 / 16, 9 / 16, 10 / 16, 3 / 4, 9 / 21, 16 / 9])))))
    if not chroma444:
        width, height = width & ~1, height & ~1
    bits = 16 if kind in ("encode", "decode", "roundtrip", "host") and rng.random() < 0.25 else 8
    precision = "reference" if rng.random() < 0.2 else "default"
    bits_per_pixel = math.exp(rng.uniform(math.log(0.6), math.log(2.4)))
    budget = max(4000, int(width * height * bits_per_pixel / 8) & ~3)
    return _case(kind, width, height, chroma444, budget, bits, precision)


def _frames(case):
    """(width, height, chroma444, budget) of every frame of a case."""
    if case["kind"] != "batch":
        return [(case["width"], case["height"], case["chroma444"], case["budget"])]
    out = []
    for i in range(case["frames"]):
        w, h = MIXED_SIZES[i % len(MIXED_SIZES)]
        # Budgets spread by +-20% around the case's, as 150-250 Mbit/s at 60 fps are.
        out.append((w, h, (i // len(MIXED_SIZES)) % 2 == 1, int(case["budget"] * (0.8 + 0.4 * ((i * 5) % 12) / 11)) & ~3))
    return out


def _plane_sizes(width, height, chroma444):
    chroma = (width, height) if chroma444 else (width // 2, height // 2)
    return [(width, height), chroma, chroma]


def _blur(a):
    a = torch.nn.functional.pad(a[None, None], (1, 1, 1, 1), mode="reflect")[0, 0]
    a = 0.25 * a[:, :-2] + 0.5 * a[:, 1:-1] + 0.25 * a[:, 2:]
    return 0.25 * a[:-2] + 0.5 * a[1:-1] + 0.25 * a[2:]


def _plane(width, height, luma, bits, dense, gen, rng):
    """One plane like those of pyrowave_b200.synth (gradient, band-limited noise,
    flat rectangles, line patterns where dense), made on the GPU."""
    lo, hi = (16.0, 235.0) if luma else (16.0, 240.0)
    angle = rng.uniform(0.0, 2.0 * math.pi)
    x = torch.arange(width, device="cuda", dtype=torch.float32) * (math.cos(angle) / width)
    y = torch.arange(height, device="cuda", dtype=torch.float32) * (math.sin(angle) / height)
    t = x[None, :] + y[:, None]
    img = 48.0 + 140.0 * (0.5 + 0.5 * t) if luma else 128.0 + 60.0 * (rng.random() - 0.5) * 2.0 * t
    noise = torch.randn((height, width), device="cuda", generator=gen)
    noise = _blur(_blur(noise))
    img = img + noise * (6.0 / noise.std())
    for _ in range(200 if dense else 40):
        w, h = max(1, int(rng.random() * width * 0.25)), max(1, int(rng.random() * height * 0.25))
        x0, y0 = int(rng.random() * max(width - w, 1)), int(rng.random() * max(height - h, 1))
        img[y0:y0 + h, x0:x0 + w] = lo + (hi - lo) * rng.random()
    for _ in range(12 if dense else 0):
        w, h = max(2, int(rng.random() * width * 0.15)), max(2, int(rng.random() * height * 0.15))
        x0, y0 = int(rng.random() * max(width - w, 1)), int(rng.random() * max(height - h, 1))
        a = lo + (hi - lo) * rng.random()
        region = img[y0:y0 + h, x0:x0 + w]
        across = rng.random() < 0.5
        (region[0::2] if across else region[:, 0::2]).fill_(a)
        (region[1::2] if across else region[:, 1::2]).fill_(hi + lo - a)
    img = img.clamp(lo, hi)
    if bits == 16:
        v = torch.round(img * (65535.0 / 255.0)).to(torch.int32)
        return torch.where(v > 32767, v - 65536, v).to(torch.int16)  # the 16 bits of an unsigned sample
    return torch.round(img).to(torch.uint8)


def _planes(width, height, chroma444, bits, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = random.Random(seed)
    return [_plane(w, h, i == 0, bits, chroma444, gen, rng)
            for i, (w, h) in enumerate(_plane_sizes(width, height, chroma444))]


def _ptrs(planes):
    return [p.data_ptr() for p in planes], [p.stride(0) * p.element_size() for p in planes]


class _Words:
    """Device words that belong to `owner`, which lives as long as a tensor of them does."""

    def __init__(self, owner, ptr, count):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<i4", "data": (ptr, False), "version": 2}


def _words(owner, ptr, count):
    return torch.as_tensor(_Words(owner, ptr, count), device="cuda")


_device = None


def _dev():
    """The program's device object: its encoders and decoders queue on one stream."""
    global _device
    if _device is None:
        _device = capi.Device()
    return _device


def prepare(case, seed):
    kind, bits = case["kind"], case["bits"]
    mask = capi.REFERENCE_PRECISION if case["precision"] == "reference" else 0
    frames = _frames(case)
    inputs = [_planes(w, h, c444, bits, seed * 64 + i) for i, (w, h, c444, _) in enumerate(frames)]
    torch.cuda.synchronize()
    state = {"kind": kind, "bits": bits, "budget": case["budget"]}
    if kind == "batch":
        # The shape that the library's autotuner settles on for such a mix, kept by the program.
        chroma = [capi.CHROMA_444 if c else capi.CHROMA_420 for _, _, c, _ in frames]
        batch = capi.Batch(_dev(), [(w, h, ch, b) for (w, h, _, b), ch in zip(frames, chroma)])
        batch.set_shape(persistent=False, frame_graphs=True, branches=4)
        outputs = [[torch.zeros_like(p) for p in f] for f in inputs]
        ins, outs = [_ptrs(f) for f in inputs], [_ptrs(f) for f in outputs]
        args = ([p for p, _ in ins], [s for _, s in ins], [b for *_, b in frames], [p for p, _ in outs],
                [s for _, s in outs])
        capi.check(batch.encode(*args), "batch_encode")
        streams, metas = [], []
        for i, (w, h, c444, b) in enumerate(frames):
            s, m = batch.device_bitstream(i)
            streams.append(_words(batch, s, b // 4))
            metas.append(_words(batch, m, 2 * _block_count(w, h, c444)))
        state.update(batch=batch, args=args, inputs=inputs, out=[streams, metas, outputs])
        torch.cuda.synchronize()
        for t in streams:
            t.zero_()  # what lies beyond the coded frame is no output
        torch.cuda.synchronize()
        return state

    width, height, c444, budget = frames[0]
    chroma = capi.CHROMA_444 if c444 else capi.CHROMA_420
    enc = capi.Encoder(_dev(), width, height, chroma, mask)
    planes = inputs[0]
    decoded = [torch.zeros_like(p) for p in planes]
    # The program has been coding for a while: one frame went through before.
    encode = enc.encode_device16 if bits == 16 else enc.encode_device
    if kind == "host":
        dtype = np.uint16 if bits == 16 else np.uint8
        dec = capi.Decoder(_dev(), width, height, chroma, mask)
        host_in = [p.cpu().pin_memory().numpy().view(dtype) for p in planes]
        host_out = [torch.zeros_like(p, device="cpu").pin_memory().numpy().view(dtype) for p in planes]
        state.update(enc=enc, dec=dec, host_in=host_in, host_out=host_out)
        run(state)
        for p in host_out:
            p.fill(0)
        return state
    encode(*_ptrs(planes), budget)
    torch.cuda.synchronize()
    s, m, capacity = enc.device_bitstream()
    words, meta = _words(enc, s, capacity), _words(enc, m, 2 * enc.layout().block_count_32x32)
    size = enc.size()
    words[(size + 3) // 4:].zero_()  # what lies beyond the coded frame is no output
    state.update(planes=planes, decoded=decoded, in_args=_ptrs(planes), out_args=_ptrs(decoded))
    if kind in ("encode", "roundtrip"):
        state.update(enc=enc, words=words, meta=meta)
    if kind == "decode":
        state.update(words=words.clone(), meta=meta.clone())
    if kind == "packets":
        capi.check(enc.encode_cpu([p.cpu().numpy() for p in planes], budget), "encode_cpu")
        data, packets = enc.packetize(PACKET_BYTES, budget)
        total = packets[-1][0] + packets[-1][1]
        state.update(data=torch.from_numpy(data[:total].copy()).cuda(), total=total, count=len(packets),
                     packets=torch.from_numpy(np.array(packets, np.int64)).cuda())
    if kind != "encode":
        state["dec"] = capi.Decoder(_dev(), width, height, chroma, mask)
        torch.cuda.synchronize()
        _decode(state)
    torch.cuda.synchronize()
    for p in decoded:
        p.zero_()
    torch.cuda.synchronize()
    return state


def _block_count(width, height, chroma444):
    enc = capi.Encoder(_dev(), width, height, capi.CHROMA_444 if chroma444 else capi.CHROMA_420)
    n = enc.layout().block_count_32x32
    enc.close()
    return n


def _decode(state):
    if state["kind"] == "packets":
        capi.check(state["dec"].decode_packets(state["data"].data_ptr(), state["total"], state["packets"].data_ptr(),
                                               state["count"], *state["out_args"]), "decode_packets")
        return
    decode = state["dec"].decode_blocks16 if state["bits"] == 16 else state["dec"].decode_blocks
    words = state["words"]
    decode(state["meta"].data_ptr(), words.data_ptr() + 8, words.numel() - 2, *state["out_args"])


def run(state):
    kind, budget = state["kind"], state["budget"]
    if kind == "batch":
        capi.check(state["batch"].encode(*state["args"]), "batch_encode")
        return state["out"]
    if kind == "host":
        capi.check(state["enc"].encode_cpu(state["host_in"], budget), "encode_cpu")
        data, packets = state["enc"].packetize(PACKET_BYTES, budget)
        dec = state["dec"]
        dec.clear()
        capi.check(dec.push_packet(data[:packets[-1][0] + packets[-1][1]]), "push_packet")
        code, planes = dec.decode_cpu(state["host_out"])
        capi.check(code, "decode_cpu")
        return [data, planes]
    if kind in ("encode", "roundtrip"):
        encode = state["enc"].encode_device16 if state["bits"] == 16 else state["enc"].encode_device
        encode(*state["in_args"], budget)
    if kind != "encode":
        _decode(state)
    if kind == "encode":
        return [state["words"], state["meta"]]
    if kind == "roundtrip":
        return [state["words"], state["meta"], state["decoded"]]
    return state["decoded"]


def work(case):
    """Planes and bitstream read and written once; the separable 9/7 transform
    (14 operations per sample and 4/3 of the samples over all levels) and one
    scaling, comparison and squared error per coefficient."""
    total_bytes, flops = 0.0, 0.0
    passes = {"encode": 1, "decode": 1, "packets": 1}.get(case["kind"], 2)
    for w, h, c444, budget in _frames(case):
        samples = sum(a * b for a, b in _plane_sizes(w, h, c444))
        total_bytes += passes * (samples * case["bits"] / 8 + budget)
        flops += passes * samples * 18.7
        if case["kind"] not in ("decode", "packets"):
            flops += samples * 4.0
    return {"bytes": total_bytes, "flops": flops}


def exact(case, seed):
    """None: bitstream words and samples are whole numbers, which stay equal."""
    return None
