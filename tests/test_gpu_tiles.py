"""Edges of the transform tiles, the quantiser and the block decoder on the GPU,
bit for bit against the CPU oracle:

  * planes whose rows and base addresses have no common alignment, at sizes
    around the 64-sample tiles and the 32-sample band tiles (the tile loader's
    vector, shifted and gathered paths; the stores' widths);
  * quantiser inputs on and next to the steps of the 8x8 scale code, and maxima
    on both sides of the fast path's limit;
  * damaged block payloads, with the right and with too small a word count (reads
    that leave the staged words).
"""
import numpy as np
import pytest

import oracle as O
from pyrowave_b200 import capi, synth

pytestmark = pytest.mark.gpu

# (width, height, 4:4:4, bits, bytes from a 16-byte boundary to the first sample, bytes added to each row)
PLANES = [
    (128, 128, True, 8, 0, 0),      # whole tiles, aligned
    (132, 130, False, 8, 1, 3),     # four samples past two tiles; odd base and pitch
    (190, 66, True, 8, 2, 1),       # two samples short of three tiles
    (194, 258, False, 8, 3, 2),
    (387, 129, True, 8, 0, 4),      # aligned base, odd width
    (1366, 770, False, 8, 0, 0),    # pitch of 1366 bytes
    (130, 128, True, 16, 0, 0),
    (257, 131, True, 16, 2, 2),     # 2-byte alignment only
    (322, 194, False, 16, 6, 6),
    (256, 64, True, 16, 8, 8),      # 8-byte alignment
]


@pytest.fixture(scope="module")
def device(gpu):
    dev = capi.Device()
    yield dev
    dev.close()


def _place(planes, base, pad):
    """The planes in one device allocation each, `base` bytes in, rows padded by `pad` bytes: (storage, pointers, strides)."""
    import torch

    store, ptrs, strides = [], [], []
    for p in planes:
        row = p.shape[1] * p.itemsize
        buf = np.full(base + (row + pad) * p.shape[0] + 64, 0xA5, np.uint8)
        for y in range(p.shape[0]):
            at = base + y * (row + pad)
            buf[at:at + row] = np.ascontiguousarray(p[y]).view(np.uint8)
        t = torch.from_numpy(buf).cuda()
        store.append(t)
        ptrs.append(t.data_ptr() + base)
        strides.append(row + pad)
    torch.cuda.synchronize()
    return store, ptrs, strides


@pytest.mark.parametrize("case", PLANES, ids=lambda c: f"{c[0]}x{c[1]}-{'444' if c[2] else '420'}-{c[3]}bit+{c[4]}+{c[5]}")
def test_unaligned_planes(device, case):
    import torch

    w, h, c444, bits, base, pad = case
    planes = synth.synth_frame(w, h, c444, w + h, 12, 4)
    if bits == 16:
        rng = np.random.default_rng(w)
        planes = [(p.astype(np.uint16) << 8) | rng.integers(0, 256, p.shape, dtype=np.uint16) for p in planes]
    budget = (w * h // 3) & ~3
    chroma = capi.CHROMA_444 if c444 else capi.CHROMA_420
    enc, dec = capi.Encoder(device, w, h, chroma), capi.Decoder(device, w, h, chroma)
    o = O.Oracle(w, h, c444)
    o.encode(planes, budget, sequence=1)
    keep, ptrs, strides = _place(planes, base, pad)
    (enc.encode_device16 if bits == 16 else enc.encode_device)(ptrs, strides, budget)
    d = enc.debug()
    assert int(d["error_flags"][0]) == 0
    assert np.array_equal(d["code_words"], o.code_words())
    assert np.array_equal(d["block_meta"], o.meta())
    pyr = torch.zeros(enc.layout().pyramid_size, dtype=torch.float32, device="cuda")
    enc.read_wavelet(pyr.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(pyr.cpu().numpy().view(np.uint32), o.dwt(planes).view(np.uint32))

    # Decoded planes, and nothing written beside them.
    ostream, opackets = o.packetize(8192, budget)
    p = o.parser()
    assert all(p.push(ostream[int(a):int(a + n)].tobytes()) for a, n in opackets)
    want = (o.idwt16 if bits == 16 else o.idwt)(o.dequant(*p.get()))
    out, optrs, ostrides = _place([np.zeros_like(q) for q in planes], base, pad)
    expect, _, _ = _place(want, base, pad)
    s, m, cap = enc.device_bitstream()
    (dec.decode_blocks16 if bits == 16 else dec.decode_blocks)(m, s + 8, cap - 2, optrs, ostrides)
    torch.cuda.synchronize()
    for i in range(3):
        assert torch.equal(out[i], expect[i]), f"plane {i}"


def _step_values(rng, count, top):
    """Magnitudes on the steps of the scale code (target * k / 8 with target = 2^e - 1/4), and one float to either side."""
    e = rng.integers(0, top, count)
    t = (2.0 ** e - 0.25).astype(np.float32)
    v = (t * rng.integers(4, 14, count).astype(np.float32) * np.float32(0.125)).astype(np.float32)
    side = rng.integers(-1, 2, count)
    return np.where(side < 0, np.nextafter(v, np.float32(0)),
                    np.where(side > 0, np.nextafter(v, np.float32(np.inf)), v)).astype(np.float32)


# (binary exponents of the values: lowest, highest; exponents of the planted steps)
@pytest.mark.parametrize("span", [(-4, 3, 4), (0, 14, 15), (-20, 1, 2), (14, 19, 18), (18, 27, 27)], ids=str)
def test_quantiser_steps(device, span):
    import torch

    lo, hi, top = span
    w, h, budget = 260, 196, 60000
    enc = capi.Encoder(device, w, h, capi.CHROMA_444)
    o = O.Oracle(w, h, True)
    rng = np.random.default_rng(hi + 100)
    n = enc.layout().pyramid_size
    pyr = (rng.standard_normal(n) * 2.0 ** rng.uniform(lo - 3, hi - 2, n)).astype(np.float32)
    pyr[rng.random(n) < 0.2] = 0.0
    pyr[rng.random(n) < 0.05] = -0.0
    at = rng.choice(n, n // 40, replace=False)
    pyr[at] = _step_values(rng, at.size, top) * np.where(rng.random(at.size) < 0.5, -1, 1).astype(np.float32)
    dev = torch.from_numpy(pyr).cuda()
    torch.cuda.synchronize()
    enc.encode_pre_transformed(dev.data_ptr(), budget, 1.0)
    o.encode_pyramid(pyr, budget, sequence=1, quant_scale=1.0)
    d = enc.debug()
    rc, dist, bk = o.rd()
    assert np.array_equal(d["code_words"], o.code_words())
    assert np.array_equal(d["rd_cost"].astype(np.uint32), rc)
    assert np.array_equal(d["rd_dist"].view(np.uint32), dist.view(np.uint32))
    assert np.array_equal(d["rd_bucket"].astype(np.uint32), bk)
    assert np.array_equal(d["quant"], o.quant())


@pytest.mark.parametrize("words", ["exact", "two"])
@pytest.mark.parametrize("damage", [0, 30, 600])
def test_damaged_blocks(device, words, damage):
    import torch

    w, h, budget = 640, 360, 60000
    o = O.Oracle(w, h, False)
    o.encode(synth.synth_frame(w, h, False, 3, 30, 6), budget, sequence=1)
    stream, packets = o.packetize(8192, budget)
    p = o.parser()
    assert all(p.push(stream[int(a):int(a + n)].tobytes()) for a, n in packets)
    offs, payload = p.get()
    payload = payload.copy()
    present = offs != 0xFFFFFFFF
    size = (payload[offs[present]] >> 16) & 0xFFF
    rng = np.random.default_rng(damage)
    at = rng.integers(0, payload.size, damage)
    payload[at] ^= (1 << rng.integers(0, 32, damage)).astype(np.uint32)
    want = o.dequant(offs, payload)
    meta = np.zeros((offs.size, 2), np.uint32)
    meta[present, 0] = offs[present]
    meta[present, 1] = size if words == "exact" else 2
    dec = capi.Decoder(device, w, h, capi.CHROMA_420)
    out = [torch.zeros(s, dtype=torch.uint8, device="cuda") for s in ((h, w), (h // 2, w // 2), (h // 2, w // 2))]
    m, q = torch.from_numpy(meta.view(np.int32)).cuda(), torch.from_numpy(payload.view(np.int32)).cuda()
    torch.cuda.synchronize()
    dec.decode_blocks(m.data_ptr(), q.data_ptr(), payload.size, [t.data_ptr() for t in out], [t.stride(0) for t in out])
    pyr = torch.zeros(dec.layout().pyramid_size, dtype=torch.float32, device="cuda")
    dec.read_wavelet(pyr.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(pyr.cpu().numpy().view(np.uint32), want.view(np.uint32))
