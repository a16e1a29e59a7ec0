"""Where the coder changes form by size or type, bit for bit against the CPU oracle:

  * every 8-bit and every 16-bit sample value through the division-free UNORM
    conversion, in planes read by vectors and sample by sample;
  * small inverse levels in pairs of one launch with any one of their levels in
    FP16 storage;
  * the packer's two forms, at a block count on either side of its line (4736);
  * the quantiser with one warp per row of 8x8 blocks (from 297 blocks on) at the
    steps of the scale code and both sides of the short form's limit.
"""
import numpy as np
import pytest

import oracle as O
from oracle_codec import oracle_frame, words_as_bytes
from pyrowave_b200 import capi, synth
from test_gpu_batch import _copy_device_words
from test_gpu_tiles import _place, _step_values

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device(gpu):
    dev = capi.Device()
    yield dev
    dev.close()


@pytest.mark.parametrize("bits,base,pad", [(8, 0, 0), (8, 1, 2), (16, 0, 0), (16, 2, 2)])
def test_every_sample_value(device, bits, base, pad):
    import torch

    w, h = 256, 256
    values = np.random.default_rng(bits).permutation(65536).reshape(h, w)
    dtype = np.uint16 if bits == 16 else np.uint8
    planes = [(v & (2 ** bits - 1)).astype(dtype) for v in (values, values.T, values[::-1])]
    enc = capi.Encoder(device, w, h, capi.CHROMA_444)
    keep, ptrs, strides = _place(planes, base, pad)
    (enc.encode_device16 if bits == 16 else enc.encode_device)(ptrs, strides, 60000)
    pyr = torch.zeros(enc.layout().pyramid_size, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    enc.read_wavelet(pyr.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(pyr.cpu().numpy().view(np.uint32), O.Oracle(w, h, True).dwt(planes).view(np.uint32))


@pytest.mark.parametrize("mask", [0x01, 0x02, 0x04, 0x08, 0x10, 0x06, 0x18, 0x0A, 0x15])
@pytest.mark.parametrize("w,h,c444", [(300, 200, False), (260, 196, True), (1280, 720, False)])
def test_pairs_with_one_level_in_fp16(device, mask, w, h, c444):
    import torch

    budget = (w * h // 5) & ~3
    chroma = capi.CHROMA_444 if c444 else capi.CHROMA_420
    planes = synth.synth_frame(w, h, c444, mask)
    data, want = oracle_frame(w, h, c444, planes, budget, 1, fp16_mask=mask)
    enc, dec = capi.Encoder(device, w, h, chroma, mask), capi.Decoder(device, w, h, chroma, mask)
    src = [torch.from_numpy(np.ascontiguousarray(p)).cuda() for p in planes]
    out = [torch.zeros_like(p) for p in src]
    torch.cuda.synchronize()
    enc.encode_device([t.data_ptr() for t in src], [t.stride(0) for t in src], budget)
    assert enc.size() == data.size
    s, m, _ = enc.device_bitstream()
    assert np.array_equal(words_as_bytes(_copy_device_words(s, data.size // 4)), data)
    dec.decode_blocks(m, s + 8, data.size // 4 - 2, [t.data_ptr() for t in out], [t.stride(0) for t in out])
    torch.cuda.synchronize()
    for i in range(3):
        assert np.array_equal(out[i].cpu().numpy(), want[i]), f"plane {i}"


@pytest.mark.parametrize("w,h,blocks", [(1216, 1232, 4674), (1616, 900, 4794)])
@pytest.mark.parametrize("bytes_per_sample", [0.005, 0.1, 2.0])
def test_packer_forms(device, w, h, blocks, bytes_per_sample):
    import torch

    budget = int(3 * w * h * bytes_per_sample) & ~3
    planes = synth.synth_frame(w, h, True, 5)
    enc = capi.Encoder(device, w, h, capi.CHROMA_444)
    assert enc.layout().block_count_32x32 == blocks
    src = [torch.from_numpy(np.ascontiguousarray(p)).cuda() for p in planes]
    torch.cuda.synchronize()
    for sequence in (1, 2):  # the second frame meets the first one's magnitudes in rows that code nothing
        frame = planes if sequence == 2 else [p[::-1] for p in planes]
        put = src if sequence == 2 else [torch.flip(t, [0]) for t in src]
        torch.cuda.synchronize()
        enc.encode_device([t.data_ptr() for t in put], [t.stride(0) for t in put], budget)
        o = O.Oracle(w, h, True)
        o.encode([np.ascontiguousarray(p) for p in frame], budget, sequence=sequence)
        ostream, opackets = o.packetize(1 << 30, budget)
        total = int(sum(int(n) for _, n in opackets))
        assert enc.size() == total
        s, _, _ = enc.device_bitstream()
        assert np.array_equal(words_as_bytes(_copy_device_words(s, total // 4)), ostream[:total])


@pytest.mark.parametrize("span", [(-4, 3, 4), (0, 14, 15), (14, 19, 18)], ids=str)
def test_quantiser_steps_one_warp_per_row(device, span):
    import torch

    lo, hi, top = span
    w, h, budget = 640, 360, 200000
    enc = capi.Encoder(device, w, h, capi.CHROMA_444)
    assert enc.layout().block_count_32x32 > 296
    o = O.Oracle(w, h, True)
    rng = np.random.default_rng(hi + 200)
    n = enc.layout().pyramid_size
    pyr = (rng.standard_normal(n) * 2.0 ** rng.uniform(lo - 3, hi - 2, n)).astype(np.float32)
    pyr[rng.random(n) < 0.2] = 0.0
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
