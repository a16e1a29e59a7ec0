"""Device-side packet assembly at the edges of its work split, against the oracle
as in test_gpu_packets: packet sizes around the limit of the parallel item
search (8192 words), packets that hold as many items as fit, and packet counts
around a warp (32) and the scan's 1024 threads, of one frame and of two."""
import numpy as np
import pytest

import oracle as O
from oracle_codec import oracle_decode
from pyrowave_b200 import capi, synth
from test_gpu_packets import _device_decode, _frame_packets

pytestmark = pytest.mark.gpu

W, H, BUDGET = 640, 360, 120000


@pytest.fixture(scope="module")
def frames(gpu):
    """(decoder, packets of one block or so each of two frames in sequence)."""
    dev = capi.Device()
    enc = capi.Encoder(dev, W, H, capi.CHROMA_420)
    pa, pb = (_frame_packets(enc, synth.synth_frame(W, H, False, seed), BUDGET, 64) for seed in (3, 4))
    assert len(pa) > 100
    yield capi.Decoder(dev, W, H, capi.CHROMA_420), pa, pb
    dev.close()


def _check(dec, packets):
    o = O.Oracle(W, H, False)
    op = o.parser()
    invalid = sum(not op.push(p) for p in packets)
    want = oracle_decode(o, packets)
    got, st = _device_decode(dec, packets, [p.shape for p in synth.synth_frame(W, H, False, 3)])
    assert st.invalid_packets == invalid
    for i in range(3):
        assert np.array_equal(got[i], want[i]), f"plane {i} differs"


@pytest.mark.parametrize("size", [8, 16, 4096, 32760, 32764, 32768, 32772, 65536])
def test_packet_sizes(frames, size):
    """The frame's items in one packet of `size` bytes, whole items then sequence
    headers, the rest in its own packets."""
    dec, pa, _ = frames
    header, blob, n = pa[0][:8], b"", 0
    while n < len(pa) and len(blob) + len(pa[n]) <= size:
        blob += pa[n]
        n += 1
    blob += header * ((size - len(blob)) // 8)
    blob += b"\0" * (size - len(blob))  # four bytes left over: an invalid packet
    _check(dec, [blob] + pa[max(n, 1):])


@pytest.mark.parametrize("size", [4096, 32768, 32776])
def test_packet_of_headers(frames, size):
    dec, pa, pb = frames
    _check(dec, [pa[0][:8] * (size // 8)] + pa[1:] + [pb[0][:8] * (size // 8)] + pb[:20])


@pytest.mark.parametrize("count", [1, 2, 31, 32, 33, 64, 65, 1023, 1024, 1025, 2049])
@pytest.mark.parametrize("second", [0, 1, 40])
def test_packet_counts(frames, count, second):
    """`count` packets, repeated as needed; the last `second` are the next frame's."""
    dec, pa, pb = frames
    second = min(second, count)
    packets = (pa * (count // len(pa) + 1))[:count - second] + pb[:second]
    assert len(packets) == count
    _check(dec, packets)
