"""Device-side packet assembly of lists whose byte ranges overlap, against the
oracle as in test_gpu_packets: each packet counts as if its bytes were pushed by
themselves, whatever other packets hold the same bytes."""
import numpy as np
import pytest

import oracle as O
from oracle_codec import oracle_decode
from pyrowave_b200 import capi, synth

pytestmark = pytest.mark.gpu

W, H, C444, BUDGET = 960, 540, True, 31000


@pytest.fixture(scope="module")
def stream(gpu):
    """(decoder, one frame's sequence header, a hundred times, and blocks as bytes, byte offset of each block)."""
    dev = capi.Device()
    enc = capi.Encoder(dev, W, H, capi.CHROMA_444)
    assert enc.encode_cpu(synth.synth_frame(W, H, C444, 3), BUDGET) == capi.PYROWAVE_SUCCESS
    data, packets = enc.packetize(1 << 20, BUDGET)
    assert len(packets) == 1
    data = data[:8].tobytes() * 99 + data[:packets[0][1]].tobytes()
    words, blocks, at = np.frombuffer(data, np.uint32), [], 200
    while at < words.size:
        blocks.append(4 * at)
        at += (int(words[at]) >> 16) & 0xFFF
    # One packet of the parallel item search, with more items than the block pass has threads.
    assert len(data) <= 32768 and 100 + len(blocks) > 256
    yield capi.Decoder(dev, W, H, capi.CHROMA_444), data, blocks
    dev.close()


def _lists(size, blocks):
    half, quarter = blocks[len(blocks) // 2], blocks[len(blocks) // 4]
    return {
        "with and without the header": [(0, size), (8, size - 8)],
        "without, then with the header": [(8, size - 8), (0, size)],
        "the same range twice": [(0, size), (0, size)],
        "one start, several ends": [(0, half), (0, size), (0, quarter + 4), (0, half)],
        "from every block to the end": [(0, size)] + [(b, size - b) for b in blocks],
        "each block beside the whole": [(b, e - b) for b, e in zip(blocks, blocks[1:] + [size])] + [(0, size)],
        "halves that overlap": [(0, half), (quarter, size - quarter), (half, size - half)],
        "without the beginning": [(quarter, size - quarter), (half, size - half)],
    }


@pytest.mark.parametrize("name", list(_lists(1024, list(range(8, 512, 8)))))
def test_overlapping_ranges(stream, name):
    import torch

    dec, data, blocks = stream
    ranges = _lists(len(data), blocks)[name]
    packets = [data[a:a + n] for a, n in ranges]
    o = O.Oracle(W, H, C444)
    op = o.parser()
    invalid = sum(not op.push(p) for p in packets)
    want = oracle_decode(o, packets)
    buf = torch.from_numpy(np.frombuffer(data, np.uint8).copy()).cuda()
    desc = torch.from_numpy(np.array(ranges, np.int64)).cuda()
    for _ in range(8):
        out = [torch.full((H, W), 0x33, dtype=torch.uint8, device="cuda") for _ in range(3)]
        torch.cuda.synchronize()
        assert dec.decode_packets(buf.data_ptr(), len(data), desc.data_ptr(), len(ranges), [t.data_ptr() for t in out],
                                  [t.stride(0) for t in out]) == capi.PYROWAVE_SUCCESS
        st = dec.packet_status()
        torch.cuda.synchronize()
        assert st.invalid_packets == invalid
        assert (st.sequence != 0xFFFFFFFF and st.decoded_blocks >= st.total_blocks) == op.ready(False)
        for i in range(3):
            assert np.array_equal(out[i].cpu().numpy(), want[i]), f"plane {i}"
