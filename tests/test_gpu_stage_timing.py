"""Stage timing switched by another thread while frames are coded: every call
follows the switch's value when it began (a decode's small inverse levels share
launches without timing and have one each with it), so results stay the same."""
import threading

import numpy as np
import pytest

from pyrowave_b200 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,c444", [(256, 144, False), (640, 360, True)])
def test_switch_from_another_thread(gpu, w, h, c444):
    import torch

    dev = capi.Device()
    chroma = capi.CHROMA_444 if c444 else capi.CHROMA_420
    budget = (w * h // 4) & ~3
    planes = synth.synth_frame(w, h, c444, 3)
    enc, dec = capi.Encoder(dev, w, h, chroma), capi.Decoder(dev, w, h, chroma)
    assert enc.encode_cpu(planes, budget) == capi.PYROWAVE_SUCCESS
    data, packets = enc.packetize(2048, budget)
    data = torch.from_numpy(data.copy()).cuda()
    desc = torch.from_numpy(np.array(packets, np.int64)).cuda()
    src = [torch.from_numpy(np.ascontiguousarray(p)).cuda() for p in planes]
    out = [torch.zeros_like(p) for p in src]
    ins, outs = ([t.data_ptr() for t in x] for x in (src, out))
    strides = [t.stride(0) for t in src]

    def code(blocks):
        enc.encode_device(ins, strides, budget)
        if blocks:
            s, m, cap = enc.device_bitstream()
            dec.decode_blocks(m, s + 8, cap - 2, outs, strides)
        else:
            assert dec.decode_packets(data.data_ptr(), data.numel(), desc.data_ptr(), len(packets), outs,
                                      strides) == capi.PYROWAVE_SUCCESS
        torch.cuda.synchronize()
        return [t.cpu().numpy() for t in out]

    torch.cuda.synchronize()
    want = code(True)
    stop = threading.Event()

    def switch():
        on = True
        while not stop.is_set():
            dev.set_stage_timing(on)
            on = not on

    thread = threading.Thread(target=switch)
    thread.start()
    try:
        for i in range(100):
            for t in out:
                t.zero_()
            torch.cuda.synchronize()
            for got, ref in zip(code(i % 2 == 0), want):
                assert np.array_equal(got, ref), i
    finally:
        stop.set()
        thread.join()
    dev.set_stage_timing(False)
    assert all(np.array_equal(a, b) for a, b in zip(code(False), want))
