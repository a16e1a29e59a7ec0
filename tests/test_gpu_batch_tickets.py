"""The persistent batch kernel's two forms, which differ in when a CTA takes its
next ticket (a stage with at least two items per CTA, or none), against the
oracle: one and two frames at 1, 2 and 4 CTAs per SM, which puts the line (296,
592, 1184 items on 148 SMs) on either side of a 1080p frame's largest stage (510
items) and of two 360p frames'."""
import pytest

from pyrowave_b200 import capi, synth
from test_gpu_batch import _check_against_oracle, _ptrs

pytestmark = pytest.mark.gpu

FRAMES = {
    "1080p": [(1920, 1080, False, 400000)],
    "two 360p": [(640, 360, False, 40000), (640, 360, True, 60000)],
    "tiny and 1080p": [(34, 30, True, 20000), (1920, 1080, False, 400000)],
}


@pytest.mark.parametrize("name", list(FRAMES))
@pytest.mark.parametrize("ctas_per_sm", [1, 2, 4])
def test_ticket_forms(gpu, name, ctas_per_sm):
    import torch

    dev = capi.Device()
    frames = FRAMES[name]
    planes = [synth.synth_frame(w, h, c444, 80 + i) for i, (w, h, c444, _) in enumerate(frames)]
    dev_planes = [[torch.from_numpy(p).cuda() for p in pl] for pl in planes]
    batch = capi.Batch(dev, [(w, h, capi.CHROMA_444 if c else capi.CHROMA_420, b) for w, h, c, b in frames])
    outs = [[torch.zeros_like(p) for p in pl] for pl in dev_planes]
    in_ptrs, in_strides = _ptrs(dev_planes)
    out_ptrs, out_strides = _ptrs(outs)
    budgets = [b for *_, b in frames]
    batch.set_shape(persistent=True, ctas_per_sm=ctas_per_sm)
    torch.cuda.synchronize()
    assert batch.encode(in_ptrs, in_strides, budgets, out_ptrs, out_strides) == capi.PYROWAVE_SUCCESS
    torch.cuda.synchronize()
    _check_against_oracle(batch, frames, planes, outs, budgets, 1, f"{name}, {ctas_per_sm} CTAs per SM")
    batch.close()
    dev.close()
