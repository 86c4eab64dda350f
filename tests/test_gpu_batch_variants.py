"""Batches whose ticks take the transforms by sweeps or by tiles: streams of one
storage type, of several, with FP64 state, at even and odd widths, luma and
colour, and ticks over part of them (so the form changes from tick to tick).
Every stream's frames equal those of the same stream alone, byte for byte."""
import numpy as np
import pytest

from wema_b200 import cuda as wc
from wema_b200.synth import SynthSpec, SynthVideo

pytestmark = pytest.mark.gpu

F16, F64 = dict(planes_fp16=True), dict(state_fp64=True)
BOTH = dict(planes_fp16=True, state_fp64=True)
MIXES = {
    "fp16_ragged": [(133, 71, dict(color=True, **F16)), (320, 96, F16), (57, 130, F16), (113, 54, F16)],
    "fp64_odd": [(133, 71, F64), (115, 54, dict(color=True, **F64)), (320, 96, F64), (17, 33, F64)],
    "fp32_fp16": [(133, 71, dict(color=True)), (320, 96, F16), (57, 130, {}), (113, 54, dict(color=True, **F16))],
    "fp32_fp64": [(133, 71, {}), (320, 96, F64), (57, 130, dict(color=True)), (113, 54, dict(color=True, **F64))],
    "all": [(133, 71, dict(color=True)), (320, 96, F16), (57, 130, BOTH), (113, 54, dict(color=True, **F64)),
            (240, 136, dict(color=True, **BOTH)), (64, 48, dict(edge_aware=False)), (16, 200, F64)],
}


@pytest.mark.parametrize("mix", sorted(MIXES))
@pytest.mark.parametrize("groups", [1, 2])
def test_equals_alone(mix, groups):
    import torch
    cfgs, F = MIXES[mix], 6
    data = [torch.from_numpy(SynthVideo(SynthSpec(w, h, 30.0, 3 + k, [1.2], [0.4], max(2.0, min(w, h) / 5), 2.0))
                             .frames(0, F)).cuda() for k, (w, h, _) in enumerate(cfgs)]
    base = dict(fps=30.0, amp=60.0, f_low=0.5, f_high=3.0)
    b = wc.Batch(device=0, max_streams=len(cfgs))
    b.set_groups(groups)
    ids = [b.add(w, h, **base, **kw) for w, h, kw in cfgs]
    alone = [wc.Session(width=w, height=h, **base, **kw) for w, h, kw in cfgs]
    part = {2: [0], 3: list(range(1, len(cfgs)))}        # ticks over some of the streams
    for t in range(F):
        now = part.get(t, range(len(cfgs)))
        outs = [torch.empty_like(data[k][t]) for k in now]
        b.tick([ids[k] for k in now], [data[k][t] for k in now], outs)
        b.sync()
        for k, o in zip(now, outs):
            want = torch.empty_like(o)
            torch.cuda.synchronize()
            alone[k].process_u8(data[k][t], want)
            alone[k].sync()
            assert np.array_equal(o.cpu().numpy(), want.cpu().numpy()), f"stream {k}, tick {t}"
    for s in alone:
        s.close()
    b.close()
