"""The transforms' sweeps at the widths where a CTA's warps go over from one strip
to two and to four (60 and 120 pairs of columns), with fewer and more rows than
warps: a batched stream, swept, equals the same stream alone, by its own route,
byte for byte, over first and steady frames; and the oracle's frames."""
import numpy as np
import pytest

from oracle_frames import assert_close, oracle_u8
from wema_b200 import cuda as wc
from wema_b200.synth import SynthSpec, SynthVideo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [3, 118, 120, 121, 122, 239, 240, 241, 242, 482])
@pytest.mark.parametrize("h", [1, 5, 18, 131])
def test_narrow(oracle, w, h):
    import torch
    F = 3
    u8 = SynthVideo(SynthSpec(w, h, 30.0, w + h, [1.2], [0.4], max(2.0, min(w, h) / 5), 2.0)).frames(0, F)
    d = torch.from_numpy(u8).cuda()
    kws = [dict(fps=30.0, amp=60.0, f_low=0.5, f_high=3.0, color=c) for c in (False, True)]
    b = wc.Batch(device=0, max_streams=2)
    ids = [b.add(w, h, **kw) for kw in kws]
    got = torch.empty((2, F, h, w, 3), dtype=torch.uint8, device="cuda")
    for t in range(F):
        b.tick(ids, [d[t], d[t]], [got[0][t], got[1][t]])
    b.sync()
    b.close()
    for k, kw in enumerate(kws):
        s = wc.Session(width=w, height=h, **kw)
        want = torch.empty((F, h, w, 3), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        for t in range(F):
            s.process_u8(d[t], want[t])
        s.sync()
        s.close()
        assert np.array_equal(got[k].cpu().numpy(), want.cpu().numpy())
        assert_close(got[k].cpu().numpy(), oracle_u8(oracle, u8, **kw), kw["color"])
