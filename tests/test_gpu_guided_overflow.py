"""The guided transfer on float frames whose window sums overflow: a value of
1e20 by the frame's last corner makes E[I^2] infinite in every window that holds
it, so a = 0 and b = E[p] there, and outside the frame a = b = 0.  What is
added near the corner is then a number, large beyond the frame's own values and
odd in the corner's value: with +1e20 and -1e20 each pixel saturates to opposite
ends (a NaN would be 0 with both)."""
import numpy as np
import pytest

from wema_b200 import cuda as wc
from wema_b200.synth import SynthSpec, SynthVideo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(40, 24), (61, 33), (115, 20), (232, 49)])
def test_overflowing_sums(w, h):
    import torch
    rgb = SynthVideo(SynthSpec(w, h, 30.0, 5, [1.3], [0.4], 4.0, 2.0)).frames(0, 1)[0].astype(np.float32) / 255
    got = []
    for huge in (1e20, -1e20):
        rgb[h - 2, w - 2] = huge
        src, out = torch.from_numpy(rgb).cuda(), torch.full((h, w, 3), -1.0, device="cuda")
        out8 = torch.full((h, w, 3), 7, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        s = wc.Session(width=w, height=h, fps=30.0, amp=50.0, f_low=0.5, f_high=3.0)
        s.process_f32(src, d_out_f32=out, d_out_u8=out8)
        s.sync()
        s.close()
        assert np.array_equal(out8.cpu().numpy(), np.round(out.cpu().numpy() * 255).astype(np.uint8))
        got.append(out.cpu().numpy()[h - 6:, w - 6:].reshape(-1, 3))
    near = np.arange(36) != 4 * 6 + 4            # the corner's windows, without the value itself
    assert np.isin(got[0][near], (0, 1)).all()
    assert np.array_equal(got[0][near], 1 - got[1][near])
