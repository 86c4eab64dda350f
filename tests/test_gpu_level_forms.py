"""A stream's levels by tiles or by sweeps: frames on either side of each line
between them (luma 0.6, 1.2, 3 and 5 million pixels; colour 0.2, 0.25, 0.64, 1 and 4
million, widths that are a multiple of 4 and not; levels in one cluster and apart).
The batched stream, always swept, gives the same bytes; so do float frames of the
same values; and with FP16 planes and FP64 state."""
import numpy as np
import pytest

from wema_b200 import cuda as wc

pytestmark = pytest.mark.gpu

LUMA = [(999, 600), (1001, 600), (1095, 1095), (1096, 1096), (2236, 2236), (2237, 2236), (3463, 3465), (3465, 3465), (640, 578), (642, 579)]
COLOR = [(447, 447), (448, 447), (499, 500), (501, 500), (502, 499), (800, 799), (1001, 800), (999, 1000), (1002, 1000),
         (1999, 2000), (2001, 2000), (320, 240), (640, 360)]


@pytest.mark.parametrize("w,h,color", [(w, h, False) for w, h in LUMA] + [(w, h, True) for w, h in COLOR])
@pytest.mark.parametrize("variant", [{}, dict(planes_fp16=True), dict(state_fp64=True)])
def test_forms_equal(w, h, color, variant):
    import torch
    F = 2
    g = torch.Generator(device="cuda").manual_seed(w + h)
    base = torch.rand((1, 3, h // 16 + 2, w // 16 + 2), generator=g, device="cuda")
    base = torch.nn.functional.interpolate(base, size=(h, w), mode="bilinear")[0].permute(1, 2, 0) * 200 + 20
    u8 = torch.stack([(base + 2 * torch.randn(base.shape, generator=g, device="cuda")).clamp(0, 255).to(torch.uint8)
                      for _ in range(F)])
    kw = dict(fps=30.0, amp=60.0, f_low=0.5, f_high=3.0, color=color, **variant)
    b = wc.Batch(device=0, max_streams=1)
    sid = b.add(w, h, **kw)
    s, f = wc.Session(inspect=False, width=w, height=h, **kw), wc.Session(inspect=False, width=w, height=h, **kw)
    for t in range(F):
        ob, os, of = (torch.full_like(u8[0], 1 + k) for k in range(3))
        f32 = torch.from_numpy(u8[t].cpu().numpy().astype(np.float32) / np.float32(255)).cuda()
        torch.cuda.synchronize()
        b.tick([sid], [u8[t]], [ob])
        s.process_u8(u8[t], os)
        f.process_f32(f32, d_out_u8=of)
        b.sync(), s.sync(), f.sync()
        assert torch.equal(ob, os), f"frame {t}: batched"
        assert torch.equal(of, os), f"frame {t}: float frames"
    b.close(), s.close(), f.close()
