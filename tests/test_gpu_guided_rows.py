"""The guided transfer's row forms give the same bytes: RGB24 rows of any width
and alignment (cut from aligned words, written back as words with byte ends)
equal the float-frame form, pixel by pixel, fed the same values.  Sizes: around
a lane's 4 columns, a strip's 112 output columns and a segment's 16 rows."""
import numpy as np
import pytest

from wema_b200 import cuda as wc
from wema_b200.synth import SynthSpec, SynthVideo

pytestmark = pytest.mark.gpu


def frames(w, h, n, seed):
    return SynthVideo(SynthSpec(w, h, 30.0, seed, [1.1], [0.4], max(2.0, min(w, h) / 5), 2.0)).frames(0, n)


@pytest.mark.parametrize("w,h,off_in,off_out", [
    (4, 16, 0, 0), (5, 17, 0, 0), (7, 9, 1, 3), (111, 16, 0, 0), (112, 31, 2, 0), (113, 33, 0, 1),
    (115, 48, 3, 2), (225, 15, 0, 0), (341, 65, 1, 1), (640, 32, 0, 2), (3, 20, 0, 0)])
def test_row_forms_equal(w, h, off_in, off_out):
    import torch
    F = 3
    u8 = frames(w, h, F, seed=w + h)
    kw = dict(width=w, height=h, fps=30.0, amp=90.0, f_low=0.5, f_high=3.0)
    a, b = wc.Session(**kw), wc.Session(**kw)
    n = 3 * w * h
    src, dst = torch.full((n + 64,), 0xA5, dtype=torch.uint8, device="cuda"), \
        torch.full((n + 64,), 0xA5, dtype=torch.uint8, device="cuda")
    out = torch.empty((h, w, 3), dtype=torch.uint8, device="cuda")
    for t in range(F):
        src[16 + off_in:16 + off_in + n] = torch.from_numpy(u8[t].reshape(-1)).cuda()
        dst.fill_(0xA5)
        f32 = torch.from_numpy(u8[t].astype(np.float32) / np.float32(255)).cuda()
        torch.cuda.synchronize()
        a.process_u8(src[16 + off_in:], dst[16 + off_out:])
        b.process_f32(f32, d_out_u8=out)
        a.sync()
        b.sync()
        got = dst.cpu().numpy()
        assert np.array_equal(got[16 + off_out:16 + off_out + n].reshape(h, w, 3), out.cpu().numpy()), f"frame {t}"
        assert (got[:16 + off_out] == 0xA5).all() and (got[16 + off_out + n:] == 0xA5).all(), "bytes beside the frame"
    a.close()
    b.close()
