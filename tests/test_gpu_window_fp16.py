"""The window filter with an FP16 ring (ring_fp16) at the window sizes and positions
its kernels divide at: 256-position tiles up to window 64 and 128 beyond, copies of
8 elements where the slots' rows start at 16 bytes or element by element, the
shortest and the longest window, mean and bilateral.  Against the FP64 filter over
the history as the ring holds it, rounded to FP16, the centre and the newest sample
with it.  The bar: the filter's sums are of `ws` FP32 terms, each addition within
2^-24 of its partial sum, with about 16 more roundings on the way to a delta:
(ws + 16) 2^-24 of the history's largest magnitude at a position, in L2."""
import numpy as np
import pytest

import fp64
from wema_b200 import cuda as wc
from wema_b200.synth import SynthSpec, SynthVideo

pytestmark = pytest.mark.gpu


def unique(flat6, dims):
    out, k = [], 0
    for sw, sh in dims:
        out.append(flat6[k:k + 3 * sw * sh])
        k += 6 * sw * sh
    return np.concatenate(out)


@pytest.mark.parametrize("w,h", [(64, 48), (63, 45), (30, 22)])
@pytest.mark.parametrize("ws", [4, 33, 64, 65, 256])
@pytest.mark.parametrize("bilateral", [False, True])
def test_fp16_ring(oracle, w, h, ws, bilateral):
    import torch
    u8 = SynthVideo(SynthSpec(w, h, 30.0, 5, [1.3], [0.4], max(2.0, min(w, h) / 5), 2.0)).frames(0, ws + 2)
    d_in, dims = torch.from_numpy(u8).cuda(), oracle.subband_dims(w, h)
    out = torch.empty((h, w, 3), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    s = wc.Session(width=w, height=h, fps=30.0, amp=40.0, f_low=0.5, f_high=3.0, window=ws, bilateral=bilateral,
                   use_iir=False, ring_fp16=True)
    hist = []
    for t in range(ws + 2):
        s.process_u8(d_in[t], out)
        s.sync()
        hist.append(unique(s.read(wc.READ_ORIG6), dims).astype(np.float16).astype(np.float64))
        if t + 1 < ws:
            continue
        x = np.stack(hist[-ws:])
        got = unique(s.read(wc.READ_DELTA6), dims).astype(np.float64)
        err = np.linalg.norm(got - fp64.window_delta(x, bilateral))
        assert err <= (ws + 16) * 2.0 ** -24 * np.linalg.norm(np.abs(x).max(axis=0)), f"frame {t}"
    s.close()
