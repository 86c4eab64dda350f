"""The window filter at the window sizes and positions its kernels divide at
(256- and 128-position tiles, 16-byte rows or not, the shortest and longest
window): deltas against the oracle's within the stage's bar, relative L2 1e-5."""
import numpy as np
import pytest

from wema_b200 import cuda as wc
from wema_b200.synth import SynthSpec, SynthVideo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,ws,bilateral", [
    (64, 48, 4, True), (64, 48, 32, True), (63, 45, 33, True), (40, 32, 64, True), (37, 29, 65, True),
    (24, 18, 256, True), (64, 48, 32, False), (63, 45, 17, False), (24, 18, 256, False)])
def test_window_deltas(oracle, w, h, ws, bilateral):
    import torch
    u8 = SynthVideo(SynthSpec(w, h, 30.0, 5, [1.3], [0.4], max(2.0, min(w, h) / 5), 2.0)).frames(0, ws + 2)
    rgb = oracle.u8_to_float(u8)
    kw = dict(width=w, height=h, fps=30.0, amp=40.0, f_low=0.5, f_high=3.0, window=ws, bilateral=bilateral,
              use_iir=False)
    so, sg = oracle.stream(**kw), wc.Session(**kw)
    N = oracle.positions(w, h)
    d_in = torch.from_numpy(u8).cuda()
    out = torch.empty((h, w, 3), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    # the 6-slot indices of slots 0-2 (the others mirror them)
    n, keep = 0, []
    a, b, levels, m = w, h, 0, min(w, h)
    while m >= 16 and levels < 4:
        m //= 2
        levels += 1
    for _ in range(max(levels, 1)):
        a, b = (a + 1) // 2, (b + 1) // 2
        keep.append(np.arange(n, n + 3 * a * b))
        n += 6 * a * b
    keep = np.concatenate(keep)
    for t in range(ws + 2):
        so.process(rgb[t])
        sg.process_u8(d_in[t], out)
        if t + 1 < ws:
            continue
        sg.sync()
        got = sg.read(wc.READ_DELTA6)[keep].astype(np.float64)
        want = so.get(3, N)[keep].astype(np.float64)
        assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want), f"frame {t}"
    sg.close()
