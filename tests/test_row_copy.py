"""What the forward transform reads of a frame: the copies of its rows' parts stay
within the aligned 4-byte words that hold the frame's bytes (on the CPU, over the
header that the kernel takes them from); and on the GPU the bytes beside a frame do
not show in its output."""
import os
import subprocess

import numpy as np
import pytest

from wema_b200 import cuda as wc

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_copies_stay_in_the_frame(tmp_path):
    exe = str(tmp_path / "row_copy")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "wema_b200", "csrc"),
                    os.path.join(ROOT, "tests", "c", "row_copy.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,color", [(1, 1, False), (5, 3, True), (43, 30, False), (129, 17, True), (250, 40, False)])
def test_bytes_beside_the_frame(w, h, color):
    import torch
    n = 3 * w * h
    rng = np.random.default_rng(w)
    u8 = torch.from_numpy(rng.integers(0, 256, (2, n), dtype=np.uint8)).cuda()
    want = None
    for off in range(16):
        s = wc.Session(width=w, height=h, fps=30.0, amp=60.0, f_low=0.5, f_high=3.0, color=color)
        buf, out = torch.empty(n + 64, dtype=torch.uint8, device="cuda"), torch.empty((2, h, w, 3), dtype=torch.uint8,
                                                                                    device="cuda")
        for t in range(2):
            buf.fill_(16 * off + t)
            buf[16 + off:16 + off + n] = u8[t]
            torch.cuda.synchronize()
            s.process_u8(buf[16 + off:], out[t])
            s.sync()
        s.close()
        got = out.cpu().numpy()
        want = got if want is None else want
        assert np.array_equal(got, want), f"frame at byte {off} of 16"
