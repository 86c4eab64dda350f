"""The coarser levels of a small frame in one cluster, forward and inverse, at the
sizes where its split divides: one strip and just over, fewer rows than warps,
odd levels with stale entries, two and three levels, the largest size it takes
and the first one that it leaves to a launch per level.  Every plane is
bit-exact to the oracle; FP16 planes are the FP32 ones rounded."""
import numpy as np
import pytest

from test_gpu_parity import check_frame, frames_for, run_pair, torch_cuda  # noqa: F401
from wema_b200 import cuda as wc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,color", [
    (64, 64, True), (67, 65, False), (127, 700, False), (700, 127, True), (129, 131, True), (240, 136, False),
    (241, 137, False), (245, 143, True), (960, 576, False), (957, 573, True), (960, 580, False)])
def test_levels(oracle, torch_cuda, w, h, color):  # noqa: F811
    for t, so, sg, o, g_u8 in run_pair(oracle, torch_cuda, w, h, 3, color=color):
        check_frame(oracle, so, sg, o, g_u8, w, h, color, color)


@pytest.mark.parametrize("w,h", [(64, 66), (241, 139), (957, 573)])
def test_levels_fp16(torch_cuda, w, h):  # noqa: F811
    torch = torch_cuda
    u8 = torch.from_numpy(frames_for(w, h, 1)[0]).cuda()
    out = torch.empty_like(u8)
    got = []
    for h16 in (False, True):
        s = wc.Session(width=w, height=h, fps=30.0, amp=50.0, f_low=0.5, f_high=3.0, planes_fp16=h16)
        s.process_u8(u8, out)
        s.sync()
        got.append(s.read(wc.READ_ORIG6))
        s.close()
    assert np.array_equal(got[0].astype(np.float16).astype(np.float32), got[1])
