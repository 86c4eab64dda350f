"""The autotuner times the launches that its choices steer: each candidate's trial
of the guided sweep is the launch that a tick with that setting issues, and the
nine variants of the forward and of the inverse level-0 transform differ in it."""
import json

import pytest

from wema_b200 import cuda as wc

pytestmark = pytest.mark.gpu


def launches_of(fn, tmp_path):
    """(kernel name, grid) of every launch of fn(), in order."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        fn()
        torch.cuda.synchronize()
    path = str(tmp_path / "trace.json")
    prof.export_chrome_trace(path)
    ev = [e for e in json.load(open(path))["traceEvents"] if e.get("cat") == "kernel"]
    return [(e["name"], tuple(e["args"]["grid"])) for e in sorted(ev, key=lambda e: e["ts"])]


@pytest.fixture()
def settings():   # the choices as they were, afterwards
    keep = wc.iir_positions(0), wc.guided_rows(0), wc.dwt_variant(0, False), wc.dwt_variant(0, True)
    yield
    wc.set_iir_positions(0, keep[0])
    wc.set_guided_rows(0, keep[1])
    wc.set_dwt_variant(0, False, keep[2])
    wc.set_dwt_variant(0, True, keep[3])


def test_guided_trials(settings, tmp_path):
    import torch
    wc.autotune(0)
    trials = [x for x in launches_of(lambda: wc.autotune(0), tmp_path) if "k_guided_transfer" in x[0]]
    assert len(trials) == 18                     # three candidates, a warm-up and five launches each
    w, h = 3840, 8640                            # the trial's frame
    u8 = torch.full((h, w, 3), 90, dtype=torch.uint8, device="cuda")
    out = torch.empty_like(u8)
    b = wc.Batch(device=0, max_streams=1)
    sid = b.add(w, h, fps=30.0, amp=50.0)

    def ticks():
        for rows in (64, 128, 256):
            wc.set_guided_rows(0, rows)
            b.tick([sid], [u8], [out])
            b.sync()
    ticks()
    ticked = [x for x in launches_of(ticks, tmp_path) if "k_guided_transfer" in x[0]]
    b.close()
    assert len(ticked) == 3
    assert trials == [x for x in ticked for _ in range(6)]


def test_dwt_variants_differ(settings, tmp_path):
    wc.autotune(0)
    got = launches_of(lambda: wc.autotune(0), tmp_path)
    for kernel in ("k_dwt_fwd_multi", "k_dwt_inv_multi"):
        trials = [g for n, g in got if kernel in n]
        assert len(trials) == 54                 # nine variants, a warm-up and five launches each
        grids = [trials[6 * v] for v in range(9)]
        for unit in range(3):                    # three limits of CTAs per SM at each unit
            assert len({grids[3 * i + unit] for i in range(3)}) == 3, f"{kernel}: {grids}"
