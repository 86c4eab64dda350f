"""The exact threshold where its increments round exact halves and where a
sub-chunk is not 16-byte aligned: flat arrays of coarse values (every running
sum past a few elements meets halves) at each alignment, with single values
that leave the binade, bit for bit against the oracle's sum."""
import numpy as np
import pytest

from wema_b200 import cuda as wc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [7, 8, 2047, 2048, 2049, 6 * 2048 + 5, 40 * 2048 + 1023])
@pytest.mark.parametrize("off", [0, 1, 2, 3])
@pytest.mark.parametrize("kind", ["halves", "mixed", "jump"])
def test_threshold_halves(oracle, n, off, kind):
    import torch
    rng = np.random.default_rng(n + 17 * off)
    if kind == "halves":      # multiples of 2^-13: halves from sums of 2^11 on
        x = rng.integers(-4096, 4097, n).astype(np.float32) * np.float32(2.0 ** -13)
        x[::7] += np.float32(64.0)
    elif kind == "mixed":     # the sums pass through every step of halves
        x = (rng.standard_normal(n) * 0.01).astype(np.float16).astype(np.float32)
    else:                     # single elements that leave the binade
        x = (rng.standard_normal(n) * 0.001).astype(np.float32)
        x[n // 2] = np.float32(3.0e4)
        x[n // 3] = np.float32(2.0 ** 100)
    want = oracle.threshold(x)
    buf = torch.zeros(n + 8, dtype=torch.float32, device="cuda")
    buf[off:off + n] = torch.from_numpy(x).cuda()
    got, _ = wc.threshold_flat(buf[off:off + n])
    assert np.float32(got).view(np.uint32) == np.float32(want).view(np.uint32)
