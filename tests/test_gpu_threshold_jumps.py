"""The exact threshold's running sums over jumps that they still resolve: in each of
the 8 lanes and each quarter of a sub-chunk an element of 2 to 2^6 times the lane's
sum so far, among small values and among multiples of 2^-13 (whose increments meet
exact halves), at every alignment.  The sum and the threshold are the oracle's bit
for bit; an ordinary element in any lane or quarter changes the oracle's sum, so a
wrong one could not pass."""
import numpy as np
import pytest

from wema_b200 import cuda as wc

pytestmark = pytest.mark.gpu


def arrays(n, kind):
    """(the array, indices of ordinary elements: one of each lane and quarter)."""
    rng = np.random.default_rng(n)
    if kind == "small":
        x = (rng.standard_normal(n) * 0.001).astype(np.float32)
    else:
        x = rng.integers(-4096, 4097, n).astype(np.float32) * np.float32(2.0 ** -13)
    rows = n // 8                                       # elements per lane, 64 to a quarter of a sub-chunk
    plain = []
    for lane in range(8):
        for q in range(4):
            e = [r for r in range(q * 64 + 5 * lane + 1, rows, 256)]
            if not e:
                continue
            plain.append(8 * e[-1] + lane)
            if (lane + q) % 4 == 0:                     # one jump per lane, in a quarter of its own
                at = e[len(e) // 2] + 7
                if at < rows:
                    s = np.abs(x[lane:8 * at:8].astype(np.float64)).sum()
                    x[8 * at + lane] = np.float32(s * 2.0 ** (1 + lane % 6)) * (-1) ** lane
    return x, plain


@pytest.mark.parametrize("n", [2048, 2049, 6 * 2048 + 5, 40 * 2048 + 1023, 300001])
@pytest.mark.parametrize("kind", ["small", "halves"])
def test_jumps(oracle, n, kind):
    import torch
    x, plain = arrays(n, kind)
    want, thr = np.float32(oracle.mag_sum(x)), np.float32(oracle.threshold(x))
    assert len(plain) == 32
    for i in plain:
        y = x.copy()
        y[i] += 0.25 if y[i] >= 0 else -0.25
        assert np.float32(oracle.mag_sum(y)) != want, i
    for off in range(4):
        buf = torch.zeros(n + 8, dtype=torch.float32, device="cuda")
        buf[off:off + n] = torch.from_numpy(x).cuda()
        got = wc.threshold_flat(buf[off:off + n])
        assert got[1].view(np.uint32) == want.view(np.uint32) and got[0].view(np.uint32) == thr.view(np.uint32)
