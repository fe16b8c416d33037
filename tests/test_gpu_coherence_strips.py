"""The coherence kernel at the edges of its tiles: every range window, window
heights with and without a compiled ring of rows, image widths around the
warps' strips, rows off the 16-byte boundaries, row pitches with a gap, zero
master and slave samples -- against the FP64 oracle, and the two copy paths
(16-byte pieces, single columns) bit for bit.

Tolerance: a window sum is a tree of FP32 adds, at most 13 deep vertically
(heights to 12) and 6 horizontally, over products of 2 roundings, so each of
the four sums is off by at most 21 x 2^-24 = 1.25e-6 of the sum of magnitudes,
which by Cauchy-Schwarz is at most sqrt(sum|s|^2 sum|m|^2): sqrt(2) x 1.25e-6
from the two cross sums, 1.25e-6 from the two powers, and under 0.6e-6 from
the two reciprocal square roots and five roundings after them: 3.6e-6."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 4e-6


def _run(T, m, s, win_rg, win_az, pad, off):
    """One job; rows of W + pad samples, the slave `off` samples into its buffer."""
    import torch
    L, W = m.shape[:2]
    P = W + pad
    dm = torch.zeros(L, P, dtype=torch.int32, device="cuda")
    dm[:, :W] = torch.from_numpy(np.ascontiguousarray(m).view(np.int32).reshape(L, W)).cuda()
    buf = torch.full((L * P * 2 + 2 * off,), 1e4, dtype=torch.float32, device="cuda")
    ds = buf[2 * off:].view(L, P, 2)
    ds[:, :W] = torch.from_numpy(s).cuda()
    dm[:, W:] = 0x01000100                      # the gap must not be read as samples
    coh = torch.full((L, P), -3.0, dtype=torch.float32, device="cuda")
    job = T.CohJob(master=dm.data_ptr(), master_pitch=P * 4, slave=ds.data_ptr(),
                   slave_pitch=P * 8, coh=coh.data_ptr(), coh_pitch=P * 4, lines=L, pixels=W)
    torch.cuda.synchronize()
    T.check(T.lib.tops_coherence(C.byref(job), 1, win_rg, win_az, None), "tops_coherence")
    torch.cuda.synchronize()
    out = coh.cpu().numpy()
    assert np.all(out[:, W:] == -3.0)
    return out[:, :W]


@pytest.mark.parametrize("win_az", [1, 2, 3, 4, 5, 6, 7, 8, 9, 12])
def test_coherence_strip_edges(T, O, win_az):
    rng = np.random.default_rng(win_az)
    for win_rg in range(1, 34):
        dx = (win_rg - 1) // 2
        tw = 4 * (32 - (dx + 3) // 4 - (win_rg - dx + 2) // 4)   # columns of a strip
        L = int(rng.integers(1, 45))
        W = max(1, int(rng.integers(0, 4)) * tw + int(rng.integers(-5, 6)))
        m = rng.integers(-900, 900, (L, W, 2), dtype=np.int16)
        s = (0.7 * m + rng.normal(0, 300, (L, W, 2))).astype(np.float32)
        m[rng.random((L, W)) < 0.05] = 0
        s[rng.random((L, W)) < 0.05] = 0
        m[L // 2:, : W // 3] = 0                # whole windows without power
        ref = O.coherence(m, s, win_rg, win_az)
        pad4 = -W % 4
        a = _run(T, m, s, win_rg, win_az, pad4, 0)             # rows on 16-byte boundaries
        b = _run(T, m, s, win_rg, win_az, pad4 + 1, 0)         # an odd pitch
        c = _run(T, m, s, win_rg, win_az, pad4, 1)             # an offset slave
        assert np.abs(a - ref).max() < TOL, (win_rg, L, W)
        assert np.array_equal(a, b) and np.array_equal(a, c), (win_rg, L, W)
