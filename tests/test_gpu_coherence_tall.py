"""Coherence windows taller than the compiled heights: whole and partial groups
of 4 output rows, images shorter than the window, segments cut at every row
count, both copy paths -- against the FP64 oracle, the paths bit for bit.

Tolerance: the rows that a group's 4 windows share are added one after another,
so a window sum is a chain of at most win_az + 2 FP32 adds and a horizontal tree
of 6, over products of 2 roundings: each of the four sums is off by at most
(win_az + 10) 2^-24 of the sum of magnitudes, which by Cauchy-Schwarz is at most
sqrt(sum|s|^2 sum|m|^2): sqrt(2) times that from the two cross sums, once from
the two powers, and under 0.6e-6 from the two reciprocal square roots and five
roundings after them."""
import numpy as np
import pytest

from test_gpu_coherence_strips import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("win_az", [7, 24, 65, 130])
def test_tall_windows(T, O, win_az):
    rng = np.random.default_rng(win_az)
    tol = 2.42 * (win_az + 10) * 2.0 ** -24 + 0.6e-6
    for L in (1, 3, 4, 5, 41, 130):
        for win_rg in (1, 6, 10, 33):
            W = int(rng.integers(90, 131))
            m = rng.integers(-900, 900, (L, W, 2), dtype=np.int16)
            s = (0.7 * m + rng.normal(0, 300, (L, W, 2))).astype(np.float32)
            s[rng.random((L, W)) < 0.05] = 0
            ref = O.coherence(m, s, win_rg, win_az)
            a = _run(T, m, s, win_rg, win_az, -W % 4, 0)
            assert np.abs(a - ref).max() < tol, (win_rg, L, W)
            assert np.array_equal(a, _run(T, m, s, win_rg, win_az, -W % 4, 1)), (win_rg, L, W)
