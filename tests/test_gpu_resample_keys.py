"""Resample jobs whose range key changes every few rows, or turns round inside
the burst, and rows of up to 9 azimuth runs, in both precision modes: against
the FP64 oracle, row subsets bit for bit (a short job finds its keys in the run
tables, a long one pixel by pixel), and their cost beside a burst of one key.

Tolerance: the kernel's sums and phases are FP32 on FP64 positions and phases;
each of the two sine / cosine pairs is good to 2^-21.4 = 3.6e-7 of the
amplitude and the 12 + 12 tap sums and the rotations round to about 24 x 2^-25
= 7e-7 at worst, so 2e-6 relative RMS bounds an exact implementation."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_rms
from test_gpu_resample_strips import _inputs

pytestmark = pytest.mark.gpu

TOL = 2e-6


class _Job:
    """A job of one burst on the device; `pad` spare samples in a slave row."""

    def __init__(self, T, kw, prec, rows=None, pad=0):
        import torch
        L, W = kw["slave"].shape[:2]
        self.T, self.prec, self.rows = T, T.PREC_SPLIT if prec == "split" else T.PREC_FP64, rows
        self.slave = torch.zeros(L, W + pad, 2, dtype=torch.int16, device="cuda")
        self.slave[:, :W] = torch.from_numpy(kw["slave"]).cuda()
        box = [int(v) for v in kw["mbox"]]
        self.out = torch.full((box[3] - box[2] + 1, W, 2), 7.0, device="cuda")
        self.par = [torch.from_numpy(np.ascontiguousarray(kw[k])).cuda() for k in ("kt", "tref", "fdc")]
        self.lut = C.c_void_p()
        T.check(T.lib.tops_lut_create(T.ptr(kw["kaz"], C.c_float), T.ptr(kw["krg"], C.c_float),
                                      C.byref(self.lut)), "lut")
        j = self.job = T.ResampleJob()
        j.slave, j.slave_pitch, j.out, j.out_pitch = (self.slave.data_ptr(), (W + pad) * 4,
                                                      self.out.data_ptr(), W * 8)
        j.kt, j.tref, j.fdc = (t.data_ptr() for t in self.par)
        for i in range(4):
            j.mbox[i], j.sbox[i] = int(kw["mbox"][i]), int(kw["sbox"][i])
        for i in range(6):
            j.cpm_az[i], j.cpm_rg[i] = kw["cpm_az"][i], kw["cpm_rg"][i]
        j.s_first_line, j.dt = kw["s_burst_idx"] * kw["lines_per_burst"], kw["dt"]
        j.out_row0, j.out_rows = (0, -1) if rows is None else rows

    def launch(self):
        import torch
        s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        self.T.check(self.T.lib.tops_resample_ex(self.lut, C.byref(self.job), 1, self.prec, s),
                     "tops_resample_ex")

    def result(self):
        import torch
        torch.cuda.synchronize()
        self.launch()
        torch.cuda.synchronize()
        a = self.out.cpu().numpy()
        return (a[..., 0] + 1j * a[..., 1])[:None if self.rows is None else self.rows[1]].astype(
            np.complex64)

    def close(self):
        self.T.lib.tops_lut_destroy(self.lut)


def _run(T, kw, prec, **opt):
    j = _Job(T, kw, prec, **opt)
    a = j.result()
    j.close()
    return a


# name: burst, additions to the range polynomial (coefficient: value)
CASES = {
    "two_keys_per_row": (dict(L=60, W=260, rg_tilt=0.06), {}),
    "many_keys_per_row": (dict(L=40, W=113, rg_tilt=0.5), {}),
    "down": (dict(L=130, W=225, rg_tilt=-0.03, x0=3, y0=7), {}),
    "runs_of_a_tile": (dict(L=130, W=224, rg_tilt=0.026), {}),
    "short_job": (dict(L=17, W=130, rg_tilt=0.02), {}),
    "some_columns": (dict(L=110, W=240), {4: 0.02}),
    "vertex_in_tables": (dict(L=100, W=230), {3: 4e-4}),
    "vertex": (dict(L=120, W=230, rg_tilt=0.01), {3: 0.02}),
    "with_entries": (dict(L=90, W=300, az_tilt=0.008, rg_tilt=0.05), {}),
    "with_line_skips": (dict(L=130, W=150, rg_tilt=0.05, az_scale=1.004), {}),
    "nine_entries": (dict(L=67, W=301, az_tilt=-0.0115), {}),
    "entry_table": (dict(L=200, W=301, az_tilt=0.0115, rg_tilt=0.004), {}),
    "too_many_entries": (dict(L=40, W=301, az_tilt=0.03, rg_tilt=0.03), {}),
}


@pytest.mark.parametrize("prec", ["split", "fp64"])
@pytest.mark.parametrize("name", CASES)
def test_resample_keys(T, O, name, prec):
    burst, rg = CASES[name]
    kw = _inputs(T, **burst)
    for i, v in rg.items():
        kw["cpm_rg"][i] += v
    ref, cnt = O.resample(**kw)
    gpu = _run(T, kw, prec)
    assert cnt[2] > 0
    assert rel_rms(gpu, ref) < TOL, rel_rms(gpu, ref)
    assert np.all(gpu[np.abs(ref) == 0] == 0)
    assert np.array_equal(_run(T, kw, prec, pad=1), gpu)
    L = gpu.shape[0]
    for r0, n in ((0, 1), (5, 7), (11, 3), (L - 9, 9)):
        assert np.array_equal(_run(T, kw, prec, rows=(r0, n)), gpu[r0:r0 + n]), (r0, n)


@pytest.mark.parametrize("prec", ["split", "fp64"])
def test_positions_spread_beyond_int(T, O, prec):
    """Range positions from -2^31 + 48 to 2.1e9 across a strip, one column of them
    inside the slave box, in rows of one and of several azimuth runs: the strip's
    bounds and that column's ring position overflow, but no tile offset or ring
    column follows them."""
    kw = _inputs(T, 60, 96, az_tilt=0.001)
    c = 48                                 # this column is at sample 40.3
    slope = (40.3 + 2147483600.5) / c
    kw["cpm_rg"][:] = [40.3 + (0.5 * 95 - c) * slope, 0, slope * 0.25 * 95, 0, 0, 0]
    ref, _ = O.resample(**kw)
    gpu = _run(T, kw, prec)
    assert np.abs(ref[:, c]).max() > 100 and not np.delete(ref, c, 1).any()
    assert rel_rms(gpu, ref) < TOL and np.all(gpu[np.abs(ref) == 0] == 0)


@pytest.mark.parametrize("prec", ["split", "fp64"])
def test_box_of_more_than_2_19_lines(T, O, prec):
    """The last lines of a slave box of 2^19 + 600 lines, in rows of four or five
    azimuth runs from its interior over its edge to the outside.  The burst's
    time starts near them and its ramp is the same in all columns: FP32 phases
    do not hold a ramp of 9 minutes."""
    kw = _inputs(T, 60, 20)
    n, W = 2 ** 19 + 600, 20
    rng = np.random.default_rng(7)
    slave = np.zeros((n, W, 2), np.int16)
    slave[-200:] = rng.normal(0, 700, (200, W, 2)).round()
    m0 = n - 55                            # the last 9 rows lie outside
    kw.update(slave=slave, mbox=np.array([0, W - 1, m0, m0 + 59], np.int32),
              sbox=np.array([0, W - 1, 0, n - 1], np.int32), s_burst_idx=1, lines_per_burst=n - 200)
    for k in ("kt", "tref", "fdc"):
        kw[k] = np.full(W, kw[k][0])
    kw["cpm_az"][:] = [m0 + 29.5 + 0.3, 0.25 * 59, 0.0005, 0.0, 0.0, 0.0]
    ref, cnt = O.resample(**kw)
    gpu = _run(T, kw, prec)
    assert cnt[2] > 0 and cnt[1] > 0 and not ref[-4:].any()
    assert rel_rms(gpu, ref) < TOL, rel_rms(gpu, ref)
    assert np.all(gpu[np.abs(ref) == 0] == 0)


def _time(jobs, reps=9):
    """Median time of each job (us), the jobs in turn."""
    import torch
    t = [[] for _ in jobs]
    for _ in range(reps):
        for i, j in enumerate(jobs):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(4):
                j.launch()
            b.record()
            torch.cuda.synchronize()
            t[i].append(a.elapsed_time(b) * 250.0)
    return [sorted(v)[len(v) // 2] for v in t]


def test_cost_of_dense_range_keys(T):
    """A key per row costs each pixel its key, 36 more products and its taps: about
    twice a pixel of a long run (measured 1.8).  Chunks that end where the run
    tables are full, 4 rows here, cost 4.6 times as much; the bound lies between."""
    jobs = [_Job(T, _inputs(T, 310, 12000, rg_tilt=t), "fp64") for t in (0.0, 0.2)]
    one, dense = _time(jobs)
    for j in jobs:
        j.close()
    print(f"one key {one:.0f} us, a key per row {dense:.0f} us")
    assert dense < 3.0 * one, (one, dense)


def test_cost_of_per_pixel_rows(T):
    """Rows of more azimuth runs than a strip takes are computed pixel by pixel, a
    thread per pixel and the rows end to end: 68 interior columns on 64 threads
    cost little more than 60 (twice as much when every row starts anew).  Columns
    0 to 3 and the last 8 are off the interior and cost next to nothing."""
    jobs = [_Job(T, _inputs(T, 1200, w, az_tilt=0.5), "split") for w in (72, 80)]
    a, b = _time(jobs)
    for j in jobs:
        j.close()
    print(f"60 interior columns {a:.0f} us, 68 {b:.0f} us")
    assert b < 1.5 * a, (a, b)
