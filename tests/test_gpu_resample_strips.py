"""The resample kernel at the edges of its tiles: strip widths, rows whose
azimuth key changes along the strip (several runs, a line crossing, descending
positions), range keys that change every few rows and odd box origins --
against the FP64 oracle, and row subsets bit for bit.

Tolerance: the kernel's sums and phases are FP32 on FP64 positions and phases;
each of the two sine / cosine pairs is good to 2^-21.4 = 3.6e-7 of the
amplitude and the 12 + 12 tap sums and the rotations round to about 24 x 2^-25
= 7e-7 at worst, so 2e-6 relative RMS bounds an exact implementation."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_rms

pytestmark = pytest.mark.gpu

TOL = 2e-6
DT, KT, FDC = 2.055e-3, 1735.0, 40.0


def _inputs(T, L, W, az_tilt=0.0, rg_tilt=0.0, az_off=0.41, rg_off=1.8, x0=0, y0=0, kt=KT,
            az_scale=1.0):
    rng = np.random.default_rng(L * 1000 + W)
    x = np.arange(x0 + W)
    kt = kt * (1.0 + 1e-6 * x)
    tref = 0.5 * L * DT + 1e-6 * x
    fdc = FDC + 2e-4 * x
    kaz, krg = T.lut(1.0 / DT, 327.0, 2 * 64.345e6)
    # positions over the master box, normalised coordinates in [-2, 2]
    cy, cx = y0 + 0.5 * (L - 1), x0 + 0.5 * (W - 1)
    az = np.array([cy + az_off, 0.25 * (L - 1) * az_scale, az_tilt / 4, 0.0, 0.0, 1e-4])
    rg = np.array([cx + rg_off, rg_tilt / 4, 0.25 * (W - 1), 0.0, 0.0, 0.0])
    slave = rng.normal(0, 700, (L, W, 2)).round().astype(np.int16)
    box = np.array([x0, x0 + W - 1, y0, y0 + L - 1], np.int32)
    return dict(slave=slave, cpm_az=az, cpm_rg=rg, az_shift=0.0, kaz=kaz, krg=krg, s_burst_idx=0,
                mbox=box, sbox=box, lines_per_burst=L, dt=DT, kt=kt, tref=tref, fdc=fdc)


def _run(T, kw, rows=None, pitch_pad=0):
    import torch
    L, W = kw["slave"].shape[:2]
    s = torch.zeros(L, W + pitch_pad, 2, dtype=torch.int16, device="cuda")
    s[:, :W] = torch.from_numpy(kw["slave"]).cuda()
    out = torch.full((L, W, 2), 7.0, device="cuda")
    par = [torch.from_numpy(np.ascontiguousarray(kw[k])).cuda() for k in ("kt", "tref", "fdc")]
    lut = C.c_void_p()
    T.check(T.lib.tops_lut_create(T.ptr(kw["kaz"], C.c_float), T.ptr(kw["krg"], C.c_float),
                                  C.byref(lut)), "lut")
    j = T.ResampleJob()
    j.slave, j.slave_pitch, j.out, j.out_pitch = s.data_ptr(), (W + pitch_pad) * 4, out.data_ptr(), W * 8
    j.kt, j.tref, j.fdc = (t.data_ptr() for t in par)
    for i in range(4):
        j.mbox[i], j.sbox[i] = int(kw["mbox"][i]), int(kw["sbox"][i])
    for i in range(6):
        j.cpm_az[i], j.cpm_rg[i] = kw["cpm_az"][i], kw["cpm_rg"][i]
    j.s_first_line, j.dt = kw["s_burst_idx"] * kw["lines_per_burst"], kw["dt"]
    j.out_row0, j.out_rows = (0, -1) if rows is None else rows
    torch.cuda.synchronize()
    T.check(T.lib.tops_resample_ex(lut, C.byref(j), 1, T.PREC_SPLIT, None), "tops_resample_ex")
    torch.cuda.synchronize()
    T.lib.tops_lut_destroy(lut)
    a = out.cpu().numpy()
    return (a[..., 0] + 1j * a[..., 1])[:None if rows is None else rows[1]].astype(np.complex64)


CASES = {
    "strip_minus_1": dict(L=40, W=111),
    "one_strip": dict(L=41, W=112),
    "strip_plus_1": dict(L=125, W=113),
    "strip_pair_plus_1": dict(L=121, W=225),
    "smallest": dict(L=16, W=16),
    "odd_origin": dict(L=61, W=263, x0=3, y0=7),
    "few_keys": dict(L=130, W=481, az_tilt=0.005),
    "many_keys": dict(L=67, W=301, az_tilt=-0.03),
    "too_many_keys": dict(L=33, W=250, az_tilt=0.2),
    "line_crossing": dict(L=130, W=300, az_tilt=0.004, az_off=0.9999),
    "line_crossing_down": dict(L=130, W=300, az_tilt=-0.004, az_off=1.0001),
    "crossing_and_skips": dict(L=250, W=260, az_tilt=0.01, az_scale=1.004, az_off=0.5),
    "repeated_lines": dict(L=250, W=260, az_scale=0.996, az_off=0.5),
    "range_runs": dict(L=250, W=260, rg_tilt=0.05),
    "range_run_per_row": dict(L=60, W=260, rg_tilt=0.06),
    "both": dict(L=120, W=500, az_tilt=0.02, rg_tilt=-0.04),
}


@pytest.mark.parametrize("name", CASES)
def test_resample_strips(T, O, name):
    kw = _inputs(T, **CASES[name])
    ref, cnt = O.resample(**kw)
    gpu = _run(T, kw)
    if CASES[name]["L"] > 16:
        assert cnt[2] > 0
    assert rel_rms(gpu, ref) < TOL, rel_rms(gpu, ref)
    assert np.all(gpu[np.abs(ref) == 0] == 0)
    # an odd pitch takes the 4-byte staging; subsets start inside halves
    assert np.array_equal(_run(T, kw, pitch_pad=1), gpu)
    L = gpu.shape[0]
    for r0, n in ((0, 1), (5, 7), (L - 9, 9)):
        assert np.array_equal(_run(T, kw, rows=(r0, n)), gpu[r0:r0 + n]), (r0, n)
