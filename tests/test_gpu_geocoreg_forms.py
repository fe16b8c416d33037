"""The two forms of the geocoreg kernel (a pair of warps, or one warp, for the
master and slave solves of 32 DEM columns) at the edges of its tiles: a launch
of few tiles takes the pairs, one that carries a large job as well does not,
and a job's polynomials are the same bit for bit; and against the FP64 oracle.

Tolerance: both evaluate the same FP64 normal equations, whose right-hand sides
carry the rounding of seconds of day (7e-12 s, 4e-9 lines) per pixel; a window
on part of the burst extrapolates at most a few hundredfold, so 1e-5 px."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_stages import _poly_grid

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _job(T, torch, g, dem, r0, c0, out, status, pad):
    """A burst's job on a DEM window whose corner is (r0, c0) of its own."""
    d = torch.full((dem.shape[0], dem.shape[1] + pad), 5000.0, device="cuda")
    d[:, :dem.shape[1]] = torch.from_numpy(dem).cuda()
    j = T.GeoJob()
    j.dem, j.dem_pitch = d.data_ptr(), d.shape[1] * 4
    j.dem_lines, j.dem_pixels = dem.shape
    j.lat0, j.lon0 = g["lat0"] - r0 * g["dlat"], g["lon0"] + c0 * g["dlon"]
    j.dlat, j.dlon, j.nodata = g["dlat"], g["dlon"], -32768.0
    for k in ("xmin", "xmax", "ymin", "ymax"):
        setattr(j, k, g[k])
    for k in ("dt", "first_line_time", "slr_time", "range_spacing", "mid_time", "azi_init",
              "line_offset"):
        for w in (0, 1):
            getattr(j, k)[w] = g[k][w]
    for w in (0, 1):
        c = np.asarray(g["coefs"][w])
        j.ncoef[w] = c.shape[1]
        for a in range(3):
            for i in range(c.shape[1]):
                j.coef[w][a][i] = c[a, i]
    j.cpm_dev, j.status_dev = out.data_ptr(), status.data_ptr()
    return j, d


def _launch(T, torch, jobs):
    arr = (T.GeoJob * len(jobs))(*jobs)
    n = T.lib.tops_geocoreg_scratch_bytes(arr, len(jobs))
    scratch = torch.empty(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    T.check(T.lib.tops_geocoreg(arr, len(jobs), C.c_void_p(scratch.data_ptr()), n, None),
            "tops_geocoreg")
    torch.cuda.synchronize()


@pytest.mark.parametrize("h,w,pad", [(64, 64, 0), (33, 31, 1), (65, 33, 3), (32, 32, 0),
                                     (31, 97, 2), (111, 140, 0)])
def test_forms_agree_and_match_oracle(T, O, scene_small, h, w, pad):
    import torch
    g = scene_small.geo_args(0)
    r0, c0 = (0, 0) if h == 111 else (20, 20)
    dem = np.ascontiguousarray(g["dem"][r0:r0 + h, c0:c0 + w], np.float32)
    dem[3, 5:9] = -32768.0                      # samples without data break the rows' chains
    assert dem.shape == (h, w)
    out = torch.zeros(3, 12, dtype=torch.float64, device="cuda")
    status = torch.full((3,), -9, dtype=torch.int32, device="cuda")
    few, d0 = _job(T, torch, g, dem, r0, c0, out[0], status[0:], pad)
    again, d1 = _job(T, torch, g, dem, r0, c0, out[1], status[1:], pad)
    tall = np.tile(np.asarray(g["dem"], np.float32), (60, 1))      # over 200 tiles
    big, d2 = _job(T, torch, g, tall, 0, 0, out[2], status[2:], 0)
    _launch(T, torch, [few])
    _launch(T, torch, [again, big])
    assert status.cpu().tolist() == [0, 0, 0]
    a = out.cpu().numpy()
    assert np.array_equal(a[0], a[1])
    az, rg, st, nv = O.geocoreg(dem, g["lat0"] - r0 * g["dlat"], g["lon0"] + c0 * g["dlon"],
                                g["dlat"], g["dlon"], g["xmin"], g["xmax"], g["ymin"], g["ymax"],
                                g["dt"], g["first_line_time"], g["slr_time"], g["range_spacing"],
                                g["mid_time"], g["azi_init"], g["line_offset"], g["coefs"])
    assert st == 0 and nv > 100
    box = (g["ymin"], g["ymax"], g["xmin"], g["xmax"])
    for ours, ref in ((a[0, :6], az), (a[0, 6:], rg)):
        assert np.abs(_poly_grid(ours, *box) - _poly_grid(ref, *box)).max() < TOL
