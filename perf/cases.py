"""Performance cases of the burst-pair path, through its public entry points.

Each case is one thing a user of this library has it do, at a size that the
repository's configurations, tests or benchmark use:

  kind "pair"      a device-resident plan (tops_pair_*): geocoreg, ReSlave, ESD,
                   ReSlaveESD and coherence of one sub-swath pair
  kind "host"      the same from page-locked host buffers to page-locked host
                   buffers (tops_pair_process), as the product run and the
                   server call it
  kind "batch"     three sub-swaths of different sizes in one batch (tops_batch_*)
  kind "resample"  the deramp + resample + reramp stage on one burst
  kind "coh"       the coherence stage on one burst
  kind "esd"       the ESD stage on the overlaps of a sub-swath
  kind "geo"       the geometric coregistration stage on one burst's DEM window

The geometry follows the synthetic generator's (two circular orbits, S1-IW
timing, steering and band widths); images are a band-limited speckle field
seen by both acquisitions, with each one's TOPS ramp, made on the GPU.
`exact` is the same chain in 64 bits with torch and numpy only.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "insar-on-sentinel-1-tops-data_b200"))

import ctypes as C  # noqa: E402

import topsb200 as T  # noqa: E402

DEV = "cuda"
C0 = 299792458.0
ELL_A, ELL_B = 6378137.0, 6356752.3142451794975639665996337
ELL_E2 = 1.0 - (ELL_B * ELL_B) / (ELL_A * ELL_A)
GM, WE = 3.986004418e14, 7.2921159e-5
T_MID = 50000.0
DT, RSR, ABW, WAVE, STEER = 2.055e-3, 64.345e6, 327.0, 0.05547, 1.59
DR = C0 / (2.0 * RSR)
H_MAX = 1500.0


# ------------------------------------------------------------------- the cases
def listed():
    return [
        # the headline workload: a full sub-swath pair, inputs and outputs in
        # HBM, replayed as a CUDA graph
        dict(name="subswath_pair", kind="pair", bursts=9, lines=1500, samples=21000, overlap=100,
             dem=3600, graph=True, win_rg=10, win_az=3, full=True, prec=0, comp=0),
        # a small product (the precision workload): two bursts of a narrow swath
        dict(name="small_pair", kind="pair", bursts=2, lines=1500, samples=4096, overlap=100,
             dem=512, graph=True, win_rg=10, win_az=3, full=True, prec=0, comp=0),
        # only ReSlaveESD and coherence wanted: ReSlave on the overlap bands,
        # FP64 deramp phases, compensated sums, the reference driver's window
        dict(name="bands_pair_ref_window", kind="pair", bursts=3, lines=1500, samples=6250,
             overlap=97, dem=1024, graph=True, win_rg=24, win_az=6, full=False, prec=1, comp=1),
        # the smallest pair of the tests, launched eagerly: latency
        dict(name="tiny_pair", kind="pair", bursts=2, lines=300, samples=512, overlap=30, dem=192,
             graph=False, win_rg=10, win_az=3, full=True, prec=0, comp=0),
        # three sub-swaths of a product, uneven lines and samples, one batch
        dict(name="batch_uneven", kind="batch", bursts=2, overlap=100, dem=1200, shape=0),
        # host to host: what the product run does per sub-swath (here the
        # small product), bounded by the copies
        dict(name="host_pair", kind="host", bursts=2, lines=1500, samples=4096, overlap=100,
             dem=512, full=True),
        # one full-width burst
        dict(name="resample_burst", kind="resample", lines=1500, samples=21000, prec=0,
             az_tilt=0.0, rg_tilt=0.0, shift=0.0),
        # one burst of a pair whose orbits cross: the azimuth offset changes
        # by 0.05 lines across the swath and the range offset by 0.05 samples
        # along the burst; an odd width, a shift, FP64 deramp phases
        dict(name="resample_crossing", kind="resample", lines=1539, samples=10867, prec=1,
             az_tilt=0.05, rg_tilt=0.05, shift=0.0371),
        # coherence of a full-width burst, the configuration's 10 x 3 window
        dict(name="coh_burst", kind="coh", lines=1500, samples=21000, win_rg=10, win_az=3, pad=0),
        # another window, on rows that are no multiple of 16 bytes
        dict(name="coh_odd_window", kind="coh", lines=1523, samples=8193, win_rg=5, win_az=5,
             pad=0),
        # the 8 overlaps of the headline sub-swath
        dict(name="esd_overlaps", kind="esd", overlaps=8, lines=100, samples=21000, win_rg=10,
             win_az=3),
        # the DEM window of one full-width burst
        dict(name="geocoreg_burst", kind="geo", lines=1500, samples=21000, dem=1800),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair", "pair", "resample", "resample", "coh", "coh", "esd", "geo", "host"])
    lines = rng.randint(300, 1560)
    if kind in ("pair", "host"):
        c = dict(kind=kind, bursts=rng.randint(2, 4), lines=lines, samples=_logint(rng, 512, 21000),
                 overlap=max(8, int(lines * rng.uniform(0.05, 0.09))), dem=_logint(rng, 192, 2000),
                 full=rng.random() < 0.75)
        if kind == "host":
            c["bursts"], c["samples"], c["full"] = 2, _logint(rng, 512, 6000), True
            return c
        w = rng.choice([(10, 3), (10, 3), (24, 6), (5, 5)])
        c.update(graph=rng.random() < 0.7, win_rg=w[0], win_az=w[1], prec=rng.randint(0, 1),
                 comp=rng.randint(0, 1))
        return c
    if kind == "resample":
        return dict(kind=kind, lines=lines, samples=_logint(rng, 300, 25300),
                    prec=rng.randint(0, 1), az_tilt=rng.choice([0.0, rng.uniform(-0.08, 0.08)]),
                    rg_tilt=rng.choice([0.0, rng.uniform(-0.08, 0.08)]),
                    shift=rng.uniform(-0.05, 0.05))
    if kind == "coh":
        w = rng.choice([(10, 3), (24, 6), (10, 6), (24, 3), (5, 5), (rng.randint(2, 30), rng.randint(1, 9))])
        return dict(kind=kind, lines=lines, samples=_logint(rng, 200, 25300), win_rg=w[0],
                    win_az=w[1], pad=rng.choice([0, 0, 1, 3]))
    if kind == "esd":
        w = rng.choice([(10, 3), (24, 6), (5, 5)])
        return dict(kind=kind, overlaps=rng.randint(1, 8), lines=rng.randint(20, 150),
                    samples=_logint(rng, 500, 25300), win_rg=w[0], win_az=w[1])
    return dict(kind=kind, lines=lines, samples=_logint(rng, 2000, 25300), dem=_logint(rng, 300, 2400))


BATCH_SHAPES = [[(1523, 25073), (1539, 21835), (1544, 25322)]]


def work(case):
    k = case["kind"]
    fir, coh_f = 2 * 2 * 24 + 40, 70      # flops per pixel: the separable taps and both phases; coherence
    if k in ("pair", "host", "batch"):
        shapes = BATCH_SHAPES[case["shape"]] if k == "batch" else [(case["lines"], case["samples"])]
        px = sum(a * b for a, b in shapes) * case["bursts"]
        full = case.get("full", True)
        return {"bytes": px * (8 + 12 + (8 if full else 0)) + 4 * case["dem"] ** 2 * len(shapes),
                "flops": px * (fir * (2 if full else 1) + coh_f)}
    px = case["lines"] * case["samples"]
    if k == "resample":
        return {"bytes": 12 * px, "flops": fir * px}
    if k == "coh":
        return {"bytes": 16 * px, "flops": coh_f * px}
    if k == "esd":
        return {"bytes": 24 * px * case["overlaps"], "flops": 2 * coh_f * px * case["overlaps"]}
    dem = _geo_case(case)["dem_shape"]
    return {"bytes": 4 * dem[0] * dem[1], "flops": 390 * dem[0] * dem[1]}


# -------------------------------------------------------------------- geometry
class Orbit:
    """Circular inertial orbit in the Earth-fixed frame (numpy, vectorised in t)."""

    def __init__(self, shift=0.0, bperp=0.0, bpar=0.0, inc=math.radians(35.0)):
        self.Rs = ELL_A + 693000.0
        self.n = math.sqrt(GM / self.Rs ** 3)
        self.incl, self.Om = math.radians(98.18), 0.3
        self.u0 = math.asin(math.sin(math.radians(38.0)) / math.sin(self.incl))
        re = 6371000.0
        look = math.asin(re / self.Rs * math.sin(inc))
        self.r_mid = self.Rs * math.cos(look) - math.sqrt(re * re - (self.Rs * math.sin(look)) ** 2)
        self.shift = shift
        self.b_out = -(bpar * math.sin(look) + bperp * math.cos(look))
        self.b_rad = -bpar * math.cos(look) + bperp * math.sin(look)

    def pos(self, t):
        t = np.asarray(t, np.float64)
        u = self.u0 + self.n * (t - T_MID + self.shift)
        e1 = np.array([math.cos(self.Om), math.sin(self.Om), 0.0])
        e2 = np.array([-math.sin(self.Om) * math.cos(self.incl),
                       math.cos(self.Om) * math.cos(self.incl), math.sin(self.incl)])
        nrm = np.cross(e1, e2)
        q = ((self.Rs + self.b_rad) * (np.cos(u)[..., None] * e1 + np.sin(u)[..., None] * e2) +
             self.b_out * nrm)
        th = WE * (t - T_MID)
        c, s = np.cos(th), np.sin(th)
        return np.stack([c * q[..., 0] + s * q[..., 1], -s * q[..., 0] + c * q[..., 1], q[..., 2]], -1)

    def pva(self, t):
        h = 0.01
        r, p, m = self.pos(t), self.pos(np.asarray(t) + h), self.pos(np.asarray(t) - h)
        return r, (p - m) / (2 * h), (p - 2 * r + m) / (h * h)

    def zero_doppler(self, X, t):
        t = np.array(t, np.float64)
        for _ in range(10):
            r, v, a = self.pva(t)
            d = X - r
            t = t - (v * d).sum(-1) / ((a * d).sum(-1) - (v * v).sum(-1))
        return t, np.linalg.norm(X - self.pos(t), axis=-1)


def xyz2llh(X):
    lon = np.arctan2(X[..., 1], X[..., 0])
    p = np.hypot(X[..., 0], X[..., 1])
    lat = np.arctan2(X[..., 2], p * (1.0 - ELL_E2))
    for _ in range(6):
        N = ELL_A / np.sqrt(1.0 - ELL_E2 * np.sin(lat) ** 2)
        h = p / np.cos(lat) - N
        lat = np.arctan2(X[..., 2], p * (1.0 - ELL_E2 * N / (N + h)))
    return lat, lon, p / np.cos(lat) - ELL_A / np.sqrt(1.0 - ELL_E2 * np.sin(lat) ** 2)


def geocode(orb, t, R, h0):
    """Ground points (right looking) at azimuth times t, slant ranges R, height h0."""
    r, v, _ = orb.pva(t)
    vh = v / np.linalg.norm(v, axis=-1, keepdims=True)
    rs = np.linalg.norm(r, axis=-1, keepdims=True)
    e1 = -r / rs
    e1 = e1 - (e1 * vh).sum(-1, keepdims=True) * vh
    e1 /= np.linalg.norm(e1, axis=-1, keepdims=True)
    e2 = np.cross(vh, e1)
    e2 = np.where((np.cross(v, r) * e2).sum(-1, keepdims=True) < 0, -e2, e2)
    re = 6371000.0
    ca = (rs[..., 0] ** 2 + R * R - re * re) / (2 * rs[..., 0] * R)
    a0 = np.arccos(np.clip(ca, -1, 1))
    lo, hi = a0 - 0.05, a0 + 0.05
    point = lambda al: r + R[..., None] * (np.cos(al)[..., None] * e1 + np.sin(al)[..., None] * e2)
    for _ in range(50):
        mid = 0.5 * (lo + hi)
        up = xyz2llh(point(mid))[2] - h0 > 0
        lo, hi = np.where(up, lo, mid), np.where(up, mid, hi)
    return point(0.5 * (lo + hi))


def make_geometry(nb, L, W, ov, dem):
    """Timing, orbits and the DEM grid of a sub-swath pair (plain numbers)."""
    M, S = Orbit(), Orbit(-0.3 * DT, 40.0, -4.0)
    tcyc = (L - ov - 1) * DT - 1e-6 * DT
    t0 = T_MID - 0.5 * ((nb - 1) * tcyc + (L - 1) * DT)
    first = t0 + tcyc * np.arange(nb)
    g = dict(nb=nb, L=L, W=W, ov=ov, first=first, last=first + (L - 1) * DT,
             slr=(M.r_mid - 0.5 * W * DR) / C0, orb=(M, S),
             sv_t=T_MID + 10.0 * (np.arange(17) - 8))
    g["sv"] = [o.pos(g["sv_t"]) for o in (M, S)]
    t0w = 2 * (g["slr"] + 0.5 * W * DR / C0)
    g["dc"], g["fm"] = [], []
    for w in (0, 1):
        kk = np.arange(nb + 2) - 1 + 0.37 * w
        tc = t0 + (np.arange(nb + 2) - 1) * tcyc + 0.5 * (L - 1) * DT
        g["dc"].append([(tc[k], t0w, 25.0 + 3.0 * math.sin(0.7 * kk[k]), 3.0e4, 0.0) for k in range(nb + 2)])
        g["fm"].append([(tc[k], t0w, -2300.0 + 1.5 * kk[k], 4.3e5, -7.6e7) for k in range(nb + 2)])
    # footprint of each burst: 3 x 3 image points at the lowest and highest terrain
    a, c = np.meshgrid([0.0, 0.5, 1.0], [0.0, 0.5, 1.0], indexing="ij")
    boxes = []
    for b in range(nb):
        la, lo = [], []
        for h in (0.0, H_MAX):
            X = geocode(M, (first[b] + a * (L - 1) * DT).ravel(),
                        (g["slr"] * C0 + c * (W - 1) * DR).ravel(), h)
            q = xyz2llh(X)
            la.append(np.degrees(q[0]))
            lo.append(np.degrees(q[1]))
        boxes.append((np.min(la), np.max(la), np.min(lo), np.max(lo)))
    bx = np.array(boxes)
    lamin, lamax, lomin, lomax = bx[:, 0].min(), bx[:, 1].max(), bx[:, 2].min(), bx[:, 3].max()
    dlat = max(1 / 3600, (lamax - lamin) / (dem - 80))
    dlon = max(1 / 3600, (lomax - lomin) / (dem - 80))
    g["dem"] = dem
    g["dlat"], g["dlon"] = dlat, dlon
    g["lat0"] = 0.5 * (lamax + lamin) + 0.5 * (dem - 1) * dlat
    g["lon0"] = 0.5 * (lomax + lomin) - 0.5 * (dem - 1) * dlon
    g["win"] = []
    for la0, la1, lo0, lo1 in boxes:
        r0 = max(0, math.floor((g["lat0"] - la1) / dlat - 24))
        c0 = max(0, math.floor((lo0 - g["lon0"]) / dlon - 24))
        r1 = min(dem - 1, math.ceil((g["lat0"] - la0) / dlat + 24))
        c1 = min(dem - 1, math.ceil((lo1 - g["lon0"]) / dlon + 24))
        g["win"].append((r0, c0, r1 - r0 + 1, c1 - c0 + 1))
    return g


def orbit_fit(g, w):
    """Degree-5 polynomials of the normalised time (t - t_mid) / 10: [3][6], by
    Cholesky's method on the normal equations.  The sums run in index order:
    offsets hardly change across a burst of parallel orbits, so where a LUT
    bin changes depends on the last digits of these coefficients."""
    A = [[float(v) ** j for j in range(6)] for v in (g["sv_t"] - g["sv_t"][8]) / 10.0]
    dot = lambda u, v: sum(a * b for a, b in zip(u, v))
    cols = list(zip(*A))
    n = [[dot(cols[i], cols[j]) for j in range(6)] for i in range(6)]
    for i in range(6):
        for j in range(i, 6):
            s = n[i][j]
            for k in range(i - 1, -1, -1):
                s -= n[i][k] * n[j][k]
            n[j][i] = math.sqrt(s) if i == j else s / n[i][i]
    out = []
    for axis in range(3):
        b = [dot(c, [float(v) for v in g["sv"][w][:, axis]]) for c in cols]
        for i in range(6):
            for j in range(i - 1, -1, -1):
                b[i] -= n[i][j] * b[j]
            b[i] /= n[i][i]
        for i in range(5, -1, -1):
            for j in range(i + 1, 6):
                b[i] -= n[j][i] * b[j]
            b[i] /= n[i][i]
        out.append(b)
    return np.array(out)


def deramp_rows(g, w):
    """kt, tref, fdc [nb][W] of image w (azimuth-steered TOPS ramp)."""
    x = np.arange(g["W"])
    slrt = 2 * (g["slr"] + x * DR / C0)
    dc = np.stack([p[2] + p[3] * (slrt - p[1]) + p[4] * (slrt - p[1]) ** 2 for p in g["dc"][w][:g["nb"]]])
    fm = np.stack([p[2] + p[3] * (slrt - p[1]) + p[4] * (slrt - p[1]) ** 2 for p in g["fm"][w][:g["nb"]]])
    tref = g["L"] * DT / 2 + dc[:, :1] / fm[:, :1] - dc / fm
    c = orbit_fit(g, w)
    tn = (0.5 * (g["first"][0] + g["last"][-1]) - g["sv_t"][8]) / 10.0
    v = sum(i * c[:, i] * tn ** (i - 1) for i in range(1, 6)) / 10.0
    krot = 2 * np.linalg.norm(v) * math.radians(STEER) / WAVE
    return fm * krot / (fm - krot), tref, dc


def lut_tables():
    """Raised-cosine windowed 12-point sinc tables [2048][12], as float32."""
    out = []
    for v in (1.0 - ABW * DT, 1.0 - ABW / RSR):
        x = 1.0 - 6 + np.arange(12)[None, :] - np.arange(2048)[:, None] / 2047
        w = np.sinc(x) * np.where(np.abs(x) < 6, 1.0, np.where(np.abs(x) == 6, 0.5, 0.0))
        w = w * np.cos(v * math.pi * x) / (1.0 - (2.0 * v * x) ** 2)
        out.append((w.astype(np.float32).astype(np.float64) / w.sum(1, keepdims=True)).astype(np.float32))
    return out


def offset_poly(g, b, h=0.5 * H_MAX):
    """Offset polynomials (azimuth, range) of burst b for flat terrain at height h:
    slave position over the master grid, in the library's normalisation."""
    L, W = g["L"], g["W"]
    l, x = np.meshgrid(np.linspace(0, L - 1, 9), np.linspace(0, W - 1, 17), indexing="ij")
    X = geocode(g["orb"][0], g["first"][b] + l.ravel() * DT, g["slr"] * C0 + x.ravel() * DR, h)
    t, R = g["orb"][1].zero_doppler(X, g["first"][b] + l.ravel() * DT)
    sl, sx = b * L + (t - g["first"][b]) / DT, (R - g["slr"] * C0) / DR
    y0, y1 = b * L, (b + 1) * L - 1
    Lh = (l.ravel() + y0 - 0.5 * (y0 + y1)) / (0.25 * (y1 - y0))
    Ph = (x.ravel() - 0.5 * (W - 1)) / (0.25 * (W - 1))
    A = np.stack([np.ones_like(Lh), Lh, Ph, Lh * Lh, Lh * Ph, Ph * Ph], 1)
    return np.linalg.lstsq(A, np.stack([sl, sx], 1), rcond=None)[0].T.copy()


# --------------------------------------------------------------- inputs on GPU
def _rand(seed, *shape):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) & 0x7FFFFFFF)
    return torch.randn(*shape, generator=gen, device=DEV)


def make_dem(n, seed):
    """Rough terrain of 0..1500 m: octaves of bicubic noise."""
    z = torch.zeros(1, 1, n, n, device=DEV)
    for k in range(9):
        m = min(n, 4 << k)
        z += 0.57 ** k * torch.nn.functional.interpolate(_rand(seed * 31 + k, 1, 1, m, m), (n, n),
                                                         mode="bicubic", align_corners=True)
        if m == n:
            break
    z = z[0, 0]
    return ((z - z.min()) * (H_MAX / (z.max() - z.min()))).contiguous()


def make_field(rows, cols, seed):
    """Band-limited circular speckle [2][rows][cols]."""
    z = _rand(seed, 2, rows, cols)
    for ax, bw in ((1, ABW * DT), (2, 56.5e6 / RSR)):
        k = np.arange(-7, 8)
        h = np.sinc(bw * k) * np.hamming(15)
        h /= math.sqrt((h * h).sum())
        n = z.shape[ax]
        acc = torch.zeros_like(z)
        for o, w in zip(k, h):
            o, w = int(o), float(w)
            acc.narrow(ax, max(0, -o), n - abs(o)).add_(z.narrow(ax, max(0, o), n - abs(o)), alpha=w)
        z = acc
    return z


def _ramp(rows, l, x):
    """Deramp phase at burst lines l and columns x (rows = kt, tref, fdc of one
    burst, float64 on the GPU), reduced to [-pi, pi] as float32."""
    W = rows[0].numel()
    x = x.clamp(0, W - 1)
    x0 = x.floor().clamp(max=max(W - 2, 0)).long()
    f = x - x0
    kt, tr, fd = ((1 - f) * r[x0] + f * r[(x0 + 1).clamp(max=W - 1)] for r in rows)
    ta = l * DT
    ph = -math.pi * kt * (ta - tr) ** 2 - 2 * math.pi * fd * ta
    return (ph - 2 * math.pi * torch.round(ph / (2 * math.pi))).float()


def _cint(re, im, ph):
    c, s = torch.cos(ph), torch.sin(ph)
    z = torch.stack([re * c - im * s, re * s + im * c], -1)
    return (z * 707.0).round().clamp(-32768, 32767).to(torch.int16)


def make_slcs(g, seed, put, shift=0.02):
    """Calls put(w, b, int16 [L][W][2]) for both images of every burst: the same
    field through both geometries, misregistered by `shift` lines."""
    nb, L, W, ov, pad = g["nb"], g["L"], g["W"], g["ov"], 24
    GL = (nb - 1) * (L - ov - 1) + L + 2 * pad
    z = make_field(GL, W + 2 * pad, seed * 7 + 1)
    km = [[torch.from_numpy(r[b]).to(DEV) for r in deramp_rows(g, 0)] for b in range(nb)]
    col = torch.arange(W, device=DEV, dtype=torch.float64)[None, :]
    step = max(16, min(L, 6_000_000 // W))
    for b in range(nb):
        az, rg = offset_poly(g, b)
        m = torch.empty(L, W, 2, dtype=torch.int16, device=DEV)
        s = torch.empty(L, W, 2, dtype=torch.int16, device=DEV)
        for r0 in range(0, L, step):
            r1 = min(L, r0 + step)
            lin = torch.arange(r0, r1, device=DEV, dtype=torch.float64)[:, None]
            q = pad + b * (L - ov - 1)
            zr = z[:, q + r0:q + r1, pad:pad + W]
            m[r0:r1] = _cint(zr[0], zr[1], -_ramp(km[b], lin, col.expand(r1 - r0, W)))
            Lh = (lin - 0.5 * (L - 1)) / (0.25 * (L - 1))
            Ph = (col - 0.5 * (W - 1)) / (0.25 * (W - 1))
            p = lambda c: c[0] + c[1] * Lh + c[2] * Ph + c[3] * Lh * Lh + c[4] * Lh * Ph + c[5] * Ph * Ph
            v0 = lin - (p(az) - b * L - lin) + shift        # master position of the slave sample
            dx = p(rg) - col
            v1 = col - dx
            gx = (2 * (v1 + pad) / (W + 2 * pad - 1) - 1).float()
            gy = (2 * (v0 + q) / (GL - 1) - 1).float()
            zz = torch.nn.functional.grid_sample(z[None], torch.stack([gx, gy], -1)[None], mode="bicubic",
                                                 padding_mode="border", align_corners=True)[0]
            topo = -4 * math.pi / WAVE * DR * dx
            topo = (topo - 2 * math.pi * torch.round(topo / (2 * math.pi))).float()
            s[r0:r1] = _cint(zz[0], zz[1], topo - _ramp(km[b], v0, v1))
        put(0, b, m)
        put(1, b, s)


def swath_info(g, w):
    i = T.SwathInfo()
    nb = g["nb"]
    i.n_bursts, i.lines_per_burst, i.samples_per_burst, i.first_valid_pixel = nb, g["L"], g["W"], 0
    i.dt, i.prf, i.slr_time, i.range_spacing = DT, 1.0 / DT, g["slr"], DR
    i.wavelength, i.rsr, i.az_bandwidth, i.steering_rate_deg = WAVE, RSR, ABW, STEER
    i.first_line_time, i.last_line_time = g["first"][0], g["last"][-1]
    for b in range(nb):
        i.burst_first_line_time[b], i.burst_last_line_time[b] = g["first"][b], g["last"][b]
    i.n_dc = i.n_fm = nb + 2
    for k in range(nb + 2):
        i.dc_list[k], i.fm_list[k] = T.Poly(*g["dc"][w][k]), T.Poly(*g["fm"][w][k])
    i.n_sv = 17
    for k in range(17):
        i.sv_t[k] = g["sv_t"][k]
        i.sv_x[k], i.sv_y[k], i.sv_z[k] = g["sv"][w][k]
    return i


class _DeviceArray:
    """A plan's device buffer for torch; keeps the plan alive."""

    def __init__(self, owner, ptr, shape, strides, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, strides=strides,
                                             typestr=typestr, version=3)


def _view(owner, ptr, rows, cols, pitch, comps, typestr):
    size = int(typestr[-1])
    shape = (rows, cols, comps) if comps > 1 else (rows, cols)
    strides = (pitch, comps * size, size) if comps > 1 else (pitch, size)
    return torch.as_tensor(_DeviceArray(owner, ptr, shape, strides, typestr), device=DEV)


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _geom(case, shape=None):
    L, W = shape or (case["lines"], case["samples"])
    return make_geometry(case["bursts"], L, W, case["overlap"], case["dem"])


def _plan(g, opts, seed, host=None):
    """A plan with its DEM and (unless `host`) its SLCs in place."""
    P = T.Pair(swath_info(g, 0), swath_info(g, 1), (g["dem"], g["dem"]), opts)
    win = (T.DemWindow * g["nb"])(*[T.DemWindow(*w) for w in g["win"]])
    P.set_dem(make_dem(g["dem"], seed).cpu().numpy(), g["lat0"], g["lon0"], g["dlat"], g["dlon"], win,
              _stream())
    B, n = P.buffers(), g["nb"] * g["L"]
    if host is None:
        img = [_view(P, p, n, g["W"], B.slc_pitch, 2, "<i2") for p in (B.master, B.slave)]
        put = lambda w, b, a: img[w][b * g["L"]:(b + 1) * g["L"]].copy_(a)
    else:
        put = lambda w, b, a: host[w][b * g["L"]:(b + 1) * g["L"]].copy_(a)
    make_slcs(g, seed, put)
    out = {"reslave_esd": _view(P, B.reslave_esd, n, g["W"], B.cplx_pitch, 2, "<f4"),
           "coh": _view(P, B.coh, n, g["W"], B.coh_pitch, 1, "<f4")}
    if P.opts.reslave_full:
        out["reslave"] = _view(P, B.reslave, n, g["W"], B.cplx_pitch, 2, "<f4")
    return P, out


def _pair_opts(case):
    return T.pair_opts(win_rg=case.get("win_rg", 10), win_az=case.get("win_az", 3),
                       reslave_full=int(case.get("full", True)), precision=case.get("prec", 0),
                       compensated=case.get("comp", 0))


def _resample_inputs(case, seed):
    L, W = case["lines"], case["samples"]
    g = make_geometry(1, L, W, 10, 192)
    az, rg = offset_poly(g, 0)
    # crossing orbits: the offsets change linearly across / along the burst
    # (the normalised coordinates run over [-2, 2])
    az[2] += case["az_tilt"] / 4
    rg[1] += case["rg_tilt"] / 4
    z = make_field(L, W, seed * 7 + 1)
    rows = [torch.from_numpy(r[0]).to(DEV) for r in deramp_rows(g, 1)]
    s = torch.empty(L, W, 2, dtype=torch.int16, device=DEV)
    col = torch.arange(W, device=DEV, dtype=torch.float64)[None, :]
    for r0 in range(0, L, 256):
        r1 = min(L, r0 + 256)
        lin = torch.arange(r0, r1, device=DEV, dtype=torch.float64)[:, None]
        s[r0:r1] = _cint(z[0, r0:r1], z[1, r0:r1], -_ramp(rows, lin, col.expand(r1 - r0, W)))
    return s, rows, az, rg


def _coh_inputs(L, W, seed):
    """Master CInt16 and resampled slave complex64 of a pair (coherence 0.4 to
    1 across the image), zero outside the slave's coverage."""
    z, n = make_field(L, W, seed * 7 + 1), make_field(L, W, seed * 7 + 2)
    g = torch.linspace(0.4, 1.0, W, device=DEV)[None, None, :]
    s = g * z + torch.sqrt(1 - g * g) * n
    col = torch.arange(W, device=DEV)[None, :] * 0.01
    lin = torch.arange(L, device=DEV)[:, None] * 0.003
    m = _cint(z[0], z[1], col + lin)
    s = (s.permute(1, 2, 0) * 707.0).contiguous()
    s[:, :2] = 0
    s[-1:] = 0
    return m, s


def _esd_inputs(case, seed):
    """Master and slave bands (forward, backward) of the overlaps, stacked, with
    a misregistration of 0.03 lines in the double difference."""
    n, L, W = case["overlaps"], case["lines"], case["samples"]
    out = []
    for k, ph in ((0, 0.0), (1, ESD_SEP * 2 * math.pi * DT * 0.03)):
        m, s = _coh_inputs(n * L, W, seed * 3 + k)
        c, q = math.cos(ph), math.sin(ph)
        out += [m, torch.stack([s[..., 0] * c - s[..., 1] * q, s[..., 0] * q + s[..., 1] * c], -1).contiguous()]
    return out


ESD_SEP = 4000.0     # spectral separation of the overlaps, Hz


def _geo_case(case):
    g = make_geometry(1, case["lines"], case["samples"], 10, case["dem"])
    g["dem_shape"] = g["win"][0][2:]
    return g


# ------------------------------------------------------------------ the passes
def prepare(case, seed):
    k = case["kind"]
    st = {"case": case}
    if k == "pair":
        st["plan"], st["out"] = _plan(_geom(case), _pair_opts(case), seed)
    elif k == "host":
        g = _geom(case)
        n = g["nb"] * g["L"]
        st["slc"] = [torch.empty(n, g["W"], 2, dtype=torch.int16, pin_memory=True) for _ in (0, 1)]
        st["plan"], _ = _plan(g, _pair_opts(case), seed, host=st["slc"])
        st["keep"] = [torch.empty(n, g["W"], 2, pin_memory=True) for _ in (0, 1)] + \
                     [torch.empty(n, g["W"], pin_memory=True)]
        st["np"] = [a.numpy() for a in st["slc"]]
        st["out"] = dict(reslave=st["keep"][0].numpy(), reslave_esd=st["keep"][1].numpy(),
                         coh=st["keep"][2].numpy())
    elif k == "batch":
        st["plans"], st["out"] = [], []
        for i, shape in enumerate(BATCH_SHAPES[case["shape"]]):
            P, out = _plan(_geom(case, shape), T.pair_opts(), seed * 5 + i)
            st["plans"].append(P)
            st["out"].append(out)
        st["batch"] = T.Batch(st["plans"])
    elif k == "resample":
        L, W = case["lines"], case["samples"]
        s, rows, az, rg = _resample_inputs(case, seed)
        st["in"] = [s] + rows
        st["out"] = torch.empty(L, W, 2, device=DEV)
        kaz, krg = T.lut(1.0 / DT, ABW, 2 * RSR)
        st["lut"] = C.c_void_p()
        T.check(T.lib.tops_lut_create(T.ptr(kaz, C.c_float), T.ptr(krg, C.c_float), C.byref(st["lut"])),
                "tops_lut_create")
        st["guard"] = _LutGuard(st["lut"])
        j = T.ResampleJob()
        j.slave, j.slave_pitch, j.out, j.out_pitch = s.data_ptr(), W * 4, st["out"].data_ptr(), W * 8
        j.kt, j.tref, j.fdc = (r.data_ptr() for r in rows)
        for i, v in enumerate((0, W - 1, 0, L - 1)):
            j.mbox[i] = j.sbox[i] = v
        for i in range(6):
            j.cpm_az[i], j.cpm_rg[i] = az[i], rg[i]
        j.az_shift, j.s_first_line, j.dt, j.out_row0, j.out_rows = case["shift"], 0, DT, 0, -1
        st["job"] = j
    elif k == "coh":
        L, W, pitch = case["lines"], case["samples"], case["samples"] + case["pad"]
        m, s = _coh_inputs(L, W, seed)
        mp = torch.zeros(L, pitch, 2, dtype=torch.int16, device=DEV)
        sp = torch.zeros(L, pitch, 2, device=DEV)
        mp[:, :W], sp[:, :W] = m, s
        out = torch.empty(L, W, device=DEV)
        st["in"], st["out"] = [mp, sp], out
        st["job"] = T.CohJob(master=mp.data_ptr(), master_pitch=pitch * 4, slave=sp.data_ptr(),
                             slave_pitch=pitch * 8, coh=out.data_ptr(), coh_pitch=W * 4, lines=L, pixels=W)
    elif k == "esd":
        n, L, W = case["overlaps"], case["lines"], case["samples"]
        mF, sF, mB, sB = st["in"] = _esd_inputs(case, seed)
        st["ovs"] = (T.EsdOverlap * n)(*[
            T.EsdOverlap(mF[i * L].data_ptr(), mB[i * L].data_ptr(), W * 4, sF[i * L].data_ptr(),
                         sB[i * L].data_ptr(), W * 8, L, W, ESD_SEP, DT) for i in range(n)])
        st["bytes"] = T.lib.tops_esd_scratch_bytes(st["ovs"], n)
        st["scratch"] = torch.empty(st["bytes"], dtype=torch.uint8, device=DEV)
        st["out"] = torch.zeros(n, dtype=torch.float64, device=DEV)
    else:
        g = _geo_case(case)
        dem = make_dem(g["dem"], seed)
        r0, c0, nr, nc = g["win"][0]
        st["dem"], st["out"] = dem, torch.zeros(12, dtype=torch.float64, device=DEV)
        st["status"] = torch.zeros(1, dtype=torch.int32, device=DEV)
        j = T.GeoJob()
        j.dem, j.dem_pitch, j.dem_lines, j.dem_pixels = dem[r0, c0:].data_ptr(), g["dem"] * 4, nr, nc
        j.lat0, j.lon0 = g["lat0"] - r0 * g["dlat"], g["lon0"] + c0 * g["dlon"]
        j.dlat, j.dlon, j.nodata = g["dlat"], g["dlon"], -32768.0
        j.xmin, j.xmax, j.ymin, j.ymax = 0, case["samples"] - 1, 0, case["lines"] - 1
        for w in (0, 1):
            j.dt[w], j.first_line_time[w], j.slr_time[w], j.range_spacing[w] = DT, g["first"][0], g["slr"], DR
            j.mid_time[w], j.azi_init[w] = g["sv_t"][8], 0.5 * (g["first"][0] + g["last"][0])
            j.line_offset[w], j.ncoef[w] = 0, 6
            c = orbit_fit(g, w)
            for a in range(3):
                for i in range(6):
                    j.coef[w][a][i] = c[a, i]
        j.cpm_dev, j.status_dev = st["out"].data_ptr(), st["status"].data_ptr()
        st["job"] = j
        st["bytes"] = T.lib.tops_geocoreg_scratch_bytes(C.byref(j), 1)
        st["scratch"] = torch.empty(st["bytes"], dtype=torch.uint8, device=DEV)
    return st


class _LutGuard:
    def __init__(self, lut):
        self.lut = lut

    def __del__(self):
        torch.cuda.synchronize()
        T.lib.tops_lut_destroy(self.lut)


def run(st):
    """One pass.  A plan's outputs are the rasters a product run writes; the
    offsets and shifts it computes on the way are their inputs and are
    outputs of the "geo" and "esd" cases."""
    case = st["case"]
    k = case["kind"]
    s = _stream()
    if k == "pair":
        st["plan"].run(s, graph=case["graph"])
    elif k == "host":
        st["plan"].process(st["np"][0], st["np"][1], out=st["out"], stream=s)
        T.check(T.lib.tops_stream_synchronize(C.c_void_p(s)), "tops_stream_synchronize")
    elif k == "batch":
        st["batch"].run(s, graph=True)
    elif k == "resample":
        T.check(T.lib.tops_resample_ex(st["lut"], C.byref(st["job"]), 1, case["prec"], C.c_void_p(s)),
                "tops_resample_ex")
    elif k == "coh":
        T.check(T.lib.tops_coherence(C.byref(st["job"]), 1, case["win_rg"], case["win_az"], C.c_void_p(s)),
                "tops_coherence")
    elif k == "esd":
        T.check(T.lib.tops_esd(st["ovs"], case["overlaps"], case["win_az"], case["win_rg"], 0.3,
                               C.c_void_p(st["out"].data_ptr()), None, C.c_void_p(st["scratch"].data_ptr()),
                               st["bytes"], C.c_void_p(s)), "tops_esd")
    else:
        T.check(T.lib.tops_geocoreg(C.byref(st["job"]), 1, C.c_void_p(st["scratch"].data_ptr()), st["bytes"],
                                    C.c_void_p(s)), "tops_geocoreg")
    return st["out"]


# ------------------------------------------------------- the same, in 64 bits
def x_resample(slc, rows, az, rg, shift, y0, s_first, dt, out_rows=None):
    """Deramp, 12 x 12 LUT sinc, reramp of one burst (int16 [L][W][2]; box lines
    start at y0): complex128 [L][W]."""
    L, W = slc.shape[:2]
    kaz, krg = (torch.from_numpy(k.astype(np.float64)).to(DEV) for k in lut_tables())
    kt, tr, fd = rows
    a2, a1, a0 = -math.pi * kt, 2 * math.pi * kt * tr - 2 * math.pi * fd, -math.pi * kt * tr * tr
    raw = torch.complex(slc[..., 0].double(), slc[..., 1].double())
    d = torch.empty_like(raw)
    for r in range(0, L, 256):
        ta = (torch.arange(r, min(L, r + 256), device=DEV, dtype=torch.float64) + y0 - s_first)[:, None] * dt
        d[r:r + 256] = raw[r:r + 256] * torch.exp(1j * ((a2 * ta + a1) * ta + a0))
    out = torch.zeros(L, W, dtype=torch.complex128, device=DEV)
    Ph = ((torch.arange(W, device=DEV, dtype=torch.float64) - 0.5 * (W - 1)) / (0.25 * (W - 1)))[None, :]
    for r in range(0, L, 128):
        n = min(L, r + 128) - r
        Lh = ((torch.arange(r, r + n, device=DEV, dtype=torch.float64) - 0.5 * (L - 1)) / (0.25 * (L - 1)))[:, None]
        p = lambda c: c[0] + c[1] * Lh + c[2] * Ph + c[3] * Lh * Lh + c[4] * Lh * Ph + c[5] * Ph * Ph
        y, x = p(az) + shift, p(rg)
        l0, p0 = y.trunc(), x.trunc()
        ba = ((y - l0) * 2047 + 0.5).trunc().clamp(0, 2047).long()
        br = ((x - p0) * 2047 + 0.5).trunc().clamp(0, 2047).long()
        l0, p0 = l0.long() - y0, p0.long()
        inside = (l0 >= 0) & (l0 < L) & (p0 >= 0) & (p0 < W)
        inner = (l0 >= 5) & (l0 <= L - 8) & (p0 >= 5) & (p0 <= W - 8)
        acc = torch.zeros(n, W, dtype=torch.complex128, device=DEV)
        wa = [kaz[:, j][ba] for j in range(12)]
        t0 = (l0 + y0 - s_first).double() * dt
        s0 = sum(wa)
        s1 = sum(w * (t0 + (j - 5) * dt) for j, w in enumerate(wa))
        s2 = sum(w * (t0 + (j - 5) * dt) ** 2 for j, w in enumerate(wa))
        ph = torch.zeros(n, W, dtype=torch.float64, device=DEV)
        flat = d.reshape(-1)
        for i in range(12):
            xi = (p0 - 5 + i).clamp(0, W - 1)
            wr = krg[:, i][br]
            col = torch.zeros_like(acc)
            for j in range(12):
                col += wa[j] * flat[(l0 - 5 + j).clamp(0, L - 1) * W + xi]
            acc += wr * col
            ph += wr * (a2[xi] * s2 + a1[xi] * s1 + a0[xi] * s0)
        near = raw.reshape(-1)[l0.clamp(0, L - 1) * W + p0.clamp(0, W - 1)]
        res = torch.where(inner, acc * torch.exp(-1j * ph), near)
        out[r:r + n] = torch.where(inside, res, torch.zeros_like(res))
    return out


def _box(a, win_az, win_rg):
    """Sums over rows r - dy .. r - dy + win_az - 1 and columns likewise, zero pad."""
    for ax, w in ((0, win_az), (1, win_rg)):
        d, n = (w - 1) // 2, a.shape[ax]
        acc = torch.zeros_like(a)
        for o in range(-d, w - d):
            if abs(o) < n:
                acc.narrow(ax, max(0, -o), n - abs(o)).add_(a.narrow(ax, max(0, o), n - abs(o)))
        a = acc
    return a


def _gamma(m, s, win_az, win_rg):
    num = _box(m * s.conj(), win_az, win_rg).abs()
    den = _box(s.abs() ** 2, win_az, win_rg) * _box(m.abs() ** 2, win_az, win_rg)
    return torch.where(den > 0, num / den.clamp(min=1e-300).sqrt(), torch.zeros_like(num))


def _c128(a):
    return torch.complex(a[..., 0].double(), a[..., 1].double())


def x_coherence(m, s, win_az, win_rg):
    """m int16 [L][W][2], s complex128."""
    L, W = s.shape
    out = torch.empty(L, W, dtype=torch.float64, device=DEV)
    for r in range(0, L, 256):
        a, b = max(0, r - 16), min(L, r + 256 + 16)
        g = _gamma(_c128(m[a:b]), s[a:b], win_az, win_rg)
        out[r:r + 256] = g[r - a:min(L, r + 256) - a]
    return torch.where(s.abs() < 1e-3, torch.zeros_like(out), out)


def x_esd(mF, sF, mB, sB, win_az, win_rg, sep, thr=0.3):
    """ESD shift (lines) of one overlap; complex128 bands.  A double difference of
    zero (a slave sample outside its box) has the phase that atan2 gives its
    signed zeros, so the products are written out in real terms."""
    g = 0.5 * (_gamma(mF, sF, win_az, win_rg) + _gamma(mB, sB, win_az, win_rg))
    f, b = ((m.real * s.real + m.imag * s.imag, m.imag * s.real - m.real * s.imag)
            for m, s in ((mF, sF), (mB, sB)))
    ph = torch.atan2(f[1] * b[0] - f[0] * b[1], f[0] * b[0] + f[1] * b[1])
    ph = ph[(g >= thr) & (g < 1)]
    return math.atan2(torch.sin(ph).sum().item(), torch.cos(ph).sum().item()) / (2 * math.pi * sep * DT)


def x_geocoreg(g, b, dem):
    """Offset polynomials [12] of burst b from the DEM window (float32 heights)."""
    r0, c0, nr, nc = g["win"][b]
    L, W = g["L"], g["W"]
    h = dem[r0:r0 + nr, c0:c0 + nc].double()
    d64 = dict(device=DEV, dtype=torch.float64)
    lat = torch.deg2rad(g["lat0"] - g["dlat"] * (r0 + torch.arange(nr, **d64)))[:, None]
    lon = torch.deg2rad(g["lon0"] + g["dlon"] * (c0 + torch.arange(nc, **d64)))[None, :]
    N = ELL_A / torch.sqrt(1.0 - ELL_E2 * torch.sin(lat) ** 2)
    X = [(N + h) * torch.cos(lat) * torch.cos(lon), (N + h) * torch.cos(lat) * torch.sin(lon),
         ((N + h) - ELL_E2 * N) * torch.sin(lat)]
    pos = []
    for w in (0, 1):
        c = orbit_fit(g, w)
        t = torch.full_like(h, 0.5 * (g["first"][b] + g["last"][b]) - g["sv_t"][8])
        ev = lambda k, n, u: sum(float(c[k, i]) * math.perm(i, n) * u ** (i - n) for i in range(n, 6))
        for _ in range(8):
            u = t * 0.1
            f = fp = 0.0
            for k in range(3):
                dx, v, a = X[k] - ev(k, 0, u), ev(k, 1, u) * 0.1, ev(k, 2, u) * 0.01
                f, fp = f + v * dx, fp + a * dx - v * v
            t = t - f / fp
        u = t * 0.1
        R = torch.sqrt(sum((X[k] - ev(k, 0, u)) ** 2 for k in range(3)))
        pos.append((b * L + (t + g["sv_t"][8] - g["first"][b]) / DT, (R - g["slr"] * C0) / DR))
    (ml, mp), (sl, sp) = pos
    ok = (ml >= b * L) & (ml <= (b + 1) * L - 1) & (mp >= 0) & (mp <= W - 1)
    Lh = ((ml - 0.5 * (b * L + (b + 1) * L - 1)) / (0.25 * (L - 1)))[ok]
    Ph = ((mp - 0.5 * (W - 1)) / (0.25 * (W - 1)))[ok]
    A = torch.stack([torch.ones_like(Lh), Lh, Ph, Lh * Lh, Lh * Ph, Ph * Ph], 1)
    sol = torch.linalg.solve(A.T @ A, A.T @ torch.stack([sl[ok], sp[ok]], 1))
    return sol.T.reshape(-1)


def _x_pair(case, seed):
    g = _geom(case)
    nb, L, W = g["nb"], g["L"], g["W"]
    img = [[None] * nb, [None] * nb]
    make_slcs(g, seed, lambda w, b, a: img[w].__setitem__(b, a))
    dem = make_dem(g["dem"], seed)
    rows = [torch.from_numpy(r[0]).to(DEV) for r in deramp_rows(g, 1)]   # burst 0's rows for every burst
    cpm = [x_geocoreg(g, b, dem) for b in range(nb)]
    rs = lambda b, sh: x_resample(img[1][b], rows, cpm[b][:6].tolist(), cpm[b][6:].tolist(), sh, b * L, b * L, DT)
    res = [rs(b, 0.0) for b in range(nb)]
    sep = float((deramp_rows(g, 0)[0] * (L * DT)).sum() / W / nb)
    win = case.get("win_az", 3), case.get("win_rg", 10)
    esd = [res[0]]
    for i in range(nb - 1):
        n = int(math.floor((g["last"][i] - g["first"][i + 1]) / DT))
        sh = x_esd(_c128(img[0][i][L - n:]), res[i][L - n:], _c128(img[0][i + 1][:n]), res[i + 1][:n],
                   win[0], win[1], sep)
        esd.append(rs(i + 1, sh if abs(sh) <= 100 else 0.0))
    coh = [x_coherence(img[0][b], esd[b], *win) for b in range(nb)]
    out = {"reslave_esd": torch.view_as_real(torch.cat(esd)), "coh": torch.cat(coh)}
    if case.get("full", True):
        out["reslave"] = torch.view_as_real(torch.cat(res))
    return out


def exact(case, seed):
    k = case["kind"]
    if k == "batch" or (k in ("pair", "host") and case["bursts"] * case["lines"] * case["samples"] > 30_000_000):
        return None      # about a minute
    if k in ("pair", "host"):
        return _x_pair(case, seed)
    if k == "resample":
        s, rows, az, rg = _resample_inputs(case, seed)
        return torch.view_as_real(x_resample(s, rows, az.tolist(), rg.tolist(), case["shift"], 0, 0, DT))
    if k == "coh":
        m, s = _coh_inputs(case["lines"], case["samples"], seed)
        return x_coherence(m, _c128(s), case["win_az"], case["win_rg"])
    if k == "esd":
        mF, sF, mB, sB = (_c128(a) for a in _esd_inputs(case, seed))
        L = case["lines"]
        return torch.tensor([x_esd(*(a[i * L:(i + 1) * L] for a in (mF, sF, mB, sB)), case["win_az"],
                                   case["win_rg"], ESD_SEP) for i in range(case["overlaps"])],
                            dtype=torch.float64, device=DEV)
    g = _geo_case(case)
    return x_geocoreg(g, 0, make_dem(g["dem"], seed))
