"""Timed cases of the gridder: what its users have it do, through its public
entry points (hcgrid_b200.api over the C ABI).

Kinds of pass
  grid     hcg_grid on a resident field: the samples are sorted and their
           spectra attached; one map or cube is gridded into device buffers
  scan     a new scan: device positions and values -> hcg_field_create,
           hcg_field_set_spectra (and the tensor-core split), hcg_grid
  spectra  new spectra on known positions: hcg_field_share,
           hcg_field_set_spectra, hcg_field_split_spectra, hcg_grid
  batch    many small scan blocks in one hcg_grid_batch
  planes   channel planes in pinned host memory in, host cube out
           (hcg_grid_planes)

Samples are raster drift scans with 2" position jitter (rows twice as far
apart as the samples of a row); values are Gaussian sources with Gaussian line
profiles over a 1 K offset plus noise, the values of single-dish maps. A target
covers its field: nx x ny SIN pixels of `pix` arcseconds.
"""
import math

import numpy as np
import torch

from hcgrid_b200 import api

SIGMA = 1.0 / math.sqrt(8.0 * math.log(2.0))
D2R = math.pi / 180.0
RA0 = 180.0
ENGINES = {"fp64": api.ENGINE_AUTO, "fp32": api.ENGINE_FP32, "f16": api.ENGINE_TC_F16, "bf16": api.ENGINE_TC_BF16}


def _case(name, kind, n, nchan, nx, ny, pix, fwhm, dec, engine, layout="channel", kernel="gauss1d", jobs=1,
          sample_weights=False):
    c = dict(kind=kind, n=n, nchan=nchan, nx=nx, ny=ny, pix=pix, fwhm=fwhm, dec=dec, engine=engine, layout=layout,
             kernel=kernel, jobs=jobs, sample_weights=sample_weights)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a short scan mapped as it lands: latency, launches, host round trips
        _case("scan_1ch_10k", "scan", 10_000, 1, 64, 64, 60.0, 180.0, 12.0, "fp64"),
        # the ordinary continuum map, gridded again on a resident field (200,000 samples, 5 x 5 degrees)
        _case("map_1ch_200k", "grid", 200_000, 1, 300, 300, 60.0, 180.0, 40.0, "fp64"),
        # a whole survey scan to a continuum map: the sort at scale (20 x 20 degrees)
        _case("scan_1ch_4m", "scan", 4_000_000, 1, 1200, 1200, 60.0, 180.0, 30.0, "fp64"),
        # an elliptical beam with per-sample weights on a small odd-sized cube
        _case("cube_gauss2d_33ch", "grid", 150_001, 33, 251, 203, 60.0, 180.0, 40.0, "fp32", "sample", "gauss2d",
              sample_weights=True),
        # an ordinary spectral cube on the FP32 engine, channels not a multiple of the tile's
        _case("cube_fp32_100ch", "grid", 150_000, 100, 300, 300, 45.0, 180.0, -15.0, "fp32", "sample"),
        # a large cube on the FP32 engine
        _case("cube_fp32_512ch", "grid", 1_000_000, 512, 600, 600, 60.0, 180.0, 30.0, "fp32"),
        # the benchmark's survey cube on the tensor cores, FP16 hi/lo
        _case("cube_f16_1024ch", "grid", 4_000_000, 1024, 1200, 1200, 60.0, 180.0, 30.0, "f16"),
        # wide-band spectra stored as BF16 hi/lo pairs, pixel-major cube
        _case("cube_bf16_2048ch", "grid", 600_000, 2048, 464, 464, 60.0, 180.0, 30.0, "bf16", "sample"),
        # a wide beam on fine pixels (hundreds of pixels a beam): dense tiles
        _case("cube_dense_64ch", "grid", 150_000, 64, 768, 768, 5.6, 300.0, 5.0, "f16"),
        # a served request on a known field: new spectra split and gridded
        _case("spectra_f16_256ch", "spectra", 500_000, 256, 512, 500, 60.0, 180.0, 20.0, "f16"),
        # 64 small blocks of a served stream gridded together
        _case("batch_64x10k", "batch", 10_000, 64, 64, 64, 90.0, 180.0, 25.0, "f16", "sample", jobs=64),
        # host planes in, host cube out, as the command line and the FITS path use it
        _case("planes_192ch", "planes", 300_000, 192, 300, 300, 60.0, 180.0, 10.0, "f16"),
    ]


def _pairs(case):
    """Accepted (pixel, sample) pairs of one job: the beam's disc at the mean density."""
    r = _radius(case) * 3600.0
    area = case["nx"] * case["ny"] * case["pix"] ** 2
    return case["nx"] * case["ny"] * math.pi * r * r * case["n"] / area


def draw(rng):
    """A case of the listed kinds over the same ranges."""
    def logint(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    while True:
        kind = rng.choice(["grid", "grid", "grid", "scan", "scan", "spectra", "batch", "planes"])
        nchan = rng.choice([1, logint(2, 64), rng.choice([64, 128, 256, 512, 1024, 2048]), logint(64, 2048)])
        nx = logint(48, 1200)
        ny = max(32, int(nx * rng.uniform(0.6, 1.2)))
        n, jobs = logint(10_000, 4_000_000), 1
        fwhm = rng.choice([60.0, 180.0, 300.0])
        pix = fwhm / rng.uniform(2.0, 8.0)
        dec = round(rng.uniform(-30.0, 50.0), 2)
        layout = rng.choice(["channel", "sample"])
        kernel = rng.choice(["gauss1d"] * 6 + ["gauss2d", "tapered_sinc"])
        if kind == "batch":
            jobs, n, nx, ny = rng.randint(8, 96), logint(4_000, 30_000), rng.randint(40, 128), rng.randint(40, 128)
            kernel = "gauss1d"
        if kind == "planes":
            layout, nchan = "channel", max(2, nchan)
        if nchan == 1:
            kind = "scan" if kind == "spectra" else kind
            engine = "fp64"
        else:
            engine = rng.choice(["fp32", "f16", "f16", "bf16"])
        if kind == "spectra" and engine == "fp32":
            engine = "f16"
        c = _case(None, kind, n, nchan, nx, ny, round(pix, 2), fwhm, dec, engine, layout, kernel, jobs,
                  kernel == "gauss2d")
        half = 0.5 * ny * pix / 3600.0
        density = math.pi * (_radius(c) * 3600.0) ** 2 * n / (nx * ny * pix * pix)  # samples a beam
        values = jobs * n * nchan
        if (abs(dec) + half > 65.0 or 0.5 * nx * pix / 3600.0 / math.cos(dec * D2R) > 60.0
                or not 8.0 <= density <= 4000.0 or values > 1_000_000_000 or jobs * nx * ny * nchan > 700_000_000
                or jobs * _pairs(c) > 600_000_000 or jobs * _pairs(c) * nchan > 80_000_000_000
                or (kind == "planes" and values > 60_000_000)):
            continue
        return c


# ------------------------------------------------------------------- inputs
def _sigma(case):
    return case["fwhm"] / 3600.0 * SIGMA


def _kernel(case):
    """(type, parameters) as hcg_prepare_grid_kernel takes them."""
    s = _sigma(case)
    return {"gauss1d": (api.GAUSS1D, [s, 0.0, 0.0]), "gauss2d": (api.GAUSS2D, [1.2 * s, 0.8 * s, 0.9]),
            "tapered_sinc": (api.TAPERED_SINC | api.TAPER_FIX, [s, 2.52, 1.55])}[case["kernel"]]


def _radius(case):
    return 3.0 * _sigma(case)


def _resolution(case):
    """Largest HEALPix pixel size of the look-up: half the kernel's (smaller) sigma."""
    return min(_kernel(case)[1][:2]) / 2.0 if case["kernel"] == "gauss2d" else _sigma(case) / 2.0


def _positions(case, gen):
    """(lon, lat) in degrees: `n` samples of a raster over the target's extent."""
    n = case["n"]
    w, h = case["nx"] * case["pix"] / 3600.0, case["ny"] * case["pix"] / 3600.0
    rows = max(1, round(math.sqrt(n / 2.0 * h / w)))
    per_row = -(-n // rows)
    i = torch.arange(n, device="cuda", dtype=torch.float64)
    row = torch.floor(i / per_row)
    jit = 2.0 / 3600.0 * torch.randn((2, n), generator=gen, device="cuda", dtype=torch.float64)
    lat = case["dec"] - h / 2 + (row + 0.5) * (h / rows) + jit[0]
    x = -w / 2 + (i - row * per_row + 0.5) * (w / per_row) + jit[1]
    return RA0 + x / torch.cos(lat * D2R), lat


def _pixels(case):
    """Pixel centres (lon, lat) in degrees of the SIN target, yy * nx + xx."""
    x = torch.arange(1, case["nx"] + 1, device="cuda", dtype=torch.float64) - case["nx"] / 2.0
    y = torch.arange(1, case["ny"] + 1, device="cuda", dtype=torch.float64) - case["ny"] / 2.0
    p = case["pix"] / 3600.0 * D2R
    l, m = (-p * x)[None, :], (p * y)[:, None]
    n = torch.sqrt(1.0 - l * l - m * m)
    d0 = case["dec"] * D2R
    lat = torch.asin(m * math.cos(d0) + n * math.sin(d0))
    lon = RA0 * D2R + torch.atan2(l.expand_as(n), n * math.cos(d0) - m * math.sin(d0))
    return (lon / D2R).reshape(-1).contiguous(), (lat / D2R).reshape(-1).contiguous()


def _spectra(case, lon, lat, gen):
    """[n][nchan] float32: 16 sources with line profiles, an offset and noise."""
    n, nchan, k = case["n"], case["nchan"], 16
    u = torch.rand((6, k), generator=gen, device="cuda")
    w, h = case["nx"] * case["pix"] / 3600.0, case["ny"] * case["pix"] / 3600.0
    sd = case["dec"] + (u[0] - 0.5) * h
    sx = (u[1] - 0.5) * w
    amp = torch.exp(math.log(0.1) + u[2] * math.log(100.0))
    size = case["fwhm"] / 3600.0 * (0.5 + 2.0 * u[3])
    c0, cw = (0.1 + 0.8 * u[4]) * nchan, (0.01 + 0.04 * u[5]) * nchan
    ch = torch.arange(nchan, device="cuda", dtype=torch.float32)
    line = torch.exp(-((ch[None, :] - c0[:, None]) ** 2) / (2.0 * cw[:, None] ** 2)) if nchan > 1 else \
        torch.ones((k, 1), device="cuda")
    out = torch.empty((n, nchan), device="cuda")
    step = max(1, (1 << 26) // nchan)
    for i in range(0, n, step):
        x = ((lon[i:i + step] - RA0) * torch.cos(lat[i:i + step] * D2R)).float()
        dx, dy = x[:, None] - sx, lat[i:i + step].float()[:, None] - sd
        g = amp * torch.exp(-(dx * dx + dy * dy) / (2.0 * size * size))
        v = torch.mm(g, line, out=out[i:i + step])
        v.add_(torch.randn(v.shape, generator=gen, device="cuda"), alpha=0.05).add_(1.0)
    return out


def _job_inputs(case, seed, j):
    """Positions, values and sample weights (or None) of job j, on the GPU."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed((int(seed) * 1009 + j) & 0x7FFFFFFFFFFFFFFF)
    lon, lat = _positions(case, gen)
    w = 0.5 + torch.rand(case["n"], generator=gen, device="cuda", dtype=torch.float64) if case["sample_weights"] \
        else None
    return lon, lat, _spectra(case, lon, lat, gen), w


# ------------------------------------------------------------------ the pass
class _State:
    pass


def prepare(case, seed):
    st = _State()
    st.case = case
    st.kind, st.engine = case["kind"], ENGINES[case["engine"]]
    st.layout = api.CHANNEL_MAJOR if case["layout"] == "channel" else api.SAMPLE_MAJOR
    st.split = case["engine"] in ("f16", "bf16")
    npix, nchan = case["nx"] * case["ny"], case["nchan"]
    st.ctx = api.Context(0)
    kt, kp = _kernel(case)
    st.ctx.prepare_grid_kernel(kt, np.array(kp, np.float64), _radius(case), _resolution(case))
    x, y = _pixels(case)
    torch.cuda.synchronize()
    st.target = st.ctx.target(case["nx"], case["ny"], x, y)
    st.ctx.synchronize()
    shape = (npix, nchan) if st.layout == api.SAMPLE_MAJOR else (nchan, npix)
    if st.kind == "planes":
        lon, lat, values, w = _job_inputs(case, seed, 0)
        st.planes = torch.empty((nchan, case["n"]), pin_memory=True)
        st.planes.copy_(values.t().contiguous())
        torch.cuda.synchronize()
        st.field = st.ctx.field(lon, lat, w)
        st.cube = torch.empty(shape, pin_memory=True)
        st.weights = torch.empty(npix, pin_memory=True)
        st.ctx.synchronize()
        return st
    if st.kind == "batch":
        # one buffer for the blocks' cubes and one for their weight maps
        st.cube = torch.empty((case["jobs"],) + shape, device="cuda")
        st.weights = torch.empty((case["jobs"], npix), device="cuda")
        st.jobs = []
        for j in range(case["jobs"]):
            lon, lat, values, w = _job_inputs(case, seed, j)
            torch.cuda.synchronize()
            f = st.ctx.field(lon, lat, w)
            f.set_spectra(values)
            if st.split:
                f.split_spectra(st.engine, keep_fp32=False)
            st.ctx.synchronize()
            st.jobs.append((f, st.target, st.cube[j], st.weights[j], st.layout))
        return st
    st.cube = torch.empty(shape, device="cuda")
    st.weights = torch.empty(npix, device="cuda")
    lon, lat, values, w = _job_inputs(case, seed, 0)
    torch.cuda.synchronize()
    if st.kind == "scan":
        st.lon, st.lat, st.values, st.w = lon, lat, values, w
        return st
    st.field = st.ctx.field(lon, lat, w)
    if st.kind == "spectra":
        st.values = values
    else:
        st.field.set_spectra(values)
        if st.split:
            st.field.split_spectra(st.engine, keep_fp32=False)
    st.ctx.synchronize()
    return st


def run(st):
    if st.kind == "grid":
        st.ctx.grid(st.field, st.target, st.cube, st.weights, st.layout, st.engine)
    elif st.kind == "planes":
        st.ctx.grid_planes(st.field, st.target, st.planes, st.cube, st.weights, st.layout, st.engine)
    elif st.kind == "batch":
        st.ctx.grid_batch(st.jobs)
    else:
        f = st.ctx.field(st.lon, st.lat, st.w) if st.kind == "scan" else st.field.share()
        f.set_spectra(st.values)
        if st.split:
            f.split_spectra(st.engine, keep_fp32=False)
        st.ctx.grid(f, st.target, st.cube, st.weights, st.layout, st.engine)
        f.close()
    return st.cube, st.weights


def work(case):
    """Positions, spectra and pixel centres read once, cube and weights
    written once; one multiply-add per accepted pair and channel. Gridding a
    resident field also reads positions and spectra (4 bytes a value in
    either form); `spectra` and `scan` passes read the caller's."""
    n, c, p = case["n"], case["nchan"], case["nx"] * case["ny"]
    nbytes = n * (16 + 4 * c + (8 if case["sample_weights"] else 0)) + p * (16 + 4 * c + 4)
    return {"bytes": case["jobs"] * nbytes, "flops": case["jobs"] * 2.0 * _pairs(case) * c}


# -------------------------------------------------------------- 64-bit result
def _ring_half(ns, ring, tt):
    """HEALPix position along the ring numbered `ring` of longitudes tt (units
    of pi / 2): pixels of a ring count from 0 (RING scheme, Gorski et al. 2005)."""
    nl4 = 4 * ns
    k = 2 * ns - ring  # 3 ns z / 2: the ring's offset from the equator
    t1 = ns * (0.5 + tt)
    jp, jm = torch.floor(t1 - 0.5 * k), torch.floor(t1 + 0.5 * k)
    shift = torch.remainder(ring - ns, 2)  # rings start half a pixel apart
    eq = torch.remainder(torch.floor((jp + jm + shift + 1 + 2 * nl4 - ns) * 0.5), nl4)
    cap = torch.floor(tt * torch.minimum(ring, nl4 - ring))
    return torch.where((ring >= ns) & (ring <= 3 * ns), eq, cap)


def _ring_of(ns, theta, tt):
    """Ring of the pixel that holds (theta, tt)."""
    z = torch.cos(theta)
    za = z.abs()
    t1, t2 = ns * (0.5 + tt), ns * z * 0.75
    eq = 2 * ns + torch.floor(t1 - t2) - torch.floor(t1 + t2)
    tp, tmp = tt - torch.floor(tt), ns * torch.sqrt(3.0 * (1.0 - za))
    ir = torch.floor(tp * tmp) + torch.floor((1.0 - tp) * tmp) + 1
    return torch.where(za <= 2.0 / 3.0, eq, torch.where(z > 0, ir, 4 * ns - ir))


def _quarter(phi):
    return torch.remainder(phi * (2.0 / math.pi), 4.0)


def _weight(case, d, l1, b1, l2, b2):
    """Kernel weights at distance d (degrees)."""
    s = _sigma(case)
    if case["kernel"] == "gauss1d":
        return torch.exp(-d * d * (0.5 / s ** 2))
    p = _kernel(case)[1]
    if case["kernel"] == "gauss2d":
        bear = torch.atan2(torch.cos(b2) * torch.sin(l2 - l1),
                           torch.cos(b1) * torch.sin(b2) - torch.sin(b1) * torch.cos(b2) * torch.cos(l2 - l1)) - p[2]
        ell = (p[0] * torch.sin(bear)) ** 2 + (p[1] * torch.cos(bear)) ** 2
        return torch.exp(-0.5 * (d / p[0] / p[1]) ** 2 * ell)
    arg = math.pi * d / p[0]
    x = arg / p[2]
    sinc = torch.where(x.abs() < 1e-10, torch.ones_like(x), torch.sin(x) / torch.where(x == 0, torch.ones_like(x), x))
    return sinc * torch.exp(-((arg / p[1]) ** 2))


def _exact_job(case, lon, lat, values, w):
    """Weighted mean over the samples within the radius of each pixel, among
    those of the pixels [phi - disc, phi + disc] of the rings the disc reaches
    (the gridder's candidate rule; the first ring with samples is not gridded)."""
    r = _radius(case)
    ns = 1 << int(math.sqrt(math.pi / 3.0) / (_resolution(case) * D2R) + 0.5).bit_length()
    disc = r * D2R + math.sqrt(4.0 * math.pi / (12.0 * ns * ns))
    hcut = math.sin(0.5 * r * D2R) ** 2
    l2, b2 = lon * D2R, lat * D2R
    tt2 = _quarter(l2)
    ring2 = _ring_of(ns, 0.5 * math.pi - b2, tt2)
    pos2 = _ring_half(ns, ring2, tt2)
    keep = ring2 != ring2.min()
    X, Y = _pixels(case)
    nx, ny, nchan = case["nx"], case["ny"], values.shape[1]
    cube = torch.full((ny, nx, nchan), float("nan"), device="cuda", dtype=torch.float64)
    wsum = torch.zeros((ny, nx), device="cuda", dtype=torch.float64)
    T = 32
    for y0 in range(0, ny, T):
        y1 = min(ny, y0 + T)
        band = Y.view(ny, nx)[y0:y1]
        rows = torch.nonzero((lat >= band.min() - r) & (lat <= band.max() + r) & keep)[:, 0]
        lrow = lon[rows]
        wide = r / math.cos(D2R * min(89.0, float(band.abs().max()) + r)) + 1e-6
        for x0 in range(0, nx, T):
            x1 = min(nx, x0 + T)
            px = X.view(ny, nx)[y0:y1, x0:x1].reshape(-1, 1)
            l1, b1 = px * D2R, Y.view(ny, nx)[y0:y1, x0:x1].reshape(-1, 1) * D2R
            idx = rows[(lrow >= px.min() - wide) & (lrow <= px.max() + wide)]
            if idx.numel() == 0:
                continue
            ls, bs = l2[idx][None, :], b2[idx][None, :]
            h = torch.sin(0.5 * (b1 - bs)) ** 2 + torch.cos(b1) * torch.cos(bs) * torch.sin(0.5 * (l1 - ls)) ** 2
            ok = h < hcut
            rs, ps = ring2[idx][None, :], pos2[idx][None, :]
            ok &= (ps >= _ring_half(ns, rs, _quarter(l1 - disc))) & (ps <= _ring_half(ns, rs, _quarter(l1 + disc)))
            tt1 = _quarter(l1)
            ok &= (rs >= _ring_of(ns, 0.5 * math.pi - b1 - disc, tt1)) & \
                (rs <= _ring_of(ns, 0.5 * math.pi - b1 + disc, tt1))
            d = 2.0 * torch.asin(torch.sqrt(h)) / D2R
            wt = torch.where(ok, _weight(case, d, l1, b1, ls, bs), torch.zeros_like(h))
            if w is not None:
                wt = wt * w[idx]
            tot = wt.sum(1)
            wsum[y0:y1, x0:x1] = tot.view(y1 - y0, x1 - x0)
            cube[y0:y1, x0:x1] = ((wt @ values[idx].double()) / tot[:, None]).view(y1 - y0, x1 - x0, nchan)
    cube, wsum = cube.view(ny * nx, nchan), wsum.view(-1)
    return cube if case["layout"] == "sample" else cube.t().contiguous(), wsum


def exact(case, seed):
    if case["jobs"] * _pairs(case) * (4.0 + case["nchan"] / 8.0) > 4e11:
        return None  # minutes in 64 bits
    out = []
    for j in range(case["jobs"]):
        out.append(_exact_job(case, *_job_inputs(case, seed, j)))
        if case["jobs"] == 1:
            return out[0]
    return torch.stack([o[0] for o in out]), torch.stack([o[1] for o in out])
