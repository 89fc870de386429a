"""Windows of fields without pixel tables: by searches of the sorted samples, in
32-bit and (nside above 2^26) wider pixel numbers. Pair counts equal to the FP64
oracle's, cubes and weights within the bounds of the other kernel tests, over caps
and equator, whole rings, phi = 0, few and many samples a ring, odd and tiny maps."""
import numpy as np
import pytest

from hcgrid_b200 import api, synth
from oracle import oracle as O
from test_gpu_kernels import TOL, check

pytestmark = pytest.mark.gpu

CASES = {
    # ra0, dec0, size (deg), nx, ny, fwhm (arcsec), samples
    "equator": (30.0, 5.0, 1.5, 33, 17, 180.0, 6000),
    "cap_edge": (120.0, 41.8, 2.0, 40, 41, 180.0, 6000),
    "cap": (200.0, 58.0, 1.0, 31, 9, 120.0, 6000),
    "south": (10.0, -47.0, 1.0, 16, 8, 180.0, 6000),
    "whole_rings": (250.0, 75.0, 1.2, 18, 20, 300.0, 6000),
    "phi0": (0.0, 20.0, 1.0, 25, 24, 180.0, 6000),
    "dense": (75.0, -12.0, 0.4, 17, 15, 180.0, 60_000),
    "few": (75.0, -12.0, 8.0, 40, 30, 180.0, 40),
    "one_sample": (75.0, -12.0, 1.0, 9, 7, 1800.0, 1),
    "one_pixel": (60.0, 30.0, 0.3, 1, 1, 180.0, 6000),
    "wide_beam": (60.0, 10.0, 30.0, 21, 13, 12000.0, 6000),
    "fine": (75.0, -12.0, 2.5e-5, 21, 19, 0.01, 3000),
    "finest": (220.0, -35.0, 1.2e-5, 15, 17, 0.005, 3000),
    "fine_cap": (300.0, 55.0, 2.5e-5, 21, 19, 0.01, 3000),
}


@pytest.mark.parametrize("nchan", [1, 5])
@pytest.mark.parametrize("name", sorted(CASES))
def test_fields_without_tables(monkeypatch, name, nchan):
    monkeypatch.setenv("HCG_RING_TABLE_MAX", "0")
    ra, dec, size, nx, ny, fwhm, n = CASES[name]
    rng = np.random.default_rng(n + nx)
    lon, lat = synth.raster_scan(n, ra, dec, size, 0.01 * fwhm, rng)
    vals = rng.normal(1.0, 0.3, (n, nchan)).astype(np.float32)
    s = fwhm / 3600.0 * synth.FWHM_TO_SIGMA
    g = O.prepare_grid_kernel(s, 3 * s, s / 2)
    assert (g.hpx.nside > 1 << 26) == name.startswith("fine")
    ctx = api.Context(0)
    ctx.prepare_grid_kernel(api.GAUSS1D, np.array([s, 0.0, 0.0]), 3 * s, s / 2)
    f = ctx.field(lon, lat)
    f.set_spectra(vals)
    t = ctx.target_from_header(synth.sin_header(nx, ny, ra, dec, size / max(nx, ny)))
    xw, yw = t.coords()
    engine = api.ENGINE_FP32 if nchan > 1 else api.ENGINE_AUTO
    cube, w = ctx.grid(f, t, engine=engine)
    st = ctx.stats()
    ps = O.presort(g.hpx, lon, lat)
    oc, ow, os_, wabs = O.grid(g, ps, lon[ps.perm], lat[ps.perm], vals[ps.perm].astype(np.float64), xw, yw,
                               want_abs=True)
    assert st.pairs_candidate == os_.pairs_visited and st.pairs_within == os_.pairs_within and st.ring_skips == os_.a3_events
    with np.errstate(invalid="ignore", divide="ignore"):
        check(np.asarray(cube).reshape(nx * ny, nchan), w, oc.reshape(nx * ny, -1), ow, wabs, vals,
              1e-6 if nchan == 1 else TOL[api.ENGINE_FP32])
    t.close()
    f.close()
    ctx.close()
