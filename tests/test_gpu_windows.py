"""The quick ring windows (per-ring pixel tables and window records) against
the general ones (HCG_RING_TABLE_MAX=0): the pair counts are equal, and so are
the maps up to the order of an FP64 sum (one rounding to FP32), over caps and
equator, whole polar rings, phi = 0, odd and tiny maps, beams of degrees,
coarsened windows and every kernel."""
import numpy as np
import pytest

from hcgrid_b200 import api, synth

pytestmark = pytest.mark.gpu

CASES = {
    # ra0, dec0, size (deg), nx, ny, fwhm (arcsec), kernel, coarsening factor
    "equator": (30.0, 5.0, 1.5, 33, 17, 180.0, "gauss1d", 1),
    "cap_edge": (120.0, 41.8, 2.0, 40, 41, 180.0, "gauss1d", 1),
    "cap": (200.0, 58.0, 1.0, 31, 9, 120.0, "gauss2d", 1),
    "south": (10.0, -47.0, 1.0, 16, 8, 180.0, "sinc", 1),
    "whole_rings": (250.0, 75.0, 1.2, 18, 20, 300.0, "gauss1d", 1),
    "phi0": (0.0, 20.0, 1.0, 25, 24, 180.0, "gauss1d", 1),
    "one_pixel": (60.0, 30.0, 0.3, 1, 1, 180.0, "gauss1d", 1),
    "wide_beam": (60.0, 10.0, 30.0, 21, 13, 12000.0, "gauss1d", 1),
    "coarse": (60.0, 30.0, 1.0, 29, 21, 180.0, "gauss1d", 3),
}


def grid(monkeypatch, tables, name, nchan, weights):
    ra, dec, size, nx, ny, fwhm, kernel, factor = CASES[name]
    if tables:
        monkeypatch.delenv("HCG_RING_TABLE_MAX", raising=False)
    else:
        monkeypatch.setenv("HCG_RING_TABLE_MAX", "0")
    rng = np.random.default_rng(5)
    lon, lat = synth.raster_scan(6000, ra, dec, size, 2.0, rng)
    vals = rng.normal(1.0, 0.3, (6000, nchan)).astype(np.float32)
    s = fwhm / 3600.0 * synth.FWHM_TO_SIGMA
    kt, kp = {"gauss1d": (api.GAUSS1D, [s, 0.0, 0.0]), "gauss2d": (api.GAUSS2D, [1.3 * s, 0.8 * s, 0.9]),
              "sinc": (api.TAPERED_SINC | api.TAPER_FIX, [s, 2.52, 1.55])}[kernel]
    ctx = api.Context(0)
    ctx.prepare_grid_kernel(kt, np.array(kp), 3 * s, s / 2)
    ctx.set_coarsening_factor(factor)
    f = ctx.field(lon, lat, rng.uniform(0.5, 1.5, 6000) if weights else None)
    f.set_spectra(vals)
    t = ctx.target_from_header(synth.sin_header(nx, ny, ra, dec, size / max(nx, ny)))
    cube, w = ctx.grid(f, t, engine=api.ENGINE_FP32 if nchan > 1 else api.ENGINE_AUTO)
    st = ctx.stats()
    t.close()
    f.close()
    ctx.close()
    return cube, w, (st.pairs_candidate, st.pairs_within, st.ring_skips)


@pytest.mark.parametrize("nchan,weights", [(1, False), (5, False), (5, True)])
@pytest.mark.parametrize("name", sorted(CASES))
def test_quick_windows_equal_general(monkeypatch, name, nchan, weights):
    c0, w0, s0 = grid(monkeypatch, False, name, nchan, weights)
    c1, w1, s1 = grid(monkeypatch, True, name, nchan, weights)
    assert s0 == s1 and s0[1] > 0
    # FP64 sums in another order, rounded to FP32 once
    np.testing.assert_allclose(w1, w0, rtol=2e-7, atol=0)
    np.testing.assert_array_equal(np.isnan(c0), np.isnan(c1))
    scale = np.nanmax(np.abs(c0))
    assert np.nanmax(np.abs(c1 - c0)) <= 1e-6 * scale
