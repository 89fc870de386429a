"""Blank pixels (non-finite coordinates): NaN with weight 0 whatever windows they
take, and the pixels around them as without them. With a coarsening factor a
blank pixel takes the windows of its run's first pixel (HCGrid/gridding.cu:284-308),
and its own NaN distance accepts nothing; a run whose first pixel is blank has no
windows at all. The field holds (0, 0), so that operands of a zero position would
accept samples of it; no window of a pixel wraps at longitude 0 (the reference
finds nothing in one that does)."""
import numpy as np
import pytest

from hcgrid_b200 import api, synth

pytestmark = pytest.mark.gpu

NX, NY, N = 37, 18, 8000
S = 0.02


def grid(xw, yw, factor, kernel, nchan, how, weights):
    rng = np.random.default_rng(8)
    lon, lat = synth.raster_scan(N, 0.4, 0.0, 1.0, 2.0, rng)
    vals = rng.normal(1.0, 0.3, (N, nchan)).astype(np.float32)
    kt, kp = {"gauss1d": (api.GAUSS1D, [S, 0.0, 0.0]), "gauss2d": (api.GAUSS2D, [1.3 * S, 0.8 * S, 0.9]),
              "sinc": (api.TAPERED_SINC | api.TAPER_FIX, [S, 2.52, 1.55])}[kernel]
    ctx = api.Context(0)
    ctx.prepare_grid_kernel(kt, np.array(kp), 3 * S, S / 2)
    ctx.set_coarsening_factor(factor)
    f = ctx.field(lon, lat, rng.uniform(0.5, 1.5, N) if weights else None)
    f.set_spectra(vals)
    t = ctx.target(NX, NY, xw, yw)
    if how in ("entries", "direct", "batch"):
        ctx.tc_set_weights(api.TC_WEIGHTS_DIRECT if how == "direct" else api.TC_WEIGHTS_ENTRIES)
        f.split_spectra(api.ENGINE_TC_F16)
    if how == "batch":
        import torch
        cube = torch.empty((NX * NY, nchan), device="cuda")
        w = torch.empty(NX * NY, device="cuda")
        ctx.grid_batch([(f, t, cube, w, api.SAMPLE_MAJOR)])
        ctx.synchronize()
        cube, w = cube.cpu().numpy(), w.cpu().numpy()
    else:
        engine = {"fp32": api.ENGINE_FP32, "fp64": api.ENGINE_AUTO}.get(how, api.ENGINE_TC_F16)
        cube, w = ctx.grid(f, t, engine=engine)
    t.close()
    f.close()
    ctx.close()
    return np.asarray(cube).reshape(NX * NY, nchan), np.asarray(w).reshape(-1)


@pytest.mark.parametrize("kernel,nchan,how,weights", [
    ("gauss1d", 1, "fp64", False), ("gauss1d", 1, "fp64", True), ("gauss2d", 1, "fp64", False),
    ("sinc", 1, "fp64", False), ("gauss1d", 5, "fp32", False), ("gauss1d", 5, "fp32", True),
    ("gauss2d", 5, "fp32", False), ("sinc", 5, "fp32", False), ("gauss1d", 5, "entries", False),
    ("gauss1d", 5, "direct", False), ("gauss1d", 5, "direct", True), ("gauss1d", 5, "batch", False)])
@pytest.mark.parametrize("factor", [1, 2, 3])
@pytest.mark.parametrize("tables", [True, False])
def test_blank_pixels(monkeypatch, tables, factor, kernel, nchan, how, weights):
    if tables:
        monkeypatch.delenv("HCG_RING_TABLE_MAX", raising=False)
    else:
        monkeypatch.setenv("HCG_RING_TABLE_MAX", "0")
    xw, yw = np.tile(0.08 + 0.02 * np.arange(NX), NY), np.repeat(0.02 * (np.arange(NY) - NY / 2 + 0.25), NX)
    want, ww = grid(xw, yw, factor, kernel, nchan, how, weights)
    assert np.isfinite(want).all() and (ww != 0).all()
    rng = np.random.default_rng(2)
    blank = rng.random(NX * NY) < 0.3
    bx, by = xw.copy(), yw.copy()
    bx[blank] = np.where(rng.random(blank.sum()) < 0.7, np.nan, np.inf)
    by[blank] = np.where(rng.random(blank.sum()) < 0.7, np.nan, by[blank])
    col = np.arange(NX * NY) % NX
    none = blank | blank[np.arange(NX * NY) - col % factor]
    assert factor == 1 or (blank & ~blank[np.arange(NX * NY) - col % factor]).sum() > 50
    got, gw = grid(bx, by, factor, kernel, nchan, how, weights)
    assert np.isnan(got[none]).all() and (gw[none] == 0).all()
    # another order of the FP64 sums, rounded to FP32 once; the engines' own sums beyond that
    tol = 1e-6 if how in ("fp64", "fp32") else 1e-5
    np.testing.assert_allclose(gw[~none], ww[~none], rtol=3e-7 if kernel != "sinc" else 1e-5)
    assert np.abs(got[~none] - want[~none]).max() <= tol * np.abs(want).max() * (1 if kernel != "sinc" else 10)
