"""The pair tests' forms (unit or given sample weights, Gaussians evaluated in
a known range or by exp, series or arcsine, entries or tensor-core operand) on
either side of the rules that choose them, against the FP64 oracle, with
samples on pixel centres (no distance, no bearing) and a partial tile. The
bounds are those of the other kernel tests (per pixel tol * kappa * max|x|)."""
import numpy as np
import pytest

from hcgrid_b200 import api, synth
from test_gpu_kernels import ENGINES, SINGLE, TOL, check, oracle, run

pytestmark = pytest.mark.gpu

# kernel, parameters (degrees), radius, field size: the radius in sigmas decides
# between the forms (FP32 weights below 2^-120 beyond 12.9, FP64 weights below
# 2^-1000 beyond 37), 3.6 degrees between series and arcsine
CASES = {
    "unit": (api.GAUSS1D, [0.02, 0.0, 0.0], 0.06, 0.5),
    "beyond_fp32": (api.GAUSS1D, [0.01, 0.0, 0.0], 0.14, 0.5),
    "beyond_fp64": (api.GAUSS1D, [0.003, 0.0, 0.0], 0.12, 0.3),
    "arcsine": (api.GAUSS1D, [2.0, 0.0, 0.0], 6.0, 15.0),
    "ellipse": (api.GAUSS2D, [0.028, 0.014, 0.9], 0.06, 0.5),
    "thin_ellipse": (api.GAUSS2D, [0.03, 0.002, -0.4], 0.09, 0.5),
    "wide_ellipse": (api.GAUSS2D, [2.0, 1.0, 0.3], 6.0, 15.0),
}


@pytest.mark.parametrize("given", [False, True])
@pytest.mark.parametrize("engine", ENGINES)
@pytest.mark.parametrize("name", sorted(CASES))
def test_forms_match_oracle(name, engine, given):
    kt, params, r, size = CASES[name]
    rng = np.random.default_rng(11)
    ctx = api.Context(0)
    t = ctx.target_from_header(synth.sin_header(19, 11, 40.0, 25.0, size / 40))
    xw, yw = t.coords()
    lon, lat = synth.raster_scan(3000, 40.0, 25.0, size, 2.0, rng)
    lon[:60], lat[:60] = xw[:60], yw[:60]
    vals = rng.normal(1.0, 0.5, (3000, 3)).astype(np.float32)
    win = rng.uniform(0.2, 3.0, 3000) if given else None
    res = max(params[0] / 2, 0.004)
    cube, w = run(ctx, lon, lat, vals, t, kt, params, r, res, engine, weights=win)
    v = vals[:, :1] if engine == SINGLE else vals
    oc, ow, wabs = oracle(lon, lat, v, xw, yw, params[0], r, res, kt, params, weights=win)
    check(cube, w, oc, ow, wabs, v, TOL[engine])
    t.close()
    ctx.close()


@pytest.mark.parametrize("mode", [api.TC_WEIGHTS_ENTRIES, api.TC_WEIGHTS_DIRECT])
@pytest.mark.parametrize("nchan", [3, 130])
def test_unit_weights_equal_ones_on_tensor_cores(nchan, mode):
    """No weights against weights of one, both operand forms, many chunks a tile."""
    rng = np.random.default_rng(3)
    lon, lat = synth.raster_scan(30_000, 40.0, 25.0, 0.5, 2.0, rng)
    vals = rng.normal(1.0, 0.5, (30_000, nchan)).astype(np.float32)
    out = []
    for win in (None, np.ones(30_000)):
        ctx = api.Context(0)
        ctx.tc_set_weights(mode)
        t = ctx.target_from_header(synth.sin_header(37, 21, 40.0, 25.0, 0.5 / 40))
        out.append(run(ctx, lon, lat, vals, t, api.GAUSS1D, [0.05, 0.0, 0.0], 0.15, 0.025, api.ENGINE_TC_F16,
                       weights=win))
        t.close()
        ctx.close()
    # FP32 weights that differ by a rounding of the exponent's scale at most
    np.testing.assert_allclose(out[1][1], out[0][1], rtol=1e-6)
    np.testing.assert_allclose(out[1][0], out[0][0], atol=1e-5 * np.abs(vals).max())
