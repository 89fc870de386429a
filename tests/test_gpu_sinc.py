"""TAPERED_SINC on either side of the rule that chooses its form (taper in range or
not, series or arcsine), with the reference's growing taper and the falling one,
unit and given sample weights, samples on pixel centres, against the FP64 oracle
within the bounds of the other kernel tests."""
import numpy as np
import pytest

from hcgrid_b200 import api, synth
from test_gpu_kernels import ENGINES, SINGLE, TOL, check, oracle, run

pytestmark = pytest.mark.gpu

# parameters (sigma, a, b in degrees), radius, field size; exponent of the taper in
# powers of two at the radius: 20, 20, 900, 2000, 20
CASES = {
    "falling": (api.TAPERED_SINC | api.TAPER_FIX, [0.02, 2.52, 1.55], 0.06, 0.5),
    "growing": (api.TAPERED_SINC, [0.02, 2.52, 1.55], 0.06, 0.5),
    "in_range": (api.TAPERED_SINC | api.TAPER_FIX, [0.006, 2.52, 1.55], 0.12, 0.3),
    "beyond_range": (api.TAPERED_SINC | api.TAPER_FIX, [0.004, 2.52, 1.55], 0.12, 0.3),
    "arcsine": (api.TAPERED_SINC | api.TAPER_FIX, [2.0, 2.52, 1.55], 6.0, 15.0),
}


@pytest.mark.parametrize("given", [False, True])
@pytest.mark.parametrize("engine", ENGINES)
@pytest.mark.parametrize("name", sorted(CASES))
def test_tapered_sinc_forms(name, engine, given):
    kt, params, r, size = CASES[name]
    rng = np.random.default_rng(11)
    ctx = api.Context(0)
    t = ctx.target_from_header(synth.sin_header(19, 11, 40.0, 25.0, size / 40))
    xw, yw = t.coords()
    lon, lat = synth.raster_scan(8000, 40.0, 25.0, size, 2.0, rng)
    lon[:60], lat[:60] = xw[:60], yw[:60]
    vals = rng.normal(1.0, 0.5, (8000, 3)).astype(np.float32)
    win = rng.uniform(0.2, 3.0, 8000) if given else None
    res = max(params[0] / 2, 0.004)
    cube, w = run(ctx, lon, lat, vals, t, kt, params, r, res, engine, weights=win)
    v = vals[:, :1] if engine == SINGLE else vals
    oc, ow, wabs = oracle(lon, lat, v, xw, yw, params[0], r, res, kt, params, weights=win)
    check(cube, w, oc, ow, wabs, v, TOL[engine])
    t.close()
    ctx.close()
