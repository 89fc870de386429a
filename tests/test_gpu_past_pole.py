"""Target pixels past a pole (|latitude| above 90 degrees: the point on the
other side): the reference's distance formula (helpers.cu:128-130) holds there as
it stands, with a negative cos(latitude), and so do its whole-ring windows. (The
rings reach as far past the pole as the disc does, so pixels farther out have
vanishing weights: not taken.) Every
pair form and engine against the FP64 oracle; the bounds are those of the other
kernel tests."""
import numpy as np
import pytest

from hcgrid_b200 import api
from test_gpu_kernels import ENGINES, SINGLE, TOL, check, oracle, run

pytestmark = pytest.mark.gpu

DIRECT = "direct"  # the tensor-core kernel that evaluates the weights itself

CASES = {
    "unit": (api.GAUSS1D, [0.2, 0.0, 0.0], 0.6),
    "arcsine": (api.GAUSS1D, [1.4, 0.0, 0.0], 4.2),
    "ellipse": (api.GAUSS2D, [0.25, 0.14, 0.9], 0.6),
    "sinc": (api.TAPERED_SINC | api.TAPER_FIX, [0.2, 2.52, 1.55], 0.6),
}


@pytest.mark.parametrize("tables", [True, False])
@pytest.mark.parametrize("pole", [1, -1])
@pytest.mark.parametrize("given", [False, True])
@pytest.mark.parametrize("engine", ENGINES + [DIRECT])
@pytest.mark.parametrize("name", sorted(CASES))
def test_pixels_past_a_pole(monkeypatch, name, engine, given, pole, tables):
    if tables:
        monkeypatch.delenv("HCG_RING_TABLE_MAX", raising=False)
    else:
        monkeypatch.setenv("HCG_RING_TABLE_MAX", "0")
    kt, params, r = CASES[name]
    if engine == DIRECT and kt != api.GAUSS1D:
        pytest.skip("direct weights are GAUSS1D's")
    rng = np.random.default_rng(4)
    n = 6000
    lat = pole * (90.0 - 3.0 * np.sqrt(rng.random(n)))
    lon = rng.uniform(0.0, 360.0, n)
    xw, yw = (v.ravel() for v in np.meshgrid(40.0 + 20.0 * np.arange(13), pole * (89.6 + 0.06 * np.arange(15))))
    yw = yw + pole * rng.uniform(0.0, 0.03, yw.size)
    assert (np.abs(yw) > 90).sum() > 70
    vals = rng.normal(1.0, 0.5, (n, 3)).astype(np.float32)
    win = rng.uniform(0.2, 3.0, n) if given else None
    ctx = api.Context(0)
    t = ctx.target(13, 15, xw, yw)
    if engine == DIRECT:
        ctx.tc_set_weights(api.TC_WEIGHTS_DIRECT)
        engine = api.ENGINE_TC_F16
    cube, w = run(ctx, lon, lat, vals, t, kt, params, r, params[0] / 2, engine, weights=win)
    v = vals[:, :1] if engine == SINGLE else vals
    oc, ow, wabs = oracle(lon, lat, v, xw, yw, params[0], r, params[0] / 2, kt, params, weights=win)
    assert (wabs[np.abs(yw) > 90] > 0).any()
    check(cube, w, oc, ow, wabs, v, TOL[engine])
    t.close()
    ctx.close()
