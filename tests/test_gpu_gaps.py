"""Ring tables of samples that lie apart: gaps along a ring and between rings, from
no pixel to most of the circle (runs that a lane or a warp fills), against the FP64
oracle: sorted keys, ring table, pair counts and maps."""
import numpy as np
import pytest

from hcgrid_b200 import api
from oracle import oracle as O
from test_gpu_kernels import check

pytestmark = pytest.mark.gpu

PIXELS = [0, 1, 2, 15, 16, 17, 18, 31, 32, 33, 48, 64, 65, 1000, 9000]
RINGS = [1, 2, 15, 16, 17, 18, 33, 64, 300, 0]


@pytest.mark.parametrize("dec0", [-12.0, 44.0])
@pytest.mark.parametrize("copies", [1, 3])
def test_gaps_of_every_length(monkeypatch, copies, dec0):
    monkeypatch.delenv("HCG_RING_TABLE_MAX", raising=False)
    s = 0.02
    g = O.prepare_grid_kernel(s, 3 * s, s / 2)
    rng = np.random.default_rng(copies)
    dpix = 360.0 / (4 * g.hpx.nside)  # an equatorial ring's pixel; a cap's are longer
    lon, lat = [], []
    dec = dec0
    for r in RINGS:
        for _ in range(4):  # the gaps in four orders, so that warps begin anywhere
            x = 10.3 + np.cumsum(rng.permutation(PIXELS)) * dpix
            lon.append(np.repeat(x, copies))
            lat.append(np.full(len(x) * copies, dec))
        dec += r * 2.0 / 3.0 / g.hpx.nside * 180.0 / np.pi
    lon = np.mod(np.concatenate(lon) + 355.0, 360.0)  # some rings cross longitude 0
    lat = np.concatenate(lat) + 1e-7 * rng.normal(size=lon.size)
    order = rng.permutation(lon.size)
    lon, lat = lon[order], lat[order]
    n = lon.size
    xw, yw = (v.ravel() for v in np.meshgrid(np.mod(np.unique(np.round(lon, 2))[::7] + 0.003, 360.0),
                                             np.unique(np.round(lat, 2)) + 0.004))
    vals = rng.normal(1.0, 0.3, n).astype(np.float32)
    ctx = api.Context(0)
    ctx.prepare_grid_kernel(api.GAUSS1D, np.array([s, 0.0, 0.0]), 3 * s, s / 2)
    f = ctx.field(lon, lat)
    f.set_spectra(vals)
    nx = len(np.unique(xw))
    t = ctx.target(nx, len(xw) // nx, xw, yw)
    cube, w = ctx.grid(f, t)
    st = ctx.stats()
    keys, _, lut = f.sorted()[:3]
    ps = O.presort(g.hpx, lon, lat)
    np.testing.assert_array_equal(keys, ps.keys)
    np.testing.assert_array_equal(lut, ps.lut)
    oc, ow, os_, wabs = O.grid(g, ps, lon[ps.perm], lat[ps.perm], vals[ps.perm].astype(np.float64)[:, None], xw, yw,
                               want_abs=True)
    assert os_.pairs_within > 100
    assert st.pairs_candidate == os_.pairs_visited and st.pairs_within == os_.pairs_within
    with np.errstate(invalid="ignore", divide="ignore"):
        check(np.asarray(cube).reshape(len(xw), 1), w, oc.reshape(len(xw), 1), ow, wabs, vals, 1e-6)
    t.close()
    f.close()
    ctx.close()
