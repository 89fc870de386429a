"""Spectra given as device rows (channel maxima taken while they are put in
order) against the same spectra given as device planes and as host rows
(maxima in a pass of their own): the tensor-core engines' results are equal,
at channel counts around the quads and the 128-channel blocks and sample
counts around a block's rows, and non-finite values are found by each."""
import numpy as np
import pytest

from hcgrid_b200 import api, synth

pytestmark = pytest.mark.gpu


def split_and_grid(n, nchan, how, bad):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + nchan)
    lon, lat = synth.raster_scan(n, 30.0, 20.0, 0.5, 2.0, rng)
    # channel scales over 24 powers of ten
    vals = (rng.normal(0.0, 1.0, (n, nchan)) * 10.0 ** rng.uniform(-12, 12, nchan)).astype(np.float32)
    if bad:
        vals[n - 1, nchan - 1] = np.nan
        vals[n // 2, 0] = np.inf
    s = 180.0 / 3600.0 * synth.FWHM_TO_SIGMA
    ctx = api.Context(0)
    ctx.prepare_grid_kernel(api.GAUSS1D, np.array([s, 0.0, 0.0]), 3 * s, s / 2)
    f = ctx.field(lon, lat, None)
    if how == "host":
        f.set_spectra(vals)
    elif how == "planes":
        f.set_spectra(torch.from_numpy(np.ascontiguousarray(vals.T)).cuda(), api.CHANNEL_MAJOR)
    else:
        wide = torch.zeros(n * nchan + 1, device="cuda")
        rows = wide[how:how + n * nchan].view(n, nchan)  # how = 1: rows that no 16-byte load may touch
        rows.copy_(torch.from_numpy(vals))
        torch.cuda.synchronize()
        f.set_spectra(rows)
    t = ctx.target_from_header(synth.sin_header(17, 9, 30.0, 20.0, 0.5 / 17))
    f.split_spectra(api.ENGINE_TC_F16)
    out = None
    if bad:
        with pytest.raises(api.HcgError, match="2 non-finite"):
            ctx.grid(f, t, engine=api.ENGINE_TC_F16)
    else:
        out = ctx.grid(f, t, engine=api.ENGINE_TC_F16)
    t.close()
    f.close()
    ctx.close()
    return out


@pytest.mark.parametrize("bad", [False, True])
@pytest.mark.parametrize("n,nchan", [(255, 2), (257, 3), (1023, 5), (1025, 64), (900, 127), (900, 128), (1100, 129),
                                     (700, 260)])
def test_device_rows_equal_planes_and_host_rows(n, nchan, bad):
    ref = split_and_grid(n, nchan, "planes", bad)
    for how in ("host", 0, 1):
        got = split_and_grid(n, nchan, how, bad)
        if not bad:  # one operand, one order of accumulation
            np.testing.assert_array_equal(got[0], ref[0])
            np.testing.assert_array_equal(got[1], ref[1])
