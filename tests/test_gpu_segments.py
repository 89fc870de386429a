"""Items of several accumulation segments on the tensor cores: the sums of the
segments go through the cube in every form of its stores (planes, rows by 32 and 16
bytes, single values, partial channel blocks, odd addresses), with the same values,
and they agree with the FP32 engine."""
import numpy as np
import pytest
import torch

from hcgrid_b200 import api, synth

pytestmark = pytest.mark.gpu

NX, NY, N = 23, 13, 9000


@pytest.mark.parametrize("mode", [api.TC_WEIGHTS_ENTRIES, api.TC_WEIGHTS_DIRECT])
@pytest.mark.parametrize("nchan", [5, 32, 60, 64, 100, 130, 250, 256, 260, 328])
def test_segments_in_every_store_form(nchan, mode):
    rng = np.random.default_rng(nchan)
    lon, lat = synth.raster_scan(N, 40.0, 25.0, 0.5, 2.0, rng)
    vals = rng.normal(1.0, 0.5, (N, nchan)).astype(np.float32)
    ctx = api.Context(0)
    ctx.prepare_grid_kernel(api.GAUSS1D, np.array([0.06, 0.0, 0.0]), 0.18, 0.03)
    ctx.tc_set_weights(mode)
    f = ctx.field(lon, lat)
    f.set_spectra(vals)
    f.split_spectra(api.ENGINE_TC_F16)
    t = ctx.target_from_header(synth.sin_header(NX, NY, 40.0, 25.0, 0.3 / NX))
    P = NX * NY

    def grid(layout, offset, engine=api.ENGINE_TC_F16):
        buf = torch.full((P * nchan + 16,), 7.0, device="cuda")
        w = torch.empty(P, device="cuda")
        torch.cuda.synchronize()
        cube = buf[offset:offset + P * nchan]
        cube = cube.view(P, nchan) if layout == api.SAMPLE_MAJOR else cube.view(nchan, P)
        ctx.grid(f, t, cube, w, layout, engine)
        ctx.synchronize()
        macs = ctx.stats().tc_macs
        out = buf.cpu().numpy()
        assert (out[:offset] == 7.0).all() and (out[offset + P * nchan:] == 7.0).all()
        c = cube.cpu().numpy()
        return (c if layout == api.SAMPLE_MAJOR else c.T), macs

    rows, macs = grid(api.SAMPLE_MAJOR, 0)
    tiles, blocks = ((NX + 15) // 16) * ((NY + 7) // 8), (nchan + 63) // 64
    assert macs >= 3 * 128 * 64 * 64 * 22 * tiles * blocks  # more than 1,344 slots a tile: segments
    for layout in (api.SAMPLE_MAJOR, api.CHANNEL_MAJOR):
        for offset in (0, 1, 2, 4):
            got, _ = grid(layout, offset)
            np.testing.assert_array_equal(got, rows)
    want, _ = grid(api.SAMPLE_MAJOR, 0, api.ENGINE_FP32)
    assert np.isfinite(want).all()
    assert np.abs(rows - want).max() <= 2e-5 * np.abs(vals).max()  # both engines' 1e-5
    t.close()
    f.close()
    ctx.close()
