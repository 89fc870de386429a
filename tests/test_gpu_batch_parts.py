"""Batches of few and many tiles (eight, four, two and one blocks a tile in the
weight pass), partial tiles among them, against the same jobs gridded one by one."""
import numpy as np
import pytest
import torch

from hcgrid_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", [api.ENGINE_FP32, api.ENGINE_TC_F16])
@pytest.mark.parametrize("weights", [False, True])
@pytest.mark.parametrize("njobs", [1, 5, 9, 10, 39, 40, 78, 79, 100])
def test_blocks_that_share_a_tile(njobs, weights, engine):
    """15 tiles a job: 147 / 148, 591 / 592 and 1183 / 1184 tiles lie between these counts."""
    rng = np.random.default_rng(njobs)
    nx, ny, n, nchan = 43, 35, 900, 3
    ctx = api.Context(0)
    ctx.prepare_grid_kernel(api.GAUSS1D, np.array([0.05, 0.0, 0.0]), 0.15, 0.025)
    fields = []
    for k in range(min(njobs, 7)):
        lon, lat = synth.raster_scan(n, 40.0, 25.0, 0.8, 5.0, rng)
        f = ctx.field(lon, lat, rng.uniform(0.5, 1.5, n) if weights else None)
        f.set_spectra(rng.normal(1.0, 0.3, (n, nchan)).astype(np.float32))
        if engine == api.ENGINE_TC_F16:
            f.split_spectra(engine)
        fields.append(f)
    t = ctx.target_from_header(synth.sin_header(nx, ny, 40.0, 25.0, 0.7 / nx))
    want = [ctx.grid(f, t, engine=engine) for f in fields]
    cube = torch.full((njobs, nx * ny, nchan), 7.0, device="cuda")
    w = torch.full((njobs, nx * ny), 7.0, device="cuda")
    torch.cuda.synchronize()
    ctx.grid_batch([(fields[j % len(fields)], t, cube[j], w[j], api.SAMPLE_MAJOR) for j in range(njobs)])
    ctx.synchronize()
    c, wt = cube.cpu().numpy(), w.cpu().numpy()
    for j in range(njobs):
        oc, ow = want[j % len(fields)]
        np.testing.assert_array_equal(wt[j], np.asarray(ow).reshape(-1))
        np.testing.assert_allclose(c[j], np.asarray(oc).reshape(nx * ny, nchan), atol=1e-5, rtol=0)
    t.close()
    for f in fields:
        f.close()
    ctx.close()
