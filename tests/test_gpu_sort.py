"""The device sort at the sizes where its form changes: one block, tiles of
1,024 and 4,096 keys, 64-bit keys (fields over most of the sky), few and many
equal keys. Keys, permutation and ring table equal the oracle's exactly."""
import numpy as np
import pytest

from hcgrid_b200 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 1025, 16384, 16385, (1 << 20) - 1, 1 << 20, (1 << 20) + 4097])
@pytest.mark.parametrize("spread", ["field", "point", "sky"])
def test_sort_equals_oracle(n, spread):
    if n > 20000 and spread == "sky":
        n = min(n, 200_001)
    rng = np.random.default_rng(n)
    if spread == "field":
        lon, lat = rng.uniform(29.0, 31.0, n), rng.uniform(39.0, 41.0, n)
        lon[n // 2:] = lon[: n - n // 2]  # equal keys far apart in input order
        lat[n // 2:] = lat[: n - n // 2]
    elif spread == "point":
        lon, lat = np.full(n, 30.0), np.full(n, 40.0)
    else:
        lon, lat = rng.uniform(0.0, 360.0, n), np.degrees(np.arcsin(rng.uniform(-1.0, 1.0, n)))
    sigma = (60.0 if spread != "sky" else 6.0) / 3600.0 / 2.3548  # 6": nside 2^17, 38-bit keys
    ctx = api.Context(0)
    ctx.prepare_grid_kernel(api.GAUSS1D, np.array([sigma, 0.0, 0.0]), 3 * sigma, sigma / 2)
    f = ctx.field(lon, lat)
    keys, perm, lut, first, used = f.sorted()
    ps = O.presort(O.prepare_grid_kernel(sigma, 3 * sigma, sigma / 2).hpx, lon, lat)
    assert np.array_equal(keys, ps.keys) and np.array_equal(perm, ps.perm) and np.array_equal(lut, ps.lut)
    f.close()
    ctx.close()
