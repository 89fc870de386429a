"""The quick forms of the HEALPix arithmetic against the general ones, built
for the host."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("hq") / "hostquick.so")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "hcgrid_b200", "csrc"), os.path.join(ROOT, "tests", "hostquick.cpp"), "-o", so],
                   check=True)
    L = C.CDLL(so)
    f64 = np.ctypeslib.ndpointer(np.float64, flags="C_CONTIGUOUS")
    L.hq_compare.argtypes = [C.c_uint64, C.c_long, f64, f64]
    L.hq_compare.restype = C.c_long
    return L


@pytest.mark.parametrize("nside", [1, 2, 64, 8192, 32768, 1 << 26, 1 << 28])
def test_quick_pixel_index(lib, nside):
    """Random points, ring centres and pixel corners a few ulps to either
    side, poles, the cap boundary, invalid and wrapped angles."""
    rng = np.random.default_rng(nside)
    th = [rng.uniform(0, np.pi, 60_000), np.array([0.0, np.pi, -1e-9, np.nan, 0.01, 0.02, 3.12, np.pi - 0.01])]
    ph = [rng.uniform(-7, 14, 60_000), np.zeros(8)]
    ring = rng.integers(nside, 3 * nside + 1, 20_000).astype(float)
    centre = np.arccos((2 * nside - ring) * 2 / (3 * nside))
    i = rng.integers(1, nside + 1, 20_000).astype(float)
    cap = np.arccos(1 - i * i / (3.0 * nside * nside))
    for base, step in ((centre, np.pi / (8 * nside)), (cap, np.pi / (4 * i)), (np.arccos(2 / 3) + np.zeros(20_000), 0.1)):
        for k in (-2, -1, 0, 1, 2):
            th.append(base + k * np.spacing(base))
            ph.append(step * rng.integers(0, 8 * nside, 20_000) % 6.2)
    th, ph = np.concatenate(th), np.concatenate(ph)
    assert lib.hq_compare(nside, len(th), th, ph) == 0
