"""The accumulation segments of the tensor-core kernels: an item is either whole,
of at most 1,344 staged slots, or falls into segments of at most 992, rounded up to
a chunk, none empty, whose lengths differ by a chunk at most and which cover it."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("hs") / "hostsegments.so")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "hcgrid_b200", "csrc"), os.path.join(ROOT, "tests", "hostsegments.cpp"), "-o",
                    so], check=True)
    return C.CDLL(so)


@pytest.mark.parametrize("kc", [32, 64])
def test_segments_are_short_and_equal(lib, kc):
    for n in list(range(0, 600)) + [1000, 4095, 4096, 100_000, 60_000_001]:
        nseg = lib.hs_segments(kc, n)
        if n * kc <= 1344:
            assert nseg == 1
        else:
            assert nseg >= 2
        qs = range(nseg) if nseg < 1000 else [0, 1, nseg // 2, nseg - 2, nseg - 1]
        size = []
        for q in qs:
            begin = lib.hs_end(n, nseg, q - 1) if q else 0
            size.append(lib.hs_end(n, nseg, q) - begin)
        assert nseg == 1 or (min(size) >= 1 and max(size) - min(size) <= 1 and (max(size) - 1) * kc < 992)
        assert lib.hs_end(n, nseg, nseg - 1) == n
