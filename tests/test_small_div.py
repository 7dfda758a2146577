"""The gather's quotients by a float reciprocal (rows of a box of sub-cells from
list positions) at sizes up to the largest grid's, for every reciprocal within 2
ulp of 1 / d, which is what the device's may be."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-photon-mapping_b200", "csrc")
SHIM = r"""
#include <cmath>
#include <cstdint>
#include "pm_div.h"
// the first u in [first, last) at which small_div is not u / d; -1: none
extern "C" int64_t first_wrong(int64_t first, int64_t last, int d, int ulps) {
    float inv = 1.0f / (float)d;
    for (int i = 0; i < std::abs(ulps); i++) inv = std::nextafter(inv, ulps > 0 ? 2.0f : 0.0f);
    for (int64_t u = first; u < last; u++)
        if (pm::small_div((int)u, d, inv) != (int)(u / d)) return u;
    return -1;
}
"""


@pytest.fixture(scope="module")
def first_wrong(tmp_path_factory):
    d = tmp_path_factory.mktemp("div")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "s.so"),
                    str(d / "shim.cpp")], check=True)
    f = ctypes.CDLL(str(d / "s.so")).first_wrong
    f.restype, f.argtypes = ctypes.c_int64, [ctypes.c_int64, ctypes.c_int64, ctypes.c_int, ctypes.c_int]
    return f


@pytest.mark.parametrize("d", [1, 2, 3, 5, 7, 13, 220, 4099])
@pytest.mark.parametrize("ulps", [-2, -1, 0, 1, 2])
def test_quotients(first_wrong, d, ulps):
    for first in (0, 1 << 21, (1 << 24) - 5000, 3 * 5_000_000, 1 << 28, (1 << 30) - 400_000):
        assert first_wrong(first, first + 400_000, d, ulps) == -1, first
