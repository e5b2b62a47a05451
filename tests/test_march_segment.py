"""The length of a march's segments: the cheapest of every division, priced in
about sqrt(n) evaluations (each sums over a batch's events at every admission)."""
import ctypes as C
import math
import os
import subprocess

import pytest

import vahlib as V

CUDA_INCLUDE = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("segmentcheck") / "libvah_segmentcheck.so")
    csrc = os.path.join(V.ROOT, "gpu-vah_b200", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I" + os.path.join(V.ROOT, "include"), "-I" + csrc,
                    "-I" + CUDA_INCLUDE, os.path.join(V.ROOT, "tests", "hostcheck", "vah_segmentcheck.cpp"), "-o", out],
                   check=True)
    return C.CDLL(out)


@pytest.mark.parametrize("minb", [4, 5])
@pytest.mark.parametrize("strips", [1, 3, 26, 148, 937, 10_000, 250_000])
def test_segment_is_the_cheapest_division(lib, minb, strips):
    calls = C.c_int()
    for n in list(range(1, 140)) + [255, 256, 257, 400, 401, 1023, 4099, 20_000]:
        got = lib.sc_segment(n, minb, C.c_longlong(strips), C.byref(calls))
        assert got == lib.sc_search(n, minb, C.c_longlong(strips)), n
        assert calls.value <= 2 * math.sqrt(n) + 1, n
