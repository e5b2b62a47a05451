"""Host build of the flux launches' pieces: the closed root against Newton's
iteration (same fallbacks, same root), the limiter's bit form against the
limiter, and the strips that divide a lattice among warps."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
D = C.POINTER(C.c_double)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    src = os.path.join(HERE, "hostcheck", "vah_rootcheck.cpp")
    out = str(tmp_path_factory.mktemp("rootcheck") / "libvah_rootcheck.so")
    root = os.path.dirname(HERE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I" + os.path.join(root, "include"),
                    "-I" + os.path.join(root, "gpu-vah_b200", "csrc"), src, "-o", out], check=True)
    L = C.CDLL(out)
    L.rc_limiter.restype = C.c_longlong
    return L


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_accepted_guesses_reach_the_root_and_no_other_outcome(lib, seed):
    """Where a state and guess are accepted, the iteration converges (never a
    fallback), to the closed root: v to a few ulp, which 1/(1 - v^2) <= 1e3
    makes at most 8 x 2^-53 x 1e3 of u_T, plus the iteration's stopping error
    (1e-7)^2 times its constant (up to 1.5 x 1e2 near the admitted top)."""
    out = np.zeros(5)
    lib.rc_roots(C.c_longlong(1_000_000), C.c_uint(seed), out.ctypes.data_as(D))
    assert out[0] == 0
    assert out[1] > 5e5 and out[2] > 5e4  # both outcomes are well represented
    assert out[3] < 5e-12
    assert out[4] < 1e-13


def test_limiter_bit_form_equals_the_limiter(lib):
    rng = np.random.default_rng(3)
    edge = np.array([0.0, -0.0, 1.0, -1.0, 1e-300, -1e-300, 1e30, 3.0, 2.9999999999999996, 1.1, 5e-324])
    x, y, z = (a.ravel() for a in np.meshgrid(edge, edge, edge))
    x = np.concatenate([x, rng.normal(size=200_000), rng.normal(size=200_000) * 1e-3 + 1])
    y = np.concatenate([y, rng.normal(size=200_000), rng.normal(size=200_000) * 1e-3 + 1])
    z = np.concatenate([z, rng.normal(size=200_000), rng.normal(size=200_000) * 1e-3 + 1])
    x, y, z = (np.ascontiguousarray(a) for a in (x, y, z))
    assert lib.rc_limiter(*(a.ctypes.data_as(D) for a in (x, y, z)), C.c_longlong(x.size)) == 0


@pytest.mark.parametrize("f32", [0, 1])
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 1), (9, 1, 1), (10, 3, 1), (26, 1, 1), (27, 2, 1), (28, 5, 3),
                                   (121, 7, 2), (13, 13, 13), (401, 3, 1)])
def test_x_strips_own_every_cell_once(lib, f32, shape):
    lo, hi = C.c_int(), C.c_int()
    lib.rc_x_cover(f32, *shape, C.byref(lo), C.byref(hi))
    assert (lo.value, hi.value) == (1, 1)
    w = 32 if f32 else 16
    for columns in (1, w - 1, w, w + 1, 1000):
        assert lib.rc_march_strips(f32, columns) == -(-columns // w)
