"""The tap records' Bessel factors on float pairs (csrc/kb_series.cuh), built for
the host: where the pair is taken, its float is the one that the FP64 form rounds
to, and the distances where 46 bits cannot decide that are left to FP64."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
from scipy.special import ive

from conftest import ROOT

SHAPES = [(4.0, 0.0), (4.0, 0.5), (3.0, 5.0), (4.0, 8.9962), (4.25, 14.9086), (4.9, 18.5)]


@pytest.fixture(scope="module")
def factors(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("kb") / "kb_series.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-w", "-shared", "-fPIC",
                    "-I", os.path.join(ROOT, "4d_lung_gb300", "csrc"), "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "drivers", "kb_series.cpp"), "-o", out], check=True)
    f = C.CDLL(out).kb_factors
    f.argtypes = [C.c_float, C.c_float, C.c_int, C.c_int, C.c_long] + [C.c_void_p] * 3

    def run(w, b, grid, slope, q):
        v, sure = np.empty(len(q), np.float32), np.empty(len(q), np.uint8)
        nd = f(w, b, grid, slope, len(q), q.ctypes.data, v.ctypes.data, sure.ctypes.data)
        return nd, v, sure.astype(bool)
    return run


def fp64(w, b, grid, slope, q):
    w, b = np.float32(w), float(np.float32(b))
    dk = np.float32(1.0 / float(np.float32(grid - 1)))
    scale = float(np.float32(100) * w * dk)
    q = q.astype(np.float64)
    s = np.sqrt(1.0 - q * q)
    if not slope:
        return ive(0, b * s) * np.exp(b * s) / scale
    i1s = np.where(s > 1e-12, ive(1, b * s) * np.exp(b * s) / np.maximum(s, 1e-300), 0.5 * b)
    return i1s * b * q * (2.0 / (float(w) * float(dk))) / scale


def distances():
    rng = np.random.default_rng(3)
    ends = np.float32([0.0, 1e-30, 1e-7, 0.5, 1.0, np.nextafter(np.float32(1), np.float32(0))])
    return np.concatenate([ends, rng.uniform(0, 1, 300000).astype(np.float32),
                           (10.0 ** rng.uniform(-8, 0, 50000)).astype(np.float32),
                           (1 - 10.0 ** rng.uniform(-7, 0, 50000)).astype(np.float32)])


@pytest.mark.parametrize("w,b", SHAPES)
@pytest.mark.parametrize("grid", [32, 256])
@pytest.mark.parametrize("slope", [0, 1])
def test_pairs_round_as_fp64_does(factors, w, b, grid, slope):
    """A pair that is taken rounds to the nearest float of the FP64 value; 2^-20
    of an ulp is FP64's own part.  The distances left to FP64 are some 1 in 10^5
    (2^-41 against the half ulp); 10^-3 leaves room for chance."""
    q = distances()
    nd, v, sure = factors(w, b, grid, slope, q)
    if nd == 0:
        pytest.skip("no series for this shape")
    r = fp64(w, b, grid, slope, q)
    ulp = np.spacing(np.abs(v)).astype(np.float64)
    # below a power of two the spacing is half as wide
    down = np.abs(np.abs(v) - np.nextafter(np.abs(v), np.float32(0))).astype(np.float64)
    half = np.where(r < v, down, ulp) / 2
    assert (np.abs(r - v)[sure] <= (half * (1 + 2.0 ** -20))[sure]).all()
    assert (~sure).mean() < 1e-3


# distances at which the pair's float is not the one of the FP64 form
HARD = [(4.0, 0.5, 64, 0, "0x1.af0de2p-1"), (4.25, 14.9086, 256, 0, "0x1.ed4c32p-1"),
        (4.25, 14.9086, 256, 1, "0x1.1fb29p-5"), (4.0, 8.9962, 256, 0, "0x1.066e3ep-2"),
        (4.0, 8.9962, 256, 1, "0x1.fca504p-7")]


@pytest.mark.parametrize("w,b,grid,slope,q", HARD)
def test_near_ties_are_left_to_fp64(factors, w, b, grid, slope, q):
    q = np.float32([float.fromhex(q)])
    _, v, sure = factors(w, b, grid, slope, q)
    assert v[0] != np.float32(fp64(w, b, grid, slope, q)[0])
    assert not sure[0]
