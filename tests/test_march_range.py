"""The sample range that type 4 interpolates without clamps (inside_range,
march_range.cuh), compiled for the host: every sample of the range has all
eight voxels in the image, axes of one voxel have no range, marches of millions
of samples that drift out along a nearly constant axis have none either, and
ordinary axes keep every sample that is clear of the faces."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "omega_b200", "csrc")
SOURCE = """
#include "march_range.cuh"
extern "C" void ranges(const float *c, const float *s, const unsigned *count, const int *size, int n, float *lo,
                       float *hi) {
    for (int i = 0; i < n; ++i) {
        lo[i] = 0.f;
        hi[i] = 3.4e38f;
        omb::inside_range(c[i], s[i], count[i], size[i], lo[i], hi[i]);
    }
}
extern "C" void interior(float lo, float hi, unsigned n, unsigned *out) { omb::interior(lo, hi, n, out[0], out[1]); }
"""


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    d = tmp_path_factory.mktemp("march")
    (d / "r.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-x", "c++", "-I", CSRC, str(d / "r.cpp"),
                    "-o", str(d / "r.so")], check=True)
    return ctypes.CDLL(str(d / "r.so"))


@pytest.fixture(scope="module")
def ranges(library):
    fn = library.ranges
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731

    def call(c, s, size, count=2000):
        c, s, size, count = np.broadcast_arrays(np.float32(c), np.float32(s), np.int32(size), np.uint32(count))
        c, s, size, count = (np.ascontiguousarray(a) for a in (c, s, size, count))
        lo, hi = np.empty(c.size, np.float32), np.empty(c.size, np.float32)
        fn(ptr(c), ptr(s), ptr(count), ptr(size), c.size, ptr(lo), ptr(hi))
        return c, s, size, lo, hi
    return call


def _at(i, s, c):
    """fmaf(i, s, c): one rounding."""
    return (i.astype(np.float64) * np.float64(s) + np.float64(c)).astype(np.float32)


@pytest.mark.parametrize("size", [1, 2, 3, 15, 200])
def test_every_sample_of_the_range_is_inside(ranges, size):
    rng = np.random.default_rng(size)
    n = 4000
    c = rng.uniform(-0.5, size - 0.5, n)
    s = rng.uniform(-1, 1, n) * 10.0 ** rng.uniform(-4, 0, n)
    s[:50] = 0.0
    c[:25] = (size - 1) / 2   # along the middle of the axis
    for ci, si, _, lo, hi in zip(*ranges(c, s, size)):
        i = np.arange(max(lo, 0.0), min(hi, 1999.0) + 1, dtype=np.float32)
        x = _at(i, si, ci)
        assert np.all((x >= 0) & (np.floor(x) + 1 <= size - 1)), (ci, si, lo, hi)


def test_one_voxel_has_no_range(ranges):
    """Two rings, one 8 mm slice, a ray from z = -2 to 2: samples within 0.01
    voxels of the slice's middle."""
    _, _, _, lo, hi = ranges([-0.25, 0.25, 0.0, 0.0], [0.5 / 64, -0.5 / 64, 0.0, 1e-3], 1)
    assert np.all(hi < lo)


def test_ordinary_axes_keep_their_samples(ranges):
    c, s = np.float32(-0.4), np.float32(0.73)
    _, _, _, lo, hi = ranges(c, s, 128)
    i = np.arange(200, dtype=np.float32)
    x = _at(i, s, c)
    clear = i[(x > 0.02) & (x < 127 - 0.02)]
    assert lo[0] <= clear[0] and hi[0] >= clear[-1]


@pytest.mark.parametrize("count", [1000, 600_000, 1_000_000, 20_000_000, 4_000_000_000])
def test_long_marches_along_a_nearly_constant_axis(ranges, count):
    """Steps on both sides of the 1e-6 below which an axis counts as constant:
    the range's first and last sample are inside (samples between them are)."""
    rng = np.random.default_rng(count % 1000)
    size = 15
    c = rng.uniform(-0.5, size - 0.5, 2000)
    s = np.clip(rng.uniform(-size, size, 2000) / count, -1.5e-6, 1.5e-6)
    _, s, _, lo, hi = ranges(c, s, size, count)
    some = (lo <= hi) & (lo < count)
    assert some.any()
    for at in (lo, np.minimum(hi, np.float32(count - 1))):
        x = _at(at, s, c.astype(np.float32))[some]
        assert np.all((x >= 0) & (np.floor(x) + 1 <= size - 1))


@pytest.mark.parametrize("lo,hi,n,first,last", [
    (3, 7, 20, 3, 8), (3, 50, 20, 3, 20), (0, 3.4e38, 20, 0, 20), (25, 30, 20, 20, 20), (7, 3, 20, 20, 20),
    (0, -1, 20, 20, 20), (3e38, 3.4e38, 20, 20, 20), (3e7, 4e7, 2 ** 24 + 3, 2 ** 24 + 3, 2 ** 24 + 3),
    (0, 3.4e38, 3_999_999_999, 0, 3_999_999_999)])
def test_sample_counts_stay_within_the_march(library, lo, hi, n, first, last):
    out = (ctypes.c_uint * 2)()
    library.interior(ctypes.c_float(lo), ctypes.c_float(hi), ctypes.c_uint(n), out)
    assert (out[0], out[1]) == (first, last)
