"""The triangle quality of the resolve (tri_quality_fast, resolve.cuh) on the
host: bit for bit the double evaluation (tri_quality, cv::norm's), also where
the longest edge lies next to a rounding boundary of its root, where two edges
tie, and for extreme coordinates."""
import ctypes

import numpy as np
import pytest

import device_host

CODE = """
#include "resolve.cuh"
using namespace rvsb::dev;
extern "C" void approximations_off_by(int ulp) { g_ulp = ulp; }
extern "C" void qualities(const float* tri, long n, float precision, float* fast, float* exact) {
    for (long k = 0; k < n; ++k) {
        const float* t = tri + 6 * k;
        const float4 A = make_float4(t[0], t[1], 1.f, 0.f), B = make_float4(t[2], t[3], 1.f, 0.f),
                     C = make_float4(t[4], t[5], 1.f, 0.f);
        fast[k] = tri_quality_fast(A, B, C, precision);
        exact[k] = tri_quality(t[0], t[1], t[2], t[3], t[4], t[5], precision);
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return device_host.build(str(tmp_path_factory.mktemp("quality")), CODE)


def _compare(lib, tri, precision=1.0):
    tri = np.ascontiguousarray(tri, np.float32).reshape(-1, 6)
    fast, exact = np.empty(len(tri), np.float32), np.empty(len(tri), np.float32)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    lib.qualities(p(tri), ctypes.c_long(len(tri)), ctypes.c_float(precision), p(fast), p(exact))
    np.testing.assert_array_equal(fast.view(np.uint32), exact.view(np.uint32))
    return exact


def _near_boundaries(rng, scale):
    """Edges (dx, dy) whose length lies within 2^-16 of the spacing of floats
    from the middle between two floats."""
    out = []
    for _ in range(8):
        d = rng.uniform(-scale, scale, (4_000_000, 2)).astype(np.float32)
        length = np.hypot(d[:, 0].astype(np.float64), d[:, 1].astype(np.float64))
        near = length.astype(np.float32).astype(np.float64)
        off = np.abs(length - near) / np.spacing(near.astype(np.float32)).astype(np.float64)
        out.append(d[np.abs(off - 0.5) < 2.0 ** -16])
    return np.concatenate(out)


@pytest.mark.parametrize("ulp", [0, 1])
@pytest.mark.parametrize("precision", [1.0, 1.5])
@pytest.mark.parametrize("scale", [1.0, 9.0])
def test_roots_next_to_rounding_boundaries(lib, scale, precision, ulp):
    """An edge from the origin of such a length (the subtraction is exact),
    the third vertex near its middle."""
    lib.approximations_off_by(ulp)
    d = _near_boundaries(np.random.default_rng(int(scale)), scale)
    assert len(d) > 500
    tri = np.zeros((len(d), 3, 2), np.float32)
    tri[:, 1] = d
    tri[:, 2] = d * np.float32(0.5) + np.float32(0.01)
    quality = _compare(lib, tri, precision)
    assert (quality > 1.0).mean() > 0.6


@pytest.mark.parametrize("ulp", [0, 1])
def test_random_and_degenerate_triangles(lib, ulp):
    lib.approximations_off_by(ulp)
    rng = np.random.default_rng(61)
    tri = rng.uniform(0, 2000, (500_000, 1, 2)) + rng.uniform(-4, 4, (500_000, 3, 2))
    tri[::5, 1] = tri[::5, 0]                                # no third edge
    tri[1::5, 2] = 2 * tri[1::5, 0] - tri[1::5, 1]           # two edges tie
    tri[2::5] = np.rint(tri[2::5])                           # right triangles, exact lengths
    _compare(lib, tri)


def test_extreme_coordinates(lib):
    lib.approximations_off_by(0)
    v = np.array([0.0, 1e-40, 1e-20, 1e-7, 1.0, 5.0, 1e4, 1e10, 1e19, 3e19, 3e38, np.inf, np.nan], np.float32)
    v = np.concatenate([v, -v])
    p = np.stack(np.meshgrid(v, v, indexing="ij"), -1).reshape(-1, 2)
    rng = np.random.default_rng(62)
    with np.errstate(all="ignore"):
        _compare(lib, p[rng.integers(0, len(p), (300_000, 3))])
