"""The arctangent table of the equirectangular projector (erp_trig.cuh) on the
host: no direction reads outside it, whatever the approximate reciprocal makes
of it, and the float results are the correctly rounded ones."""
import ctypes

import numpy as np
import pytest

import device_host

CODE = """
#include "erp_trig.cuh"
using namespace rvsb::dev;
extern "C" int directions(const float* xyz, long n, float* out) {
    g_table = kAtan64;
    g_table_bytes = sizeof(kAtan64);
    g_bad_loads = 0;
    for (long k = 0; k < n; ++k) {
        erp_direction(xyz[3 * k], xyz[3 * k + 1], xyz[3 * k + 2], out[3 * k], out[3 * k + 1], out[3 * k + 2]);
    }
    return g_bad_loads;
}
extern "C" void exact(const float* xyz, long n, float* out) {
    for (long k = 0; k < n; ++k)
        erp_direction_exact(xyz[3 * k], xyz[3 * k + 1], xyz[3 * k + 2], out[3 * k], out[3 * k + 1], out[3 * k + 2]);
}
extern "C" void approximations_off_by(int ulp) { g_ulp = ulp; }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return device_host.build(str(tmp_path_factory.mktemp("erp")), CODE)


def _run(lib, xyz):
    xyz = np.ascontiguousarray(xyz, np.float32)
    got, want = np.empty_like(xyz), np.empty_like(xyz)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    bad = lib.directions(p(xyz), ctypes.c_long(len(xyz)), p(got))
    lib.exact(p(xyz), ctypes.c_long(len(xyz)), p(want))
    return bad, got, want


def _extremes():
    """Every triple of zeros, subnormals, the smallest and largest normals,
    ones, infinities and NaN, of either sign."""
    tiny = np.finfo(np.float32).tiny
    v = [0.0, 1e-45, 3e-42, tiny / 2, tiny, 1e-30, 1e-15, 1.0, 1e15, 3e38, np.inf]
    v = np.array(v + [-x for x in v] + [np.nan], np.float32)
    return np.stack(np.meshgrid(v, v, v, indexing="ij"), -1).reshape(-1, 3)


@pytest.mark.parametrize("ulp", [0, 1])
def test_extreme_directions_stay_in_the_table(lib, ulp):
    lib.approximations_off_by(ulp)
    bad, got, want = _run(lib, _extremes())
    assert bad == 0
    np.testing.assert_array_equal(got.view(np.uint32)[~np.isnan(want)], want.view(np.uint32)[~np.isnan(want)])
    assert np.isnan(got[np.isnan(want)]).all()


@pytest.mark.parametrize("ulp", [0, 1])
def test_random_directions_are_correctly_rounded(lib, ulp):
    """A million directions, a third of them near an axis or a plane, with the
    approximations exact and up to one ulp off."""
    lib.approximations_off_by(ulp)
    rng = np.random.default_rng(510 + ulp)
    xyz = rng.normal(size=(1_000_000, 3)) * np.exp(rng.uniform(-6, 6, size=(1_000_000, 1)))
    xyz[::3] *= 10.0 ** -rng.integers(0, 8, size=(len(xyz[::3]), 3))
    bad, got, want = _run(lib, xyz)
    assert bad == 0
    np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
