"""The candidate span of a row of a large triangle (row_span,
device_common.cuh) on the host: it holds every pixel the coverage test
accepts.  The test's third coordinate is a difference of products that cancel
on long thin triangles, so its rounding, not the third edge's own size, says
how far beyond that edge a pixel can still pass."""
import ctypes

import numpy as np
import pytest

import device_host

CODE = """
#include "device_common.cuh"
using namespace rvsb;
using namespace rvsb::dev;
extern "C" void approximations_off_by(int ulp) { g_ulp = ulp; }
// Of n triangles (three (x, y) each) over a w x h output: covered pixels the
// spans leave out, covered pixels looked at; the first triangle with a miss.
extern "C" void spans(const float* tri, long n, int w, int h, long* missed, long* covered_n, long* first) {
    for (long k = 0; k < n; ++k) {
        const float* t = tri + 6 * k;
        const float4 A = make_float4(t[0], t[1], 1.f, 0.f), B = make_float4(t[2], t[3], 1.f, 0.f),
                     C = make_float4(t[4], t[5], 1.f, 0.f);
        TriSetup s;
        if (!tri_coef(A, B, C, s) || !tri_range(A, B, C, w, h, 0, w - 1, 0, h - 1, s)) continue;
        const long before = *missed;
        for (int y = s.y0; y <= s.y1; ++y) {
            int xl, xr;
            row_span(s, C.x, C.y, y, xl, xr);
            if (xl < s.x0 || xr > s.x1) *missed += 1000000;
            // A row's covered pixels lie together: near the edges' crossings
            // of the row, and next to the span if they reach beyond it.
            auto test = [&](double from, double to) {
                const int c0 = (int)std::max((double)s.x0, from), c1 = (int)std::min((double)s.x1, to);
                for (int x = c0; x <= c1; ++x) {
                    float l1, l2, l3;
                    barycentric(s, C.x, C.y, x, y, l1, l2, l3);
                    if (!covered(l1, l2, l3)) continue;
                    ++*covered_n;
                    if (x < xl || x > xr) ++*missed;
                }
            };
            const float* v[4] = {t, t + 2, t + 4, t};
            for (int e = 0; e < 3; ++e) {
                const double ya = v[e][1], yb = v[e + 1][1], f = ya == yb ? 0.5 : (y + 0.5 - ya) / (yb - ya);
                const double c = v[e][0] + std::min(1.0, std::max(0.0, f)) * ((double)v[e + 1][0] - v[e][0]);
                test(c - 40, c + 40);
            }
            if (xl > xr) continue;
            test(xl - 64.0, xl - 1.0);
            test(xr + 1.0, xr + 64.0);
        }
        if (*missed > before && *first < 0) *first = k;
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return device_host.build(str(tmp_path_factory.mktemp("span")), CODE)


def _spans(lib, tri, w, h):
    tri = np.ascontiguousarray(tri, np.float32).reshape(-1, 6)
    r = [ctypes.c_long(0), ctypes.c_long(0), ctypes.c_long(-1)]
    lib.spans(tri.ctypes.data_as(ctypes.c_void_p), ctypes.c_long(len(tri)), w, h, *[ctypes.byref(v) for v in r])
    missed, covered, first = [v.value for v in r]
    return missed, covered, tri[first].tolist() if first >= 0 else None


def test_the_pixel_on_a_short_edge(lib):
    """Barycentric (0.486, 0.514, 0.0) at pixel (1076, 1377)."""
    lib.approximations_off_by(0)
    tri = [1076.357666, 1377.454834, 1076.642578, 1377.548950, 1337.751831, 1582.264038]
    missed, covered, _ = _spans(lib, tri, 2048, 2048)
    assert covered > 0 and missed == 0


@pytest.mark.parametrize("ulp", [0, 2])
@pytest.mark.parametrize("lo,hi,n", [(20, 100, 20000), (100, 400, 10000), (400, 1000, 5000), (1000, 2000, 3000),
                                     (2000, 16000, 600)])
def test_thin_triangles(lib, lo, hi, n, ulp):
    """Triangles lo to hi pixels long with a side of 0.3 to 2 pixels, the
    short side between each pair of vertices in turn, anywhere in an output of
    up to 16384 pixels and at any angle; half of them with the short side laid
    through a pixel centre, where covered pixels lie on it."""
    lib.approximations_off_by(ulp)
    rng = np.random.default_rng(lo + ulp)
    size = 16384
    length, side = np.exp(rng.uniform(np.log(lo), np.log(hi), n)), rng.uniform(0.3, 2.0, n)
    a, b = rng.uniform(0, 2 * np.pi, n), rng.uniform(0, 2 * np.pi, n)
    p = rng.uniform(0, size, (n, 2))
    p[::2] = np.floor(p[::2]) + 0.5
    e = np.stack([np.cos(b), np.sin(b)], -1) * side[:, None]
    t = rng.uniform(0, 1, (n, 1))
    u, v = p - t * e, p + (1 - t) * e
    far = p + np.stack([np.cos(a), np.sin(a)], -1) * length[:, None]
    tri = np.stack([u, v, far], 1)
    # Front-facing (positive determinant), then the vertices rotated.
    d = (tri[:, 1, 1] - tri[:, 2, 1]) * (tri[:, 0, 0] - tri[:, 2, 0]) + \
        (tri[:, 2, 0] - tri[:, 1, 0]) * (tri[:, 0, 1] - tri[:, 2, 1])
    tri[d < 0] = tri[d < 0][:, [1, 0, 2]]
    turn = (np.arange(n) // 2) % 3
    tri = np.stack([tri[np.arange(n), (k + turn) % 3] for k in range(3)], 1)
    missed, covered, first = _spans(lib, tri, size, size)
    assert covered > n and missed == 0, (missed, covered, first)


@pytest.mark.parametrize("ulp", [0, 2])
def test_vertices_far_outside(lib, ulp):
    """Triangles with vertices up to 10^4, 10^5 and 10^6 pixels outside."""
    lib.approximations_off_by(ulp)
    rng = np.random.default_rng(77 + ulp)
    tri = rng.uniform(-1, 1, (900, 3, 2)) * (10.0 ** rng.integers(4, 7, (900, 1, 1)))
    tri[:, 0] = rng.uniform(0, 1024, (900, 2))
    tri[::2, 1] = tri[::2, 0] + rng.uniform(-3, 3, (450, 2))
    tri = np.concatenate([tri, tri[:, [1, 2, 0]], tri[:, [0, 2, 1]], tri[:, [2, 1, 0]]])
    missed, covered, first = _spans(lib, tri, 1024, 1024)
    assert covered > 100_000 and missed == 0, (missed, covered, first)
