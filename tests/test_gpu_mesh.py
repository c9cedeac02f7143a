"""The mesh kernel at the edges of its strips (31 quads) and row counts, and
the list of large triangles when it overflows, against the oracle (parity bar
of the synthesis) and between raster variants (identical bytes)."""
import copy

import numpy as np
import pytest

import oracle as O
import rvsb
from rvsb import scenes
from helpers import assert_parity, gpu_synthesize

pytestmark = pytest.mark.gpu


def _resized(target, w, h):
    t = copy.deepcopy(target)
    for i, (new, old) in enumerate(((w, target.width), (h, target.height))):
        t.focal[i] *= new / old
        t.principle_point[i] = new / 2.0
    t.width, t.height = w, h
    return t


def _each_variant(ctx, wl, target, variants):
    sc = rvsb.Scene(ctx, wl.inputs)
    for i, p in enumerate(wl.planes):
        sc.upload(i, [np.ascontiguousarray(a, np.uint16) for a in p], on_device=False)
    out = []
    for v in variants:
        sc.set_raster_variant(v)
        yuv, _ = gpu_synthesize(ctx, wl.inputs, wl.planes, target, 5.0, scene=sc)
        out.append(yuv)
    for yuv in out[1:]:
        for a, b in zip(yuv, out[0]):
            np.testing.assert_array_equal(a, b)
    return out[0]


# Widths of 1 quad, one strip of 31 and one quad more or less, and two strips;
# heights of 1 quad row and around 4, 8 and 32 rows.
@pytest.mark.parametrize("w,h", [(2, 2), (2, 34), (30, 4), (32, 6), (34, 10), (62, 32), (64, 34), (66, 66)])
def test_strip_and_row_edges(ctx, w, h):
    wl = scenes.random_pose_small(n_views=2, w=w, h=h, seed=300 + w + h)
    target = _resized(wl.targets[0], 64, 36)
    yuv = _each_variant(ctx, wl, target, [-1, 0, 3, 5, 6])
    assert_parity(yuv, O.synthesize(wl.inputs, wl.planes, target, 5.0))


@pytest.mark.parametrize("erp_in", [False, True], ids=["persp", "erp_culled"])
def test_large_triangle_list_overflow(ctx, erp_in):
    """More large triangles than the list of 16384 holds: 48,000 of 2 x 128x96
    inputs magnified 3 times with a threshold of 4 candidates (variant 0)
    against the 16-candidate threshold whose lanes keep them (variant 7); and
    the visible part of 2 x 320x160 equirectangular inputs magnified 6 times,
    whose tiles outside the view are culled."""
    if erp_in:
        wl = scenes.random_pose_small(n_views=2, w=320, h=160, seed=311, erp_in=True)
        target = _resized(wl.targets[0], 640, 480)
        target.focal[0] = target.focal[1] = 320.0
    else:
        wl = scenes.random_pose_small(n_views=2, w=128, h=96, seed=310)
        target = _resized(wl.targets[0], 384, 288)
    yuv = _each_variant(ctx, wl, target, [0, 7])
    assert_parity(yuv, O.synthesize(wl.inputs, wl.planes, target, 5.0))


# Thresholds of magnified views: 16, 36, 49 and 400 candidates (the largest).
@pytest.mark.parametrize("mag", [1.5, 4, 5.5, 24])
@pytest.mark.parametrize("erp", [False, True], ids=["persp", "erp"])
def test_threshold_follows_magnification(ctx, erp, mag):
    """Every triangle in its lane (variant 7) against nearly every one in the
    list or, when that overflows, taken from the mesh (variant 0), and the
    oracle."""
    wl = scenes.random_pose_small(n_views=2, w=64, h=32, seed=330, erp_in=erp, erp_out=erp)
    if erp:
        target = copy.deepcopy(wl.targets[0])
        target.width, target.height = int(64 * mag), int(32 * mag)
    else:
        target = _resized(wl.targets[0], int(64 * mag), int(32 * mag))
    yuv = _each_variant(ctx, wl, target, [7, 0])
    assert_parity(yuv, O.synthesize(wl.inputs, wl.planes, target, 5.0))


@pytest.mark.parametrize("precision", [1.0, 1.5])
@pytest.mark.parametrize("erp_out", [False, True], ids=["persp_out", "erp_out"])
@pytest.mark.parametrize("inputs", ["erp", "mixed"])
def test_projection_mixtures(ctx, inputs, erp_out, precision):
    """The instantiations of the mesh kernel by what a launch holds:
    equirectangular inputs alone and beside a perspective one, both kinds of
    output, with and without Precision."""
    wl = scenes.random_pose_small(n_views=2, w=128, h=64, seed=320, erp_in=True, erp_out=erp_out)
    if inputs == "mixed":
        flat = scenes.random_pose_small(n_views=1, w=96, h=54, seed=321)
        wl.inputs.append(flat.inputs[0])
        wl._planes = list(wl.planes[:2]) + [flat.planes[0]]
    p = rvsb.params(5.0, precision=precision)
    yuv, _ = gpu_synthesize(ctx, wl.inputs, wl.planes, wl.targets[0], 5.0, params=p)
    O.set_precision(precision)
    try:
        cpu = O.synthesize(wl.inputs, wl.planes, wl.targets[0], 5.0)
    finally:
        O.set_precision(1.0)
    assert_parity(yuv, cpu)
