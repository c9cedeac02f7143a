"""Strongly magnified views: triangles of up to 121 candidate pixels that stay
with their lanes, and those few in sight that all go to the list, against the
oracle and between raster variants (identical bytes)."""
import copy

import numpy as np
import pytest

import oracle as O
import rvsb
from rvsb import scenes
from helpers import assert_parity, gpu_synthesize

pytestmark = pytest.mark.gpu


def _target(wl, w, h, zoom):
    t = copy.deepcopy(wl.targets[0])
    for i, (new, old) in enumerate(((w, t.width), (h, t.height))):
        t.focal[i] *= zoom * new / old
        t.principle_point[i] = new / 2.0
    t.width, t.height = w, h
    return t


def _check(ctx, wl, target, variants):
    sc = rvsb.Scene(ctx, wl.inputs)
    for i, p in enumerate(wl.planes):
        sc.upload(i, [np.ascontiguousarray(a, np.uint16) for a in p], on_device=False)
    want = O.synthesize(wl.inputs, wl.planes, target, 5.0)
    first = None
    for v in variants:
        sc.set_raster_variant(v)
        yuv, _ = gpu_synthesize(ctx, wl.inputs, wl.planes, target, 5.0, scene=sc)
        if first is None:
            first = yuv
            assert_parity(yuv, want)
        for a, b in zip(yuv, first):
            np.testing.assert_array_equal(a, b)


# More triangles in sight than the list holds: thresholds 49, 81 and 121.
@pytest.mark.parametrize("mag", [5.5, 7.5, 9.5])
def test_lanes_keep_what_the_list_cannot_hold(ctx, mag):
    wl = scenes.random_pose_small(n_views=2, w=160, h=96, seed=360)
    target = _target(wl, 2 * int(80 * mag), 2 * int(48 * mag), 1.0)
    _check(ctx, wl, target, [7, -1, 0])


# Few in sight (all listed), and at 24 again more than the list holds.
@pytest.mark.parametrize("w,h,zoom", [(160, 96, 5.0), (160, 96, 20.0), (162, 90, 60.0), (3840, 2304, 1.0)])
def test_listed_triangles_of_a_zoomed_view(ctx, w, h, zoom):
    wl = scenes.random_pose_small(n_views=2, w=160, h=96, seed=361)
    _check(ctx, wl, _target(wl, w, h, zoom), [7, 5, 3])


def test_zoomed_equirectangular_inputs(ctx):
    wl = scenes.random_pose_small(n_views=2, w=320, h=160, seed=362, erp_in=True)
    target = copy.deepcopy(wl.targets[0])
    target.focal[0] = target.focal[1] = 1200.0  # m = 23.6
    _check(ctx, wl, target, [7, 0, 6])
