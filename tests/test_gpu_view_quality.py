"""The views' resolved triangle qualities against the oracle's, bit for bit
wherever both resolved the same fragment (equal depth and colour)."""
import numpy as np
import pytest

import oracle as O
from rvsb import scenes
from helpers import gpu_synthesize

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("erp", [False, True], ids=["persp", "erp"])
def test_view_validity_bit_exact(ctx, erp):
    wl = scenes.random_pose_small(n_views=3, w=512, h=256, seed=360, erp_in=erp, erp_out=erp)
    target = wl.targets[0]
    _, dbg, _ = gpu_synthesize(ctx, wl.inputs, wl.planes, target, 5.0, debug=True)
    for v, (cam, (y, u, w, d)) in enumerate(zip(wl.inputs, wl.planes)):
        uv, vd, wrap = O.warp(cam, target, O.decode_depth(d, cam))
        color, depth, validity = O.raster(O.decode_color(y, u, w, cam.bit_depth_color), vd, uv, target.width,
                                          target.height, wrap)
        covered = validity > 0
        np.testing.assert_array_equal(dbg["view_validity"][v] > 0, covered)
        same = covered & (dbg["view_depth"][v] == depth) & (dbg["view_color"][v] == color).all(-1)
        assert same.sum() > 0.99 * covered.sum()
        np.testing.assert_array_equal(dbg["view_validity"][v][same], validity[same])
