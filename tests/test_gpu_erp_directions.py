"""Radius, atan2 and asin of the equirectangular projector against the oracle's
correctly rounded values, bit for bit: 131,072 directions of a room in general
position, and an output camera at and in line with the input's (directions
with a zero component, on the axes and at the poles)."""
import numpy as np
import pytest

import oracle as O
import rvsb
from rvsb import abi, scenes
from helpers import gpu_synthesize

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("moved", [True, False], ids=["general", "in_place"])
def test_warped_directions_bit_exact(ctx, moved):
    wl = scenes.random_pose_small(n_views=1, w=512, h=256, seed=401, erp_in=True, erp_out=True)
    cam, target = wl.inputs[0], wl.targets[0]
    if not moved:
        target = abi.make_camera(abi.EQUIRECTANGULAR, 512, 256, tuple(cam.position), (0, 0, 0), (0.3, 20.0))
    _, dbg, _ = gpu_synthesize(ctx, wl.inputs, wl.planes, target, 5.0, debug=True)
    uv, depth, _ = O.warp(cam, target, O.decode_depth(wl.planes[0][3], cam))
    got = dbg["warped"][0]
    np.testing.assert_array_equal(got[..., 0], uv[..., 0])
    np.testing.assert_array_equal(got[..., 1], uv[..., 1])
    np.testing.assert_array_equal(got[..., 2], depth)
