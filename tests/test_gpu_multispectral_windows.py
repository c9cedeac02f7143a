"""The multispectral blur at the edges of its passes, against the oracle
(parity bar of the synthesis)."""
import pytest

import oracle as O
import rvsb
from rvsb import scenes
from helpers import assert_parity, gpu_synthesize

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(2082, 34), (34, 130), (62, 66)])
def test_multispectral_window_edges(ctx, w, h):
    """Output sizes at the edges of the blur's passes: a row longer than one
    round of the row sums (2048 columns), heights of one row more and less than
    a column segment (64 rows) and of several segments."""
    import copy
    wl = scenes.random_pose_small(n_views=2, w=64, h=36, seed=33)
    target = copy.deepcopy(wl.targets[0])
    target.focal[0] *= w / target.width
    target.focal[1] *= h / target.height
    target.width, target.height = w, h
    target.principle_point[0], target.principle_point[1] = w / 2.0, h / 2.0
    yuv, _ = gpu_synthesize(ctx, wl.inputs, wl.planes, target, 5.0, params=rvsb.params(5.0, multispectral=(1.0, 8.0)))
    O.set_multispectral(True, 1.0, 8.0)
    try:
        cpu = O.synthesize(wl.inputs, wl.planes, target, 5.0)
    finally:
        O.set_multispectral(False)
    assert_parity(yuv, cpu)
