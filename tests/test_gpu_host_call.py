"""rvsb_synthesize_host, whose mesh kernels run before the colour planes have
arrived, against the resident scene's call on the same inputs, bit for bit:
one to seven views (more than one group of views), planes that change from
call to call, outputs that grow and shrink, an error in between."""
import copy

import numpy as np
import pytest
import torch

import rvsb
from rvsb import scenes
from helpers import gpu_synthesize

pytestmark = pytest.mark.gpu


def _host_call(ctx, wl, planes, target, p, pinned, stream=None):
    make = lambda n: torch.zeros(n, dtype=torch.int16)
    w, h = target.width, target.height
    out = [make(n) for n in (w * h, w * h // 4, w * h // 4)]
    host = [[torch.from_numpy(np.ascontiguousarray(a, np.uint16).view(np.int16).reshape(-1)) for a in v] for v in planes]
    if pinned:
        out, host = [t.pin_memory() for t in out], [[t.pin_memory() for t in v] for v in host]
    ctx.synthesize_host(wl.inputs, host, target, p, out, stream)
    shapes = ((h, w), (h // 2, w // 2), (h // 2, w // 2))
    return [t.numpy().view(np.uint16).reshape(s) for t, s in zip(out, shapes)]


def _changed(planes, k):
    """The k-th frame: luma and chroma shifted, the views' depth mirrored every other time."""
    out = []
    for y, u, v, d in planes:
        shift = lambda a: ((a.astype(np.int32) + 37 * k) % 1024).astype(np.uint16)
        out.append((shift(y), shift(u), shift(v), d[:, ::-1] if k % 2 else d))
    return out


@pytest.mark.parametrize("pinned", [True, False], ids=["pinned", "pageable"])
@pytest.mark.parametrize("views,erp", [(1, False), (4, False), (5, False), (7, False), (5, True)])
def test_host_call_equals_the_resident_scene(ctx, views, erp, pinned):
    wl = scenes.random_pose_small(n_views=views, w=192, h=96, seed=370 + views, erp_in=erp)
    p = rvsb.params(5.0)
    stream = torch.cuda.Stream()
    for k, scale in enumerate((1, 2, 1, 3)):
        target = copy.deepcopy(wl.targets[0])
        target.width, target.height = 192 * scale, 96 * scale
        for i in range(2):
            target.focal[i] *= scale
            target.principle_point[i] *= scale
        planes = _changed(wl.planes, k)
        got = _host_call(ctx, wl, planes, target, p, pinned, stream if k % 2 else None)
        want, _ = gpu_synthesize(ctx, wl.inputs, planes, target, 5.0)
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)
        if k == 1:  # refused after the depth planes have gone up
            with pytest.raises(rvsb.RvsbError):
                _host_call(ctx, wl, _changed(wl.planes, 9), target, rvsb.params(0.0), pinned)
