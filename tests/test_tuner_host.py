"""The raster autotuner's choices on a fake runtime (every launch takes the same
time there, so the tuner keeps the untuned default)."""
import numpy as np
import pytest

import fake_cuda
import rvsb
from rvsb import abi


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    return fake_cuda.build(str(tmp_path_factory.mktemp("fake")))


@pytest.fixture
def fake(library, monkeypatch):
    return fake_cuda.Fake(library, monkeypatch)


def _camera(w, h, zoom=1.0):
    return abi.make_camera(abi.PERSPECTIVE, w, h, (0, 0, 0), (0, 0, 0), (0.5, 12.0), (0.8 * zoom * w, 0.8 * zoom * w))


def _batch(slots):
    ctx = rvsb.Context(0)
    scene = rvsb.Scene(ctx, [_camera(64, 32)] * 2)
    planes = [np.zeros(n, np.uint16) for n in (64 * 32, 32 * 16, 32 * 16, 64 * 32)]
    for k in range(2):
        scene.upload(k, planes, on_device=False)
    return rvsb.Batch(scene, slots)


def _run(fake, batch, zooms, precision=1.0):
    """One batch of 64x32 views; its last launch."""
    cams = [_camera(64, 32, z) for z in zooms]
    outs = [[1 << 20, 2 << 20, 3 << 20]] * len(cams)  # addresses the fake never follows
    batch.synthesize(cams, rvsb.params(5.0, precision), outs)
    return fake.launches()[-1]


def test_a_choice_is_kept_per_magnification(fake):
    """Cameras of one size that magnify differently are tuned apart: a choice
    for unmagnified triangles would list nearly every magnified one."""
    batch = _batch(2)
    batch.set_autotune(True)
    assert _run(fake, batch, [1.0, 1.0]).variant == 4
    near = _run(fake, batch, [4.0, 4.0])
    assert (near.variant, near.small) == (7, 36)
    nearer = _run(fake, batch, [20.0, 20.0])
    assert (nearer.variant, nearer.small) == (7, 4)
    count = fake.lib.fake_launches()
    for zooms, variant in (([1.0, 1.0], 4), ([4.0, 4.0], 7), ([20.0, 20.0], 7)):
        assert _run(fake, batch, zooms).variant == variant
    assert fake.lib.fake_launches() == count + 3  # all known by now
    mixed = _run(fake, batch, [1.0, 4.0])
    assert mixed.variant == 7 and fake.lib.fake_launches() > count + 4


@pytest.mark.parametrize("zoom,distinct", [(1.0, 5), (4.0, 6), (20.0, 5)])
def test_variants_of_the_same_content_are_timed_once(fake, zoom, distinct):
    """Variants 1, 2 and 4 run the same launch, and 7 too unless the view is
    magnified and its triangles stay with their lanes: a warm-up and five rounds of the distinct ones, and the call."""
    batch = _batch(2)
    batch.set_autotune(True)
    _run(fake, batch, [zoom, zoom])
    assert fake.lib.fake_launches() == 6 * distinct + 1


# 64x32 inputs, 2 views: 8,192 triangles; the list holds 16,384 and is filled to
# three quarters at most.  960x540, 4 views: 4.1 million, 188,509 entries.
@pytest.mark.parametrize("w,h,views,out,zoom,small", [
    (64, 32, 2, (64, 32), 1.0, 4), (64, 32, 2, (64, 32), 1.15, 16), (64, 32, 2, (64, 32), 2.5, 16),
    (64, 32, 2, (64, 32), 2.9, 25), (64, 32, 2, (64, 32), 4.45, 36), (64, 32, 2, (64, 32), 4.55, 4),
    (64, 32, 2, (64, 32), 40.0, 4), (64, 32, 2, (640, 320), 0.9, 4), (960, 540, 4, (960, 540), 4.6, 36),
    (960, 540, 4, (960, 540), 5.3, 49), (960, 540, 4, (960, 540), 5.5, 4), (960, 540, 4, (4800, 2700), 1.0, 49),
    (960, 540, 4, (9408, 5292), 1.0, 121), (960, 540, 4, (9620, 5412), 1.0, 4),
    (320, 180, 2, (1920, 1080), 1.0, 64), (320, 180, 1, (1920, 1080), 2.0, 4)])
def test_threshold_by_magnification_and_triangles_in_sight(fake, w, h, views, out, zoom, small):
    ctx = rvsb.Context(0)
    scene = rvsb.Scene(ctx, [_camera(w, h)] * views)
    planes = [np.zeros(n, np.uint16) for n in (w * h, w * h // 4, w * h // 4, w * h)]
    for k in range(views):
        scene.upload(k, planes, on_device=False)
    scene.synthesize(_camera(*out, zoom), rvsb.params(5.0), [1 << 20, 2 << 20, 3 << 20])
    assert fake.launches()[-1].small == small
    ctx.close()
