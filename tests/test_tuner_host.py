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
    near = _run(fake, batch, [5.0, 5.0])
    assert (near.variant, near.small) == (7, 49)
    count = fake.lib.fake_launches()
    for zooms, variant in (([1.0, 1.0], 4), ([5.0, 5.0], 7)):
        assert _run(fake, batch, zooms).variant == variant
    assert fake.lib.fake_launches() == count + 2  # both known by now
    mixed = _run(fake, batch, [1.0, 5.0])
    assert mixed.variant == 7 and fake.lib.fake_launches() > count + 3


@pytest.mark.parametrize("zoom,distinct", [(1.0, 5), (5.0, 6)])
def test_variants_of_the_same_content_are_timed_once(fake, zoom, distinct):
    """Variants 1, 2 and 4 run the same launch, and 7 too unless the view is
    magnified: a warm-up and five rounds of the distinct ones, and the call."""
    batch = _batch(2)
    batch.set_autotune(True)
    _run(fake, batch, [zoom, zoom])
    assert fake.lib.fake_launches() == 6 * distinct + 1
