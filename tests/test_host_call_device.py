"""rvsb_synthesize_host and the caller's current device, on a fake runtime with
two devices: what the call allocates lies on its context's device, whichever
is current, and a context without such calls never changes it when it goes."""
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


def _camera(w, h):
    return abi.make_camera(abi.PERSPECTIVE, w, h, (0, 0, 0), (0, 0, 0), (0.5, 12.0), (0.8 * w, 0.8 * w))


def _planes(w, h):
    return [np.zeros(n, np.uint16) for n in (w * h, w * h // 4, w * h // 4)]


def _host_call(ctx, cams, w, h):
    out = _planes(w, h)
    ctx.synthesize_host(cams, [_planes(c.width, c.height) + [np.zeros(c.width * c.height, np.uint16)] for c in cams],
                        _camera(w, h), rvsb.params(5.0), out)


def test_output_staging_on_the_contexts_device(fake):
    cams = [_camera(32, 16), _camera(32, 16)]
    ctx = rvsb.Context(1)
    _host_call(ctx, cams, 32, 16)
    # Same cameras, a larger output, another device current.
    fake.lib.fake_set_device(0)
    _host_call(ctx, cams, 64, 32)
    assert [(f.device, f.out_device) for f in fake.launches()] == [(1, 1), (1, 1)]
    ctx.close()


def test_destroying_an_idle_context_leaves_the_current_device(fake):
    ctx = rvsb.Context(1)
    fake.lib.fake_set_device(0)
    ctx.close()
    assert fake.lib.fake_device() == 0
