"""rvsb_synthesize_host and the caller's current device, on a fake runtime with
two devices: what the call allocates lies on its context's device, whichever
is current, and a context without such calls never changes it when it goes.
And the order of its work: depth planes, mesh, colour planes, resolve."""
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


@pytest.mark.parametrize("views", [1, 4, 5, 7])
def test_colour_follows_the_mesh_and_precedes_the_resolve(fake, views):
    ctx = rvsb.Context(0)
    for call in range(2):
        _host_call(ctx, [_camera(32, 16)] * views, 32, 16)
        last = fake.launches()[-1]
        assert (last.views, last.decodes_before, last.decodes_at_resolve) == (views, views * call, views * (call + 1))
    ctx.close()


# The depth copies are calls 0 and 1; 2 and 3 the first view's luma and chroma.
@pytest.mark.parametrize("call,after", [("cudaMemcpyAsync", 1), ("cudaMemcpyAsync", 2), ("cudaMemcpyAsync", 3),
                                        ("cudaStreamWaitEvent", 2), ("cudaEventRecord", 2)])
def test_an_error_leaves_no_copy_of_the_callers_planes_running(fake, call, after):
    cams = [_camera(32, 16)] * 2
    ctx = rvsb.Context(0)
    _host_call(ctx, cams, 32, 16)
    fake.fail(call, after)
    with pytest.raises(rvsb.RvsbError) as e:
        _host_call(ctx, cams, 32, 16)
    assert e.value.status == abi.RVSB_E_CUDA
    assert fake.lib.fake_pending_copies() == 0
    fake.lib.cudaGetLastError()
    launches = len(fake.launches())
    _host_call(ctx, cams, 32, 16)
    assert len(fake.launches()) == launches + 1
    ctx.close()


def test_refused_parameters_after_the_depth_upload(fake):
    cams = [_camera(32, 16)] * 2
    ctx = rvsb.Context(0)
    out = _planes(32, 16)
    planes = [_planes(32, 16) + [np.zeros(512, np.uint16)] for _ in cams]
    with pytest.raises(rvsb.RvsbError):
        ctx.synthesize_host(cams, planes, _camera(32, 16), rvsb.params(0.0), out)
    assert fake.lib.fake_pending_copies() == 0 and not fake.launches()
    _host_call(ctx, cams, 32, 16)
    ctx.close()
