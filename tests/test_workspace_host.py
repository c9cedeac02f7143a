"""A slot's workspace after an allocation that failed, on a fake runtime: the
calls that follow launch with every buffer in place and of its size."""
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


def _scene(ctx):
    sc = rvsb.Scene(ctx, [_camera(32, 16), _camera(32, 16)])
    for v in range(2):
        sc.upload(v, _planes(32, 16) + [np.zeros(32 * 16, np.uint16)], on_device=False)
    return sc


OPTIONS = {"plain": rvsb.params(5.0), "precision": rvsb.params(5.0, precision=1.5),
           "multispectral": rvsb.params(5.0, multispectral=(1.0, 8.0)), "aux": rvsb.params(5.0)}


def _call(sc, option, w, h):
    if option == "aux":
        sc.synthesize_aux(_camera(w, h), OPTIONS[option], _planes(w, h), mask=np.zeros(w * h, np.uint8))
    else:
        sc.synthesize(_camera(w, h), OPTIONS[option], _planes(w, h))


# What grows with the output: hole mask, minima, codes and scans, then the option's own buffers.
@pytest.mark.parametrize("option,after", [("plain", k) for k in range(4)] + [("precision", k) for k in range(6)] +
                         [("aux", k) for k in range(6)] + [("multispectral", k) for k in range(8)])
def test_a_failed_allocation_leaves_no_buffer_behind(fake, option, after):
    ctx = rvsb.Context(0)
    sc = _scene(ctx)
    _call(sc, option, 32, 16)
    fake.fail("cudaMalloc", after)
    with pytest.raises(rvsb.RvsbError) as e:
        _call(sc, option, 64, 32)
    assert e.value.status == abi.RVSB_E_CUDA
    fake.lib.cudaGetLastError()
    for w, h in ((32, 16), (64, 32), (32, 16)):
        _call(sc, option, w, h)
    assert [f.unbacked for f in fake.launches()] == [0, 0, 0, 0]
    sc.close()
    ctx.close()


def test_a_request_beyond_the_budget_leaves_no_buffer_behind(fake):
    probe = rvsb.Context(0)
    sc = _scene(probe)
    _call(sc, "plain", 32, 16)
    room = probe.memory_in_use()
    sc.close()
    probe.close()
    fake.lib.fake_reset()
    ctx = rvsb.Context(0, hbm_budget=room + 1000)
    sc = _scene(ctx)
    _call(sc, "plain", 32, 16)
    with pytest.raises(rvsb.RvsbError) as e:
        _call(sc, "plain", 640, 320)
    assert e.value.status == abi.RVSB_E_OOM_BUDGET
    _call(sc, "plain", 32, 16)
    assert [f.unbacked for f in fake.launches()] == [0, 0]
    sc.close()
    ctx.close()
