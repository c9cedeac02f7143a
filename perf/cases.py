"""Timed cases of the view-synthesis backend, through its public entry points.

Every case is one call a program makes per output frame (or per group of
output frames): a resident scene seen by a new virtual camera, a frame whose
raw planes are on the device, a frame in host memory, a group of poses in one
batch.  Inputs are the package's seeded ray-cast scenes at the case's sizes,
in the formats the backend reads (YUV420 colour in 16-bit samples, 16-bit
normalised-disparity depth).

A case's fields:
  call       "scene" (resident inputs), "frame" (raw planes on the device),
             "host" (raw planes in pinned host memory, result in host memory),
             "aux" (resident, with the mask, depth and masked outputs),
             "batch" (several poses of a resident scene, one graph replay)
  views      input views; in_w x in_h each, equirectangular when in_erp
  targets    output views of the call; out_w x out_h each (mixed: that size,
             15/16 and 15/32 of it in turn), equirectangular when out_erp
  bits       colour bit depth of inputs and output
  exponent   BlendingFactor (negative: blend by maximum)
  low, high  Multispectral blending factors (0, 0: simple blending)
  precision  raster oversampling
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rvs-cuda_b200"))

import rvsb  # noqa: E402
from rvsb import abi, scenes  # noqa: E402


def _case(name, call, views, in_w, in_h, out_w, out_h, *, targets=1, mixed=False, in_erp=False, out_erp=False,
          bits=10, exponent=5.0, low=0.0, high=0.0, precision=1.0):
    c = dict(call=call, views=views, in_w=in_w, in_h=in_h, in_erp=in_erp, out_w=out_w, out_h=out_h, out_erp=out_erp,
             targets=targets, mixed=mixed, bits=bits, exponent=exponent, low=low, high=high, precision=precision)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # The smallest configuration, a stereo pair seen from between: an
        # interactive viewer's frame, launches and latency count.
        _case("pair_540p", "scene", 2, 960, 540, 960, 540),
        # The headline workload: one frame of four 1080p cameras, raw planes
        # resident, decoded and synthesised at a free pose.
        _case("frame_1080p", "frame", 4, 1920, 1080, 1920, 1080),
        # The same frame through the drop-in call with host buffers.
        _case("host_1080p", "host", 4, 1920, 1080, 1920, 1080),
        # Small cameras shown on a large screen: magnified triangles.
        _case("upscale_1080p", "scene", 2, 960, 540, 1920, 1080),
        # A thumbnail or preview of full-size cameras: minified triangles.
        _case("preview_540p", "scene", 4, 1920, 1080, 960, 540),
        # Depth, mask and masked outputs for a coding tool, 12-bit material of
        # a size that is no multiple of any tile.
        _case("aux_ragged", "aux", 3, 1366, 770, 1278, 718, bits=12),
        # Multispectral blending, the reference's quality option.
        _case("multispectral_1080p", "scene", 4, 1920, 1080, 1920, 1080, low=1.0, high=8.0),
        # Oversampled synthesis (Precision 2), its other quality option.
        _case("precision2_540p", "scene", 2, 960, 540, 960, 540, precision=2.0),
        # Serving: several users' poses of one resident scene in one launch
        # group.
        _case("batch_1080p", "batch", 4, 1920, 1080, 1920, 1080, targets=8),
        # A camera array serving displays of several sizes.
        _case("batch_mixed", "batch", 11, 2048, 1088, 2048, 1088, targets=12, mixed=True),
        # 360-degree video seen through headsets.
        _case("batch_erp", "batch", 4, 4096, 2048, 1920, 1080, targets=8, in_erp=True),
        # 360-degree video at a new viewpoint.
        _case("erp_to_erp", "scene", 4, 4096, 2048, 4096, 2048, in_erp=True, out_erp=True),
    ]


def _log_even(rng, lo, hi):
    return 2 * int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2))


def draw(rng):
    kind = rng.choice(["scene", "frame", "host", "aux", "options", "batch", "mixed", "erp", "erp_out"])
    bits = rng.choice([10, 10, 10, 12, 16])
    exponent = rng.choice([5.0, 5.0, 5.0, 2.0, 1.0, -1.0])
    if kind in ("erp", "erp_out"):
        in_w = _log_even(rng, 1024, 4096)
        in_h = 2 * (in_w // 4)
        views = rng.randint(2, 4)
        if kind == "erp_out":
            out_w = _log_even(rng, 512, 4096)
            return _case("", "scene", views, in_w, in_h, out_w, 2 * (out_w // 4), in_erp=True, out_erp=True)
        out_w = _log_even(rng, 480, 1920)
        return _case("", "batch", views, in_w, in_h, out_w, _ratio(rng, out_w), targets=rng.randint(1, 8), in_erp=True,
                     exponent=exponent)
    in_w = _log_even(rng, 480, 2048)
    out_w = _log_even(rng, 480, 2048)
    in_h, out_h = _ratio(rng, in_w), _ratio(rng, out_w)
    if kind == "mixed":
        return _case("", "batch", rng.randint(5, 11), in_w, in_h, in_w, in_h, targets=rng.randint(2, 10), mixed=True,
                     exponent=exponent)
    if kind == "batch":
        return _case("", "batch", rng.randint(2, 4), in_w, in_h, out_w, out_h, targets=rng.randint(2, 16), bits=bits,
                     exponent=exponent)
    views = rng.randint(1, 5)
    if kind == "options":
        if rng.random() < 0.5:
            low, high = rng.choice([(1.0, 8.0), (5.0, 2.0), (-1.0, 4.0)])
            return _case("", "scene", views, in_w, in_h, out_w, out_h, low=low, high=high, bits=bits)
        return _case("", "scene", views, in_w, in_h, out_w, out_h, precision=rng.choice([2.0, 1.5, 0.75, 0.5]),
                     bits=bits)
    return _case("", kind, views, in_w, in_h, out_w, out_h, bits=bits, exponent=exponent)


def _ratio(rng, w):
    return 2 * int(round(w * rng.uniform(0.5, 0.7) / 2))


def _cameras(case, seed):
    """(scene, input cameras, target cameras): the package's seeded scene for
    the number and kind of views, its camera spacing, field of view, depth
    range and pose distribution at the case's sizes."""
    n, bits = case["views"], case["bits"]
    seed = 0x5EED0000 + 7919 * int(seed)
    r = random.Random(seed)
    w, h = case["in_w"], case["in_h"]
    if case["in_erp"]:
        scene, rng_d = scenes.batched_erp(seed=seed).scene, (0.3, 20.0)
        s = 0.2 / math.sqrt(3)
        at = [(s, s, s), (s, -s, -s), (-s, s, -s), (-s, -s, s)][:n]
        inputs = [abi.make_camera(abi.EQUIRECTANGULAR, w, h, p, (0, 0, 0), rng_d, bit_depth_color=bits) for p in at]
        box, turn = (0.1, 0.1, 0.05), (180.0, 8.0, 3.0)
    else:
        make = scenes.plain_small if n <= 2 else scenes.plain_1080p if n <= 5 else scenes.batched_mixed
        scene, rng_d = make(seed=seed).scene, (0.5, 12.0)
        cols = n if n <= 2 else 2 if n <= 5 else 4
        step = 0.1 if n <= 2 or n > 5 else 0.15
        rows = -(-n // cols)
        at = [(0.0, step * ((cols - 1) / 2 - k % cols), step * ((rows - 1) / 2 - k // cols)) for k in range(n)]
        f = 0.79 * w
        inputs = [abi.make_camera(abi.PERSPECTIVE, w, h, p, (0, 0, 0), rng_d, (f, f), bit_depth_color=bits) for p in at]
        box, turn = (0.08, 0.075 if cols > 1 else 0.03, 0.075 if rows > 1 else 0.02), (4.0, 4.0, 3.0)
    targets = []
    for k in range(case["targets"]):
        tw, th = case["out_w"], case["out_h"]
        if case["mixed"]:
            tw, th = [(tw, th), (_even(tw * 15 / 16), _even(th * 15 / 16)), (_even(tw * 15 / 32), _even(th * 15 / 32))][k % 3]
        pos = [r.uniform(-b, b) for b in box]
        rot = [r.uniform(-t, t) for t in turn]
        if case["out_erp"]:
            targets.append(abi.make_camera(abi.EQUIRECTANGULAR, tw, th, pos, (rot[0], 0, 0), rng_d, bit_depth_color=bits))
        else:
            f = tw / 2.0 if case["in_erp"] else 0.79 * tw  # 90 degrees, or the inputs' field of view
            targets.append(abi.make_camera(abi.PERSPECTIVE, tw, th, pos, rot, rng_d, (f, f), bit_depth_color=bits))
    return scene, inputs, targets


def _even(x):
    return max(2, 2 * int(round(x / 2)))


def _yuv(w, h, device="cuda", pin=False):
    return [torch.zeros(n, dtype=torch.int16, device=device, pin_memory=pin)
            for n in (w * h, (w // 2) * (h // 2), (w // 2) * (h // 2))]


def prepare(case, seed):
    scene, inputs, targets = _cameras(case, seed)
    planes = [[torch.from_numpy(np.ascontiguousarray(a).view(np.int16).reshape(-1)) for a in scenes.render(scene, c)]
              for c in inputs]
    st = dict(case=case, inputs=inputs, targets=targets)
    ms = (case["low"], case["high"]) if case["low"] or case["high"] else None
    st["params"] = rvsb.params(case["exponent"], case["precision"], multispectral=ms)
    ctx = st["ctx"] = rvsb.Context(torch.cuda.current_device())
    if case["call"] == "host":
        st["planes"] = [[p.pin_memory() for p in v] for v in planes]
        st["outs"] = [_yuv(t.width, t.height, "cpu", True) for t in targets]
        return st
    st["outs"] = [_yuv(t.width, t.height) for t in targets]
    sc = st["scene"] = rvsb.Scene(ctx, inputs)
    st["planes"] = [[p.cuda() for p in v] for v in planes]
    if case["call"] == "frame":
        return st
    for k, v in enumerate(st["planes"]):
        sc.upload(k, v, on_device=True)
    torch.cuda.synchronize()
    st["planes"] = None  # the scene holds its own copy
    if case["call"] == "aux":
        w, h = targets[0].width, targets[0].height
        st["aux"] = dict(mask=torch.zeros(w * h, dtype=torch.uint8, device="cuda"), masked=_yuv(w, h),
                         depth=torch.zeros(w * h, dtype=torch.int16, device="cuda"),
                         masked_depth=torch.zeros(w * h, dtype=torch.int16, device="cuda"))
    if case["call"] == "batch":
        st["batch"] = rvsb.Batch(sc, len(targets), graphs=True)
        st["batch"].reserve(case["out_w"], case["out_h"])
    return st


def run(st):
    call, p, outs = st["case"]["call"], st["params"], st["outs"]
    stream = torch.cuda.current_stream()
    if call == "scene":
        st["scene"].synthesize(st["targets"][0], p, outs[0], stream)
    elif call == "frame":
        st["scene"].synthesize_frame(st["planes"], st["targets"][0], p, outs[0], stream)
    elif call == "host":
        st["ctx"].synthesize_host(st["inputs"], st["planes"], st["targets"][0], p, outs[0], stream)
    elif call == "aux":
        st["scene"].synthesize_aux(st["targets"][0], p, outs[0], stream=stream, **st["aux"])
        return [outs, st["aux"]]
    else:
        st["batch"].synthesize(st["targets"], p, outs, stream)
    return outs


def work(case):
    """Each input sample read once (Y 2, U and V 1, depth 2 bytes a pixel),
    each output sample written once; per input pixel and target the
    unprojection, pose and projection, per output pixel and view one
    triangle's coverage, depth and colour, and the blend."""
    n_in = case["views"] * case["in_w"] * case["in_h"]
    n_out = 0
    for k in range(case["targets"]):
        s = (1.0, 15 / 16, 15 / 32)[k % 3] if case["mixed"] else 1.0
        n_out += int(case["out_w"] * case["out_h"] * s * s)
    n_bytes = 5 * n_in + 3 * n_out * (1 if case["call"] != "aux" else 2) + (5 * n_out if case["call"] == "aux" else 0)
    raster = n_out * case["precision"] ** 2
    return {"bytes": n_bytes, "flops": 30 * n_in * case["targets"] + 60 * raster * case["views"]}


def exact(case, seed):
    """Every output is a whole number: sample codes and masks."""
    return None
