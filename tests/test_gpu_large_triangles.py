"""Long stretched triangles and full lists of them, against the oracle: per-view
coverage and hole mask identical, output at the parity bar.  What each scene
puts into the list of large triangles is counted from the oracle's warped
vertices, so the scenes are known to reach what they are for."""
import copy

import numpy as np
import pytest

import oracle as O
import rvsb
from rvsb import scenes
from helpers import assert_parity, gpu_synthesize

pytestmark = pytest.mark.gpu

THRESHOLD = 4  # candidate pixels of raster variant 0
BAND = 8192    # pixels of a list entry
HUGE = 16384   # covered pixels above which a triangle is shared out


def _capacity(inputs):
    """Entries of the list, and slots for the huge triangles."""
    entries = max(1 << 14, sum(c.width * c.height for c in inputs) // 11)
    slots = min(8192, entries // 16) // 2 * 2
    return entries - slots // 2, slots


def _listed(uv, z, wo, ho):
    """(entries, bounding-box diagonals, huge ones) of one view's triangles above
    the threshold: two per quad, emitted, front-facing, their candidate boxes cut
    into bands of rows."""
    x, y = uv[..., 0].astype(np.float64), uv[..., 1].astype(np.float64)
    ok = (z > 0) & (x > 0)
    diag = ok[:-1, 1:] & ok[1:, :-1]
    entries, lengths, huge = 0, [], 0
    for corner, (a, b, c) in ((ok[:-1, :-1], ((0, 0), (0, 1), (1, 0))), (ok[1:, 1:], ((1, 1), (1, 0), (0, 1)))):
        at = lambda m, p: m[p[0]:m.shape[0] - 1 + p[0], p[1]:m.shape[1] - 1 + p[1]]
        ax, bx, cx = (at(x, p) for p in (a, b, c))
        ay, by, cy = (at(y, p) for p in (a, b, c))
        den = (by - cy) * (ax - cx) + (cx - bx) * (ay - cy)
        mnx, mxx = np.minimum(np.minimum(ax, bx), cx), np.maximum(np.maximum(ax, bx), cx)
        mny, mxy = np.minimum(np.minimum(ay, by), cy), np.maximum(np.maximum(ay, by), cy)
        w = np.minimum(wo - 1, np.rint(mxx) - 1) - np.maximum(0, np.rint(mnx)) + 1
        h = np.minimum(ho - 1, np.rint(mxy) - 1) - np.maximum(0, np.rint(mny)) + 1
        with np.errstate(invalid="ignore"):
            on = diag & corner & (den > 1e-6) & (w > 0) & (h > 0) & (w * h > THRESHOLD)
        entries += int(np.ceil(h[on] / np.maximum(1, BAND // w[on])).sum())
        lengths.append(np.hypot(mxx - mnx, mxy - mny)[on])
        huge += int((np.minimum(den / 2, w * h)[on] > 1.01 * HUGE).sum())
    return entries, np.concatenate(lengths), huge


def _against_oracle(ctx, wl, target, planes):
    """The synthesis with variant 0 (and, bit for bit, 7) against the oracle;
    returns the entries of the list, the triangles' lengths and how many are huge."""
    sc = rvsb.Scene(ctx, wl.inputs)
    for i, p in enumerate(planes):
        sc.upload(i, [np.ascontiguousarray(a, np.uint16) for a in p], on_device=False)
    sc.set_raster_variant(0)
    yuv, dbg, _ = gpu_synthesize(ctx, wl.inputs, planes, target, 5.0, debug=True, scene=sc)
    entries, lengths, huge = 0, [], 0
    for v, (cam, (y, u, w, d)) in enumerate(zip(wl.inputs, planes)):
        uv, vd, wrap = O.warp(cam, target, O.decode_depth(d, cam))
        n, l, k = _listed(uv, vd, target.width, target.height)
        entries += n
        huge += k
        lengths.append(l)
        _, _, valid = O.raster(O.decode_color(y, u, w, cam.bit_depth_color), vd, uv, target.width, target.height, wrap)
        gpu = dbg["view_validity"][v] > 0
        assert np.array_equal(gpu, valid > 0), f"view {v}: coverage differs at {np.argwhere(gpu != (valid > 0))[:5]}"
    assert_parity(yuv, O.synthesize(wl.inputs, planes, target, 5.0))
    sc.set_raster_variant(7)
    other, _ = gpu_synthesize(ctx, wl.inputs, planes, target, 5.0, scene=sc)
    for a, b in zip(other, yuv):
        np.testing.assert_array_equal(a, b)
    return entries, np.concatenate(lengths), huge


def _scaled(target, w, h):
    t = copy.deepcopy(target)
    for i, (new, old) in enumerate(((w, target.width), (h, target.height))):
        t.focal[i] *= new / old
        t.principle_point[i] = new / 2.0
    t.width, t.height = w, h
    return t


@pytest.mark.parametrize("roll", [0.0, 25.0, 60.0])
def test_depth_steps_stretch_across_the_view(ctx, roll):
    """Patches of 64 x 48 pixels, near or far, seen from beside: triangles up
    to several hundred pixels long between them, some with boxes of more than
    one band, and the list not full."""
    wl = scenes.random_pose_small(n_views=2, w=512, h=288, seed=340)
    rng = np.random.default_rng(341)
    planes = []
    for y, u, v, d in wl.planes:
        step = np.kron(rng.integers(0, 2, (6, 8)), np.ones((48, 64), int))
        planes.append((y, u, v, (step * 40000 + 6000 + d // 64).astype(np.uint16)))
    target = copy.deepcopy(wl.targets[0])
    target.position[1] += 0.5
    target.position[2] += 0.15
    target.rotation[2] += roll
    entries, lengths, _ = _against_oracle(ctx, wl, target, planes)
    bands = entries - len(lengths)
    assert entries <= _capacity(wl.inputs)[0] and bands > 100 and (lengths > 300).sum() > 500, (
        entries, bands, lengths.max())


@pytest.mark.parametrize("w,h,wo,ho", [(160, 96, 640, 384), (128, 96, 1920, 1080), (320, 160, 640, 384), (482, 270, 960, 540)])
def test_noise_overflows_the_list(ctx, w, h, wo, ho):
    """Depth samples of pure noise: nearly every triangle is stretched over
    much of the view, and there are more of them than the list holds.  The
    pass over the whole mesh takes groups of 1, 1, 2 and 4 rows."""
    wl = scenes.random_pose_small(n_views=2, w=w, h=h, seed=350)
    rng = np.random.default_rng(351)
    planes = [(y, u, v, rng.integers(0, 65536, d.shape).astype(np.uint16)) for y, u, v, d in wl.planes]
    target = _scaled(wl.targets[0], wo, ho)
    target.position[1] += 0.2
    entries, _, _ = _against_oracle(ctx, wl, target, planes)
    assert entries > 1.5 * _capacity(wl.inputs)[0], entries


@pytest.mark.parametrize("w,h,slots", [(32, 24, "enough"), (64, 48, "too few")])
def test_huge_triangles_of_a_full_list(ctx, w, h, slots):
    """Noise of few quads over a 3840x2160 view: hundreds of huge triangles among
    those whose bands overflow the list.  The 1,024 words hold the smaller mesh's;
    those of the larger that find none stay with their warps."""
    wl = scenes.random_pose_small(n_views=2, w=w, h=h, seed=370)
    rng = np.random.default_rng(371)
    planes = [(y, u, v, rng.integers(0, 65536, d.shape).astype(np.uint16)) for y, u, v, d in wl.planes]
    target = _scaled(wl.targets[0], 3840, 2160)
    target.position[1] += 1.0
    entries, _, huge = _against_oracle(ctx, wl, target, planes)
    room, there = _capacity(wl.inputs)
    assert entries > 1.2 * room and (huge > 100) and (huge <= there) == (slots == "enough"), (entries, huge)


def test_huge_triangles_across_the_seam(ctx):
    """An equirectangular output: depth steps next to its poles and its seam, with
    triangles over much of its width."""
    wl = scenes.random_pose_small(n_views=2, w=160, h=80, seed=372, erp_in=True, erp_out=True)
    rng = np.random.default_rng(373)
    planes = []
    for y, u, v, d in wl.planes:
        step = np.kron(rng.integers(0, 2, (40, 80)), np.ones((2, 2), int))
        planes.append((y, u, v, (step * 50000 + 10000 + d // 64).astype(np.uint16)))
    target = copy.deepcopy(wl.targets[0])
    target.width, target.height = 1600, 800
    target.position[1] += 0.2
    entries, _, huge = _against_oracle(ctx, wl, target, planes)
    assert entries > 1.1 * _capacity(wl.inputs)[0] and huge > 10, (entries, huge)


def test_triangles_wider_than_the_list_knows_boxes_for(ctx):
    """A camera that has moved in among the points: triangles up to its plane,
    wider than 40,000 pixels, are listed whole and shared out, the list not
    full."""
    wl = scenes.random_pose_small(n_views=2, w=96, h=48, seed=380)
    rng = np.random.default_rng(381)
    planes = [(y, u, v, rng.integers(0, 65536, d.shape).astype(np.uint16)) for y, u, v, d in wl.planes]
    target = copy.deepcopy(wl.targets[0])
    target.width, target.height = 1280, 720
    target.principle_point[0], target.principle_point[1] = 640.0, 360.0
    target.focal[0] = target.focal[1] = 1000.0
    target.position[0] += 0.5
    entries, lengths, huge = _against_oracle(ctx, wl, target, planes)
    assert entries <= _capacity(wl.inputs)[0] and (lengths > 6e4).sum() > 10 and huge > 50, (entries, lengths.max(), huge)
