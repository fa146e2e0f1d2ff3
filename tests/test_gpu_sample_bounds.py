"""The intersect's footprint and depth bounds (which pass by what a tile, a warp or a sample cannot
hit) must change no hit: hit IDs and depths equal the oracle's bit for bit, and images within 1 LSB,
where the bounds are tight - triangles far smaller and far larger than a sample, lists that end inside
a batch of chunks, a camera on the surface, scenes of extreme scale (the bounds' rounding terms), and
coincident triangles (equal depths, decided by list order)."""
import copy

import numpy as np
import pytest

import hvvr_b200 as hv
from hvvr_b200 import scenes

from helpers import render_gpu, render_oracle, scene

pytestmark = pytest.mark.gpu


def _scaled(sc, k):
    out = copy.copy(sc)
    out.verts = sc.verts.copy()
    out.verts["pos"] *= np.float32(k)
    return out


def _doubled():
    """Every triangle twice: each hit is a tie that list order decides."""
    sc = scenes.make_scene(12, 40, seed=8)
    sc.tri_shade = np.concatenate([sc.tri_shade, sc.tri_shade])
    return hv.generate_topology(sc)


def _scene(name):
    if name == "room":  # 2 + 12 triangles, each covering many tiles
        return hv.generate_topology(scenes.make_scene(1, 1, seed=4))
    if name == "doubled":
        return _doubled()
    return scene(name)


@pytest.mark.parametrize("fp_mode", [hv.HVVR_FP_FMA, hv.HVVR_FP_STRICT])
@pytest.mark.parametrize("name,scale,w,h,msaa,eye,target", [
    ("c1", 1.0, 40, 30, 8, (0.0, 2.0, 10.0), (0.0, 0.0, 0.0)),       # subpixel triangles, lists of thousands
    ("c1", 1.0, 97, 53, 1, (4.0, 1.0, 6.0), (-2.0, 0.2, 0.0)),
    ("room", 1.0, 200, 150, 16, (0.0, 2.0, 9.0), (0.0, 0.0, 0.0)),
    ("small", 1e-4, 128, 96, 4, (0.0, 2.0, 10.0), (0.0, 0.0, 0.0)),
    ("small", 1e5, 128, 96, 32, (0.0, 2.0, 10.0), (0.0, 0.0, 0.0)),
    ("small", 1e-12, 96, 64, 8, (0.0, 2.0, 10.0), (0.0, 0.0, 0.0)),  # products below the normal range
    ("doubled", 1.0, 120, 90, 8, (3.0, 1.5, 8.0), (0.0, 0.0, 0.0)),
    ("small", 1.0, 64, 48, 2, (1.0, 0.3, 1.0), (0.0, -1.0, 0.0)),    # among the boxes, looking down
])
def test_bounds_change_no_hit(oracle, name, scale, w, h, msaa, eye, target, fp_mode):
    sc = _scaled(_scene(name), scale)
    xf = scenes.camera_transform(tuple(scale * x for x in eye), tuple(scale * x for x in target))
    smp = scenes.barrel_samples(w, h)
    rc, cam = render_gpu(sc, smp, w, h, msaa, xf, fp_mode)
    for _ in range(2):  # the second frame takes its tiles in cost order
        rc.render()
        ids, depth = cam.hits()
        fo = render_oracle(oracle, sc, smp, w, h, msaa, xf, fp_mode)
        assert np.array_equal(ids, fo.hit_ids)
        assert np.array_equal(depth.view(np.uint32), fo.depth.view(np.uint32))
        d = np.abs(cam.sample_colors().view(np.uint8).astype(int) - fo.colors.view(np.uint8).astype(int))
        assert d.max() <= 1
    assert (ids != 0xFFFFFFFF).any()
    rc.close()


@pytest.mark.parametrize("fp_mode", [hv.HVVR_FP_FMA, hv.HVVR_FP_STRICT])
@pytest.mark.parametrize("name,scale,w,h,msaa,lens,eye,target", [
    ("c1", 1.0, 64, 48, 4, (0.002, 9.0), (0.0, 2.0, 10.0), (0.0, 0.0, 0.0)),   # hardly any blur
    ("c1", 1.0, 96, 72, 8, (0.5, 3.0), (0.0, 2.0, 10.0), (0.0, 0.0, 0.0)),     # focused before the scene
    ("small", 1.0, 97, 61, 1, (0.3, 40.0), (3.0, 1.5, 8.0), (0.0, 0.0, 0.0)),  # focused behind it
    ("room", 1.0, 128, 96, 16, (0.1, 8.0), (0.0, 2.0, 9.0), (0.0, 0.0, 0.0)),
    ("small", 1e4, 96, 64, 8, (400.0, 9e4), (0.0, 2.0, 10.0), (0.0, 0.0, 0.0)),
    ("small", 1e-4, 96, 64, 2, (4e-6, 9e-4), (0.0, 2.0, 10.0), (0.0, 0.0, 0.0)),
    ("doubled", 1.0, 80, 60, 4, (0.05, 7.0), (1.0, 0.6, 3.0), (0.0, -0.5, 0.0)),
])
def test_lens_bounds_change_no_hit(oracle, name, scale, w, h, msaa, lens, eye, target, fp_mode):
    sc = _scaled(_scene(name), scale)
    xf = scenes.camera_transform(tuple(scale * x for x in eye), tuple(scale * x for x in target))
    smp = scenes.barrel_samples(w, h)
    rc, cam = render_gpu(sc, smp, w, h, msaa, xf, fp_mode, lens=lens)
    ids, depth = cam.hits()
    fo = render_oracle(oracle, sc, smp, w, h, msaa, xf, fp_mode, lens=lens)
    assert np.array_equal(ids, fo.hit_ids)
    assert np.array_equal(depth.view(np.uint32), fo.depth.view(np.uint32))
    d = np.abs(cam.sample_colors().view(np.uint8).astype(int) - fo.colors.view(np.uint8).astype(int))
    assert d.max() <= 1
    assert (ids != 0xFFFFFFFF).any()
    rc.close()
