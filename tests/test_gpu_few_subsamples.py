"""The intersect's bounds at one and two subsamples are taken around the subsamples' own directions, not
around the sample's centre: hit IDs and depths equal the oracle's bit for bit with both offset patterns,
where triangles are far smaller than a sample and lists long, at extreme scales (the bounds' rounding terms
are then all that widens them), and with a depth tie in every hit."""
import copy

import numpy as np
import pytest

import hvvr_b200 as hv
from hvvr_b200 import scenes

from helpers import scene

pytestmark = pytest.mark.gpu


def _scene(name, scale):
    if name == "doubled":
        sc = scenes.make_scene(20, 60, seed=8)
        sc.tri_shade = np.concatenate([sc.tri_shade, sc.tri_shade])
        sc = hv.generate_topology(sc)
    else:
        sc = scene(name)
    out = copy.copy(sc)
    out.verts = sc.verts.copy()
    out.verts["pos"] *= np.float32(scale)
    return out


@pytest.mark.parametrize("fp_mode", [hv.HVVR_FP_FMA, hv.HVVR_FP_STRICT])
@pytest.mark.parametrize("msaa,pattern", [(1, hv.HVVR_MSAA_SPIRAL), (2, hv.HVVR_MSAA_SPIRAL), (1, hv.HVVR_MSAA_ROTATED_GRID),
                                          (2, hv.HVVR_MSAA_ROTATED_GRID)])
@pytest.mark.parametrize("name,scale,w,h,eye,target", [
    ("c1", 1.0, 96, 72, (0.0, 120.0, 160.0), (0.0, 0.0, 0.0)),   # dozens of triangles in a pixel, none hidden
    ("c1", 1.0, 64, 48, (0.0, 2.0, 10.0), (0.0, 0.0, 0.0)),
    ("small", 1e-12, 96, 64, (0.0, 2.0, 10.0), (0.0, 0.0, 0.0)),
    ("small", 1e6, 96, 64, (0.0, 2.0, 10.0), (0.0, 0.0, 0.0)),
    ("doubled", 1.0, 120, 90, (3.0, 1.5, 8.0), (0.0, 0.0, 0.0)),
])
def test_bounds_around_one_or_two_subsamples(oracle, name, scale, w, h, eye, target, msaa, pattern, fp_mode):
    sc = _scene(name, scale)
    xf = scenes.camera_transform(tuple(scale * x for x in eye), tuple(scale * x for x in target))
    smp = scenes.barrel_samples(w, h)
    rc = hv.Raycaster(fp_mode=fp_mode)
    rc.create_model(sc)
    for light in sc.lights:
        rc.create_light(light)
    cam = rc.create_camera(scenes.viewport_for(w, h))
    cam.set_render_target(w, h)
    cam.set_samples(smp)
    cam.set_camera_to_world(xf)
    cam.set_msaa(msaa)
    cam.set_msaa_pattern(pattern)
    cam.set_capture(hv.HVVR_CAPTURE_HITS)
    for _ in range(2):  # the second frame takes its tiles in cost order
        rc.render()
        ids, depth = cam.hits()
    fo = oracle.render(sc, smp, xf, scenes.viewport_for(w, h), w, h, msaa, fp_mode=fp_mode, msaa_pattern=pattern)
    assert np.array_equal(ids, fo.hit_ids)
    assert np.array_equal(depth.view(np.uint32), fo.depth.view(np.uint32))
    assert (ids != 0xFFFFFFFF).any()
    rc.close()
