"""Where few tiles have long lists (at most 256 of at least 191 visits and 592 of 47 in the last frame), four
CTAs shade each, a warp's samples apiece. A layout's frames go over to it from the fifth on, and to launches
without the pass for huge tiles where it has none. Hits, depths and images of every frame equal the oracle's and
one another, at every rate and in both arithmetic modes, also where the view moves into and out of the rule."""
import numpy as np
import pytest

import hvvr_b200 as hv
from hvvr_b200 import scenes

from helpers import render_oracle, scene

pytestmark = pytest.mark.gpu
FAR, NEAR = (0.0, 120.0, 160.0), (0.0, 2.0, 10.0)


def _camera(sc, w, h, msaa, fp_mode=hv.HVVR_FP_FMA):
    rc = hv.Raycaster(fp_mode=fp_mode)
    rc.create_model(sc)
    for light in sc.lights:
        rc.create_light(light)
    cam = rc.create_camera(scenes.viewport_for(w, h))
    cam.set_render_target(w, h)
    cam.set_samples(scenes.barrel_samples(w, h))
    cam.set_msaa(msaa)
    cam.set_capture(hv.HVVR_CAPTURE_HITS)
    return rc, cam


def _rule(cam):
    costs, counts = cam.tile_costs(), cam.tile_lists()[0]
    few = 1 <= int((costs >= 191).sum()) <= 256 and int((costs >= 47).sum()) <= 592
    return few and int(counts.max()) >= 1024


@pytest.mark.parametrize("fp_mode", [hv.HVVR_FP_FMA, hv.HVVR_FP_STRICT])
@pytest.mark.parametrize("msaa", [1, 2, 4, 8, 16, 32])
def test_split_tiles_change_nothing(oracle, msaa, fp_mode):
    sc = scene("c1")
    w, h = 101, 75
    rc, cam = _camera(sc, w, h, msaa, fp_mode)
    xf = scenes.camera_transform(FAR, (0.0, 0.0, 0.0))
    cam.set_camera_to_world(xf)
    fo = render_oracle(oracle, sc, scenes.barrel_samples(w, h), w, h, msaa, xf, fp_mode)
    images = []
    for frame in range(8):
        rc.render()
        if frame in (0, 7):
            ids, depth = cam.hits()
            assert np.array_equal(ids, fo.hit_ids)
            assert np.array_equal(depth.view(np.uint32), fo.depth.view(np.uint32))
            d = np.abs(cam.sample_colors().view(np.uint8).astype(int) - fo.colors.view(np.uint8).astype(int))
            assert d.max() <= 1
        images.append(cam.image.copy())
    assert _rule(cam)
    assert all(np.array_equal(image, images[0]) for image in images[1:])
    rc.close()


@pytest.mark.parametrize("msaa", [1, 8])
def test_view_moves_into_and_out_of_the_rule(msaa):
    sc = scene("c1")
    w, h = 1280, 960
    want = {}
    for eye in (FAR, NEAR):
        rc, cam = _camera(sc, w, h, msaa)
        cam.set_camera_to_world(scenes.camera_transform(eye, (0.0, 0.0, 0.0)))
        rc.render()
        want[eye] = (*cam.hits(), cam.image.copy())
        assert _rule(cam) == (eye == FAR)
        rc.close()
    rc, cam = _camera(sc, w, h, msaa)
    for eye in [NEAR] * 6 + [FAR] * 3 + [NEAR] * 2 + [FAR, NEAR, FAR]:
        cam.set_camera_to_world(scenes.camera_transform(eye, (0.0, 0.0, 0.0)))
        rc.render()
        got = (*cam.hits(), cam.image)
        assert all(np.array_equal(a.view(np.uint32), b.view(np.uint32)) for a, b in zip(got, want[eye]))
    rc.close()
