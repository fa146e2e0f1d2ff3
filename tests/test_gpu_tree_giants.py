"""Tiles of more visits than an SM's store holds (8,192): from the second frame that shows some on, a frame of one
rate class culls them breadth first with stores in global memory (32,768 visits), at once or from the retry
list, and leaves larger ones to the sequential kernel. Lists, visit counts and images of every frame equal the
sequential cull's, pipelined and not, with fewer and more such tiles than stores, and where the view moves."""
import numpy as np
import pytest

import hvvr_b200 as hv
from hvvr_b200 import scenes

from helpers import scene

pytestmark = pytest.mark.gpu


def _cameras(count, w, h, msaa):
    sc = scene("c2")
    rc = hv.Raycaster()
    rc.create_model(sc)
    for light in sc.lights:
        rc.create_light(light)
    cams = []
    for _ in range(count):
        cam = rc.create_camera(scenes.viewport_fov(w, h, 100.0))
        cam.set_render_target(w, h)
        cam.set_samples(scenes.grid_samples(w, h))
        cam.set_msaa(msaa)
        cams.append(cam)
    return rc, cams


def _pose(cams, eye):
    for k, cam in enumerate(cams):
        cam.set_camera_to_world(scenes.camera_transform((eye[0], eye[1] + 0.05 * k, eye[2]), (0.0, 0.0, 0.0)))


def _read(cams):
    return [x for cam in cams for x in (*cam.tile_lists(), cam.tile_costs(), cam.image.copy())]


# giants: how many tiles are above 8,192 visits, and above 32,768, so that the case stays what it is for
@pytest.mark.parametrize("pipeline", [1, 0])
@pytest.mark.parametrize("count,w,h,msaa,giants,beyond", [
    (1, 300, 225, 1, (1, 32), (0, 0)),
    (1, 256, 192, 4, (1, 64), (0, 0)),
    (8, 160, 120, 8, (33, 200), (0, 0)),
    (1, 40, 30, 1, (1, 20), (1, 20)),
])
def test_giant_tiles_equal_sequential_cull(count, w, h, msaa, giants, beyond, pipeline):
    rc, cams = _cameras(count, w, h, msaa)
    eyes = [(7.0, 2.5, 7.0), (-7.0, 2.5, 7.0)]
    want = []
    for eye in eyes:
        _pose(cams, eye)
        batch = hv.Batch(cameras=cams, config=hv.batch_config(tile_stack_entries=256, tri_index_capacity=1 << 26))
        batch.render()
        want.append(_read(cams))
        batch.close()
    costs = np.concatenate([cam.tile_costs() for cam in cams])
    assert giants[0] <= int((costs > 8192).sum()) <= giants[1] and beyond[0] <= int((costs > 32768).sum()) <= beyond[1]
    for cam in cams:
        cam.set_samples(scenes.grid_samples(w, h))  # (a new sample set has no costs)
    batch = hv.Batch(cameras=cams, config=hv.batch_config(tri_index_capacity=1 << 26, pipeline=pipeline))
    for view in (0, 0, 0, 0, 1, 0, 0, 1, 1):
        _pose(cams, eyes[view])
        batch.render()
        assert batch.stats()["status"] == 0
        for a, b in zip(_read(cams), want[view]):
            assert np.array_equal(a, b)
    batch.close()
    rc.close()
