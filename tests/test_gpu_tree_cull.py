"""The breadth-first tile cull against the sequential traversal (tile_stack_entries = 256 selects it)
and the oracle: the same ordered lists and visit counts where a tile fits one warp's store (256
visits), a CTA's (2,048), an SM's (8,192) or none (left to the sequential kernel), on geometry with
many equal keys, and with the dominant axis changing inside a block."""
import numpy as np
import pytest

import hvvr_b200 as hv
from hvvr_b200 import scenes

from helpers import list_mismatch, render_oracle, scene

pytestmark = pytest.mark.gpu

_CACHE = {}


def _scene(name):
    if name != "aligned":
        return scene(name)
    if name not in _CACHE:  # a bare heightfield: rows of boxes share their bounds, so most keys have ties
        _CACHE[name] = hv.generate_topology(scenes.make_scene(96, 1, seed=3))
    return _CACHE[name]


# visits: the range that the view's longest tile has to reach, so that the case stays what it is for
@pytest.mark.parametrize("name,w,h,eye,target,visits", [
    ("small", 97, 61, (0.0, 2.0, 10.0), (0.0, 0.0, 0.0), (1, 256)),
    ("c1", 131, 97, (0.0, 2.0, 10.0), (0.0, 0.0, 0.0), (257, 2048)),
    ("aligned", 64, 48, (7.0, 2.5, 7.0), (0.0, 0.0, 0.0), (257, 2048)),     # looking along the diagonal of x and z
    ("c1", 24, 18, (5.0, 3.0, 8.0), (0.0, 0.0, 0.0), (2049, 8192)),
    ("aligned", 13, 7, (0.0, 2.0, 10.0), (0.0, 0.0, 0.0), (257, 8192)),
    ("c2", 31, 17, (6.0, 2.0, 7.0), (0.0, 0.0, 0.0), (8193, 1 << 30)),
    ("c2", 160, 120, (-7.0, 1.5, -7.5), (0.5, 0.0, 0.0), (2049, 1 << 30)),
])
def test_lists_equal_sequential_cull_and_oracle(oracle, name, w, h, eye, target, visits):
    sc = _scene(name)
    rc = hv.Raycaster()
    rc.create_model(sc)
    for light in sc.lights:
        rc.create_light(light)
    smp = scenes.grid_samples(w, h)
    xf = scenes.camera_transform(eye, target)
    cam = rc.create_camera(scenes.viewport_for(w, h))
    cam.set_render_target(w, h)
    cam.set_samples(smp)
    cam.set_camera_to_world(xf)
    cam.set_msaa(2)
    got = []
    for entries in (256, 0):
        batch = hv.Batch(cameras=[cam], config=hv.batch_config(tile_stack_entries=entries, tri_index_capacity=1 << 24))
        # frame 1 knows no costs, so every tile starts in a warp's store; later frames start it by its cost
        for _ in range(3):
            batch.render()
            assert batch.stats()["status"] == 0
            got.append((*cam.tile_lists(), cam.tile_costs(), cam.image.copy()))
        batch.close()
    assert visits[0] <= int(got[0][2].max()) <= visits[1], int(got[0][2].max())
    for counts, idx, costs, image in got[1:]:
        assert np.array_equal(counts, got[0][0]) and np.array_equal(idx, got[0][1])
        assert np.array_equal(costs, got[0][2]) and np.array_equal(image, got[0][3])
    fo = render_oracle(oracle, sc, smp, w, h, 2, cam_xf=xf)
    assert list_mismatch(got[0][0], got[0][1], fo.tile_counts, fo.tile_indices) == 0
    rc.close()
