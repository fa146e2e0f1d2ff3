"""The tiles that get a CTA of the breadth-first cull: those of at least 47 visits where at most 592
tiles have as many, else of 95 by the same rule, else of 191. Lists, visit counts and images equal the
sequential cull's on either side of both bounds."""
import numpy as np
import pytest

import hvvr_b200 as hv
from hvvr_b200 import scenes

from helpers import scene

pytestmark = pytest.mark.gpu


# few: whether at most 592 tiles reach 47 and 95 visits, so that the view stays what it is for
@pytest.mark.parametrize("name,w,h,eye,few", [
    ("c1", 160, 120, (0.0, 2.0, 10.0), (True, True)),
    ("c1", 320, 240, (5.0, 3.0, 8.0), (True, True)),      # 576 tiles
    ("c1", 480, 360, (0.0, 2.0, 10.0), (False, True)),    # 832 and 204
    ("c1", 640, 480, (5.0, 3.0, 8.0), (False, True)),
    ("c2", 811, 613, (0.0, 2.0, 10.0), (False, False)),
])
def test_few_large_tiles_equal_sequential_cull(name, w, h, eye, few):
    sc = scene(name)
    rc = hv.Raycaster()
    rc.create_model(sc)
    for light in sc.lights:
        rc.create_light(light)
    cam = rc.create_camera(scenes.viewport_for(w, h))
    cam.set_render_target(w, h)
    cam.set_samples(scenes.grid_samples(w, h))
    cam.set_camera_to_world(scenes.camera_transform(eye, (0.0, 0.0, 0.0)))
    got = []
    for entries in (256, 0):
        batch = hv.Batch(cameras=[cam], config=hv.batch_config(tile_stack_entries=entries, tri_index_capacity=1 << 24))
        for _ in range(3):
            batch.render()
            assert batch.stats()["status"] == 0
            got.append((*cam.tile_lists(), cam.tile_costs(), cam.image.copy()))
        batch.close()
    costs = got[0][2]
    assert few == tuple(int((costs >= v).sum()) <= 592 for v in (47, 95))
    for later in got[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(later, got[0]))
    rc.close()
