"""A triangle-list pool that holds the frame's lists is enough: on a first frame (no costs are known, so
every tile starts in one warp's store) and on later ones, whatever store a tile outgrows, and whether by
its visits or by its list-bearing components (half a store's nodes), the cull takes no more chunks than
the lists have, and one chunk fewer is reported as an overflow."""
import numpy as np
import pytest

import hvvr_b200 as hv
from hvvr_b200 import _abi, scenes

from helpers import scene

pytestmark = pytest.mark.gpu


def _scene(name):
    if isinstance(name, str):
        return scene(name)
    return hv.generate_topology(scenes.make_scene(*name, seed=3))


# visits: the range that some tile has to be in. Seen from far away a whole tree passes one tile's tests, and
# three of four children are components of their own.
NEAR, FAR = (5.0, 3.0, 8.0), (0.0, 900.0, 1500.0)


@pytest.mark.parametrize("pipeline", [1, 0])
@pytest.mark.parametrize("name,w,h,eye,visits", [
    ("c1", 480, 360, NEAR, (130, 256)),
    ("c1", 48, 36, NEAR, (1030, 2048)),
    ("c2", 200, 150, NEAR, (4100, 8192)),
    ((28, 60), 64, 48, FAR, (175, 256)),       # more components than half of a warp's store
    ((84, 100), 64, 48, FAR, (1400, 2048)),    # of a CTA's
    ((160, 500), 64, 48, FAR, (5500, 8192)),   # of an SM's: left to the sequential kernel
])
def test_pool_of_the_lists_size_is_enough(name, w, h, eye, visits, pipeline):
    sc = _scene(name)
    rc = hv.Raycaster()
    rc.create_model(sc)
    for light in sc.lights:
        rc.create_light(light)
    cam = rc.create_camera(scenes.viewport_for(w, h))
    cam.set_render_target(w, h)
    cam.set_camera_to_world(scenes.camera_transform(eye, (0.0, 0.0, 0.0)))
    cam.set_samples(scenes.grid_samples(w, h))
    batch = hv.Batch(cameras=[cam], config=hv.batch_config(tile_stack_entries=256, tri_index_capacity=1 << 24))
    batch.render()
    want, costs = cam.tile_lists(), cam.tile_costs()
    batch.close()
    assert ((costs >= visits[0]) & (costs <= visits[1])).any()
    chunks = int(((want[0].astype(np.int64) + 127) // 128).sum())
    cam.set_samples(scenes.grid_samples(w, h))  # (a new sample set has no costs)
    batch = hv.Batch(cameras=[cam], config=hv.batch_config(tri_index_capacity=128 * chunks, pipeline=pipeline))
    for _ in range(3):
        batch.render()
        stats = batch.stats()
        assert stats["status"] == 0 and stats["pool_entries"] == 128 * chunks
        assert all(np.array_equal(a, b) for a, b in zip(cam.tile_lists(), want))
    batch.close()
    batch = hv.Batch(cameras=[cam], config=hv.batch_config(tri_index_capacity=128 * (chunks - 1), pipeline=pipeline))
    with pytest.raises(hv.HvvrError) as err:
        batch.render()
        batch.synchronize()
    assert err.value.code == _abi.HVVR_ERR_OVERFLOW
    batch.close()
    rc.close()
