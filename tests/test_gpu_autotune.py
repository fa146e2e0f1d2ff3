"""The autotuner times what its batch's cull uses: with the breadth-first cull the configuration with and
without the pipeline, or as it is where no class would be pipelined, and the width and share that only the
sequential cull uses come back as they were; with tile_stack_entries all twenty candidates. The tuned batch
renders the same images."""
import numpy as np
import pytest

import hvvr_b200 as hv
from hvvr_b200 import scenes

from helpers import scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("msaa,w,h,entries,distinct", [
    (1, 200, 160, 0, 2),    # 256 tiles below 16 subsamples: piped or not
    (16, 200, 160, 0, 1),   # never piped
    (1, 1100, 1000, 0, 1),  # too many tiles
    (1, 96, 80, 0, 1),      # too few
    (2, 200, 160, 64, 20),
])
def test_candidates(msaa, w, h, entries, distinct):
    sc = scene("small")
    rc = hv.Raycaster()
    rc.create_model(sc)
    for light in sc.lights:
        rc.create_light(light)
    cam = rc.create_camera(scenes.viewport_for(w, h))
    cam.set_render_target(w, h)
    cam.set_samples(scenes.grid_samples(w, h))
    cam.set_camera_to_world(scenes.camera_transform())
    cam.set_msaa(msaa)
    rc.render()
    want = cam.image.copy()
    batch = hv.Batch(cameras=[cam], config=hv.batch_config(tile_stack_entries=entries, tile_cull_warps=2, heavy_divisor=3,
                                                           tri_index_capacity=1 << 22))
    cfg = batch.autotune(frames=3)
    assert cfg.frame_ms > 0 and cfg.tile_stack_entries == entries
    if entries == 0:
        assert cfg.tile_cull_warps == 2 and cfg.heavy_divisor == 3
        if distinct == 1:
            assert cfg.pipeline == 1  # as it was
    batch.render()
    assert np.array_equal(cam.image, want)
    batch.close()
    rc.close()
