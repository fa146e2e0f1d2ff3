"""The sequential tile cull (tile_stack_entries) in every form its settings give it: CTAs of one to eight
warps, persistent or a tile a warp, with and without the heavy part on its own stream, piped to the shade or
before it, with a resident-CTA cap, replayed from a graph or not. Lists, hits, colours and images equal the
breadth-first cull's over frames (the later ones in last frame's cost order), and a list pool that is too
small is reported."""
import numpy as np
import pytest

import hvvr_b200 as hv
from hvvr_b200 import _abi, scenes

from helpers import scene

pytestmark = pytest.mark.gpu
VIEWS = (("c1", 256, 224, "barrel", 8), ("c1", 192, 160, "grid", 1), ("small", 160, 176, "barrel", 16))


def _views():
    rcs, cams = {}, []
    for k, (name, w, h, kind, msaa) in enumerate(VIEWS):
        if name not in rcs:
            rcs[name] = hv.Raycaster()
            rcs[name].create_model(scene(name))
            for light in scene(name).lights:
                rcs[name].create_light(light)
        cam = rcs[name].create_camera(scenes.viewport_for(w, h))
        cam.set_render_target(w, h)
        cam.set_samples((scenes.grid_samples if kind == "grid" else scenes.barrel_samples)(w, h))
        cam.set_msaa(msaa)
        cam.set_capture(hv.HVVR_CAPTURE_HITS)
        cam.set_camera_to_world(scenes.camera_transform((0.4 * k, 2.0, 10.0), (0.0, 0.2 * k, 0.0)))
        cams.append(cam)
    return list(rcs.values()), cams


def _read(cams):
    return [x for cam in cams for x in (*cam.tile_lists(), *cam.hits(), cam.tile_costs(), cam.sample_colors(), cam.image.copy())]


def test_every_form_equals_breadth_first():
    rcs, cams = _views()

    def frames(**cfg):
        batch = hv.Batch(rcs, hv.batch_config(tri_index_capacity=1 << 22, **cfg))
        out = []
        for _ in range(3):
            batch.render()
            assert batch.stats()["status"] == 0
            out.append(_read(cams))
        batch.close()
        return out

    want = frames()[0]
    for cfg in (dict(tile_cull_warps=1, heavy_divisor=8), dict(tile_cull_warps=4, heavy_divisor=8, pipeline=0),
                dict(tile_cull_warps=8, heavy_divisor=4, pipeline=0, use_graph=0), dict(tile_cull_warps=2, heavy_divisor=0),
                dict(tile_cull_warps=2, heavy_divisor=0, pipeline=0), dict(tile_cull_warps=1, tile_cull_persistent=0),
                dict(tile_cull_warps=4, tile_cull_persistent=0, pipeline=0), dict(tile_cull_warps=1, tile_cull_ctas_per_sm=2),
                dict(tile_cull_warps=4, heavy_divisor=16, timing=1, pipeline=0)):
        for got in frames(tile_stack_entries=256, **cfg):
            assert all(np.array_equal(a.view(np.uint32), b.view(np.uint32)) for a, b in zip(got, want)), cfg
    for rc in rcs:
        rc.close()


@pytest.mark.parametrize("pipeline", [1, 0])
def test_small_pool_is_reported(pipeline):
    rcs, cams = _views()
    batch = hv.Batch(rcs, hv.batch_config(tile_stack_entries=256, tri_index_capacity=4096, pipeline=pipeline))
    with pytest.raises(hv.HvvrError) as err:
        batch.render()
        batch.synchronize()
    assert err.value.code == _abi.HVVR_ERR_OVERFLOW
    batch.close()
    for rc in rcs:
        rc.close()
