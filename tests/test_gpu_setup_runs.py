"""The device sample setup at the edges of its sorted runs (one sample, a run of tiles, a block, a row
of blocks, one more and one less), with equal coordinates along either axis, with extents that are not
numbers (the tile rectangles' fold is then sequential), and over sample sets of changing size on one
camera whose frame is still running: beams, remap, lists and images equal the host setup's."""
import numpy as np
import pytest
import torch

import hvvr_b200 as hv
from hvvr_b200 import scenes

from helpers import scene

pytestmark = pytest.mark.gpu
W, H = 300, 260


def _samples(count, seed, columns=False):
    rng = np.random.default_rng(seed)
    s = np.repeat(scenes.grid_samples(W, H)[:1], count)
    s["position"] = rng.random((count, 2), dtype=np.float32)
    if columns:  # few distinct x: the minor axis decides within them
        s["position"][:, 0] = np.float32(0.125) * rng.integers(0, 9, count).astype(np.float32) - np.float32(0.0)
        s["position"][:, 1] = (rng.permutation(count).astype(np.float32) + np.float32(0.5)) / np.float32(count)
    s["pixel"][:, 0] = np.clip(s["position"][:, 0] * W, 0, W - 1).astype(np.uint32)
    s["pixel"][:, 1] = np.clip(s["position"][:, 1] * H, 0, H - 1).astype(np.uint32)
    return s


def _camera(setup):
    sc = scene("small")
    rc = hv.Raycaster(sample_setup=setup)
    rc.create_model(sc)
    for light in sc.lights:
        rc.create_light(light)
    cam = rc.create_camera(scenes.viewport_for(W, H))
    cam.set_render_target(W, H)
    cam.set_camera_to_world(scenes.camera_transform())
    cam.set_msaa(2)
    return rc, cam


def _read(cam):
    beams = cam.beams()  # (which not-a-number a CPU or GPU writes differs; everything else is compared as bits)
    return (np.where(np.isnan(beams), np.float32(np.nan), beams).view(np.uint32), cam.sample_remap(), *cam.block_stacks(), *cam.tile_lists(), cam.sample_colors())


def test_setup_at_run_edges_equals_host():
    dev, host = _camera(hv.HVVR_SETUP_DEVICE), _camera(hv.HVVR_SETUP_HOST)
    stream = torch.cuda.Stream()
    for k, count in enumerate([1, 2, 127, 1023, 1025, 8191, 8192, 8193, 16384, 40000, 65537, 300, 24577]):
        smp = _samples(count, 10 + k, columns=k % 3 == 2)
        if k % 4 == 3:
            smp["major"][::97] = np.nan
        for rc, cam in (dev, host):
            cam.set_samples(smp)
            on_host = cam.prepare()
            rc.render(stream=stream.cuda_stream)
            assert on_host == (cam is host[1])
        for a, b in zip(_read(dev[1]), _read(host[1])):
            assert np.array_equal(a, b), count
    dev[0].close()
    host[0].close()
