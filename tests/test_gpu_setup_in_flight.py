"""A new sample set for a camera whose frames are still running on another stream: the setup writes the
buffers that they read (beams, tile frusta, and the tile costs that order their tiles), so it waits for
them. Lists and images equal those of a camera that never had a frame running, pinhole and foveated."""
import numpy as np
import pytest
import torch

import hvvr_b200 as hv
from hvvr_b200 import _abi, scenes

from helpers import scene

pytestmark = pytest.mark.gpu
W, H = 320, 288


def _camera(foveated):
    sc = scene("c1")
    spec = hv.foveated_spec(1.0, 35.0, 0.03, 0.06, mode=_abi.HVVR_MODE_FOVEATED_POLAR) if foveated else None
    rc = hv.Raycaster(spec=spec) if foveated else hv.Raycaster()
    rc.create_model(sc)
    for light in sc.lights:
        rc.create_light(light)
    cam = rc.create_camera(scenes.viewport_for(W, H))
    image = torch.zeros((H, W), dtype=torch.int32, device="cuda")
    cam.set_render_target(W, H, device_ptr=image.data_ptr())
    cam.set_camera_to_world(scenes.camera_transform((5.0, 3.0, 8.0), (0.0, 0.0, 0.0)))
    cam.set_msaa(8)
    return rc, cam, image


def _sets(foveated):
    # (a foveated camera's own samples only bound its screen)
    return (scenes.grid_samples(W, H), scenes.barrel_samples(W, H), scenes.grid_samples(W, H))


def _read(cam, image, foveated):
    lists = cam.tile_lists()
    torch.cuda.synchronize()
    return (*lists, cam.sample_colors()) + (() if foveated else (image.cpu().numpy(),))


@pytest.mark.parametrize("foveated", [False, True])
def test_setup_waits_for_running_frames(foveated):
    want = []
    for smp in _sets(foveated):
        rc, cam, image = _camera(foveated)
        cam.set_samples(smp)
        rc.render()
        rc.synchronize()
        want.append(_read(cam, image, foveated))
        rc.close()
    rc, cam, image = _camera(foveated)
    stream = torch.cuda.Stream()
    for smp, expected in zip(_sets(foveated), want):
        cam.set_samples(smp)
        cam.prepare()  # (on the raycaster's own stream, while frames of the set before it run on `stream`)
        rc.render(stream=stream.cuda_stream)
        stream.synchronize()
        for a, b in zip(_read(cam, image, foveated), expected):
            assert np.array_equal(a, b)
        for _ in range(6):
            rc.render(stream=stream.cuda_stream)
    rc.synchronize()
    stream.synchronize()
    rc.close()


def test_new_samples_start_from_a_black_image():
    """Pixels that no sample of the new set maps to are black, not what the set before drew there."""
    sc = scene("c1")
    rc = hv.Raycaster()
    rc.create_model(sc)
    for light in sc.lights:
        rc.create_light(light)
    cam = rc.create_camera(scenes.viewport_for(W, H))
    cam.set_render_target(W, H)
    cam.set_camera_to_world(scenes.camera_transform())
    cam.set_msaa(4)
    full = scenes.grid_samples(W, H)
    for shape in ((W, H), (H, W)):  # as many pixels in another shape
        cam.set_render_target(*shape)
        cam.set_samples(full)
        rc.render()
        rc.synchronize()
        assert (cam.image != 0).sum() > 0
        half = full[full["pixel"][:, 0] < 100]
        cam.set_samples(half)
        rc.render()
        rc.synchronize()
        drawn = np.zeros(cam.image.shape, bool)
        on = half[(half["pixel"][:, 0] < shape[0]) & (half["pixel"][:, 1] < shape[1])]
        drawn[on["pixel"][:, 1], on["pixel"][:, 0]] = True
        assert (cam.image[~drawn] == 0).all() and (cam.image[drawn] != 0).any()
    rc.close()
