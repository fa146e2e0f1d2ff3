"""A server view's sample setup leaves nothing on the device beside the view itself: the memory that
add_view takes with the device setup, which works in a scratch of about 60 bytes a sample, is what it
takes with the host setup, which has none."""
import pytest
import torch

import hvvr_b200 as hv
from hvvr_b200 import scenes

from helpers import scene

pytestmark = pytest.mark.gpu
W, H = 1024, 1000


def _taken(setup):
    sc = scene("small")
    rc = hv.Raycaster(sample_setup=setup)
    rc.create_model(sc)
    for light in sc.lights:
        rc.create_light(light)
    server = hv.Server([rc], hv.server_config(slots=1, latency_slots=0, slot_list_capacity=1 << 20))
    vp = scenes.viewport_for(64, 48)
    server.add_view(0, vp, scenes.grid_samples(64, 48), 64, 48)  # (the first setup loads its kernels)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    server.add_view(0, scenes.viewport_for(W, H), scenes.grid_samples(W, H), W, H)
    torch.cuda.synchronize()
    taken = before - torch.cuda.mem_get_info()[0]
    server.close()
    rc.close()
    return taken


def test_view_setup_leaves_only_the_view():
    host, device = _taken(hv.HVVR_SETUP_HOST), _taken(hv.HVVR_SETUP_DEVICE)
    assert host > 48 * W * H  # the beams
    assert abs(device - host) <= 8 << 20  # (allocations are rounded to 2 MiB)
