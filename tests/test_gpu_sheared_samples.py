"""The intersect's boxes of beams lie along axes made from one sample's footprint. A viewport scaled very
unequally shears the footprints of rotated ellipses until their two directions are nearly parallel, and
footprints may have no extent along one of them: the boxes have to hold the beams all the same, so hit
IDs and depths equal the oracle's bit for bit."""
import numpy as np
import pytest

import hvvr_b200 as hv
from hvvr_b200 import _abi, scenes

from helpers import render_gpu, render_oracle, scene

pytestmark = pytest.mark.gpu
W, H = 96, 80


def _samples(angle, radius, major):
    smp = scenes.grid_samples(W, H)
    smp["minor"][:, 0] = np.float32(radius * np.cos(angle))
    smp["minor"][:, 1] = np.float32(radius * np.sin(angle))
    smp["major"] = np.float32(major)
    return smp


def _viewport(half_width, half_height):
    vp = _abi.FloatRect()
    vp.lower.x, vp.lower.y, vp.upper.x, vp.upper.y = -half_width, -half_height, half_width, half_height
    return vp


@pytest.mark.parametrize("fp_mode", [hv.HVVR_FP_FMA, hv.HVVR_FP_STRICT])
@pytest.mark.parametrize("half_width,half_height,angle,radius,major,msaa", [
    (1.0, 1e-2, 0.25 * np.pi, 1e-3, 1e-3, 8),
    (1.0, 1e-3, 0.25 * np.pi, 1e-7, 1e-7, 1),
    (1.0, 1e-4, 0.25 * np.pi, 1e-7, 1e-7, 4),
    (1.0, 1e-5, 0.25 * np.pi, 1e-7, 1e-7, 2),
    (1.0, 1e-7, 0.25 * np.pi, 1e-9, 1e-9, 1),
    (1e-4, 1.0, 0.25 * np.pi, 1e-7, 1e-7, 1),
    (1.0, 1e-4, 0.1, 1e-7, 3e-7, 1),
    (0.8, 0.6, 0.3, 1e-3, 0.0, 4),       # a line: one direction is zero
])
def test_sheared_footprints_change_no_hit(oracle, half_width, half_height, angle, radius, major, msaa, fp_mode):
    sc = scene("c1")
    smp, vp = _samples(angle, radius, major), _viewport(half_width, half_height)
    xf = scenes.camera_transform((5.0, 3.0, 8.0), (-1.0, 0.3, 0.4))
    rc, cam = render_gpu(sc, smp, W, H, msaa, xf, fp_mode, viewport=vp)
    ids, depth = cam.hits()
    fo = render_oracle(oracle, sc, smp, W, H, msaa, xf, fp_mode, viewport=vp)
    assert np.array_equal(ids, fo.hit_ids)
    assert np.array_equal(depth.view(np.uint32), fo.depth.view(np.uint32))
    assert (ids != 0xFFFFFFFF).any()
    rc.close()
