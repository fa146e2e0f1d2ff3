"""The block cull (node tests ahead of the visits that need them) against the oracle's block stacks,
entry for entry: trees of one node, stacks that end below and at the 60-entry cut, and nodes of no
extent along the view's axis, whose stack key equals a leaf group's."""
import numpy as np
import pytest

import hvvr_b200 as hv
from hvvr_b200 import scenes

from helpers import render_gpu, render_oracle, scene

pytestmark = pytest.mark.gpu


def _scene(name):
    if name == "one node":
        return hv.generate_topology(scenes.make_scene(1, 0, seed=4))
    if name == "flat":  # every box is flat, seen along that axis
        sc = scenes.make_scene(40, 1, seed=2)
        sc.verts["pos"][:, 1] = 0.0
        return hv.generate_topology(sc)
    return scene(name)


@pytest.mark.parametrize("name,w,h,eye,target,largest", [
    ("one node", 64, 48, (0.0, 3.0, 9.0), (0.0, 0.0, 0.0), (1, 1)),
    ("flat", 200, 150, (0.3, 9.0, 0.5), (0.0, 0.0, 0.0), (1, 63)),
    ("small", 257, 131, (0.0, 2.0, 10.0), (0.0, 0.0, 0.0), (2, 63)),
    ("c1", 640, 480, (6.0, 2.5, -7.0), (0.0, 0.0, 0.0), (60, 63)),
    ("c2", 96, 80, (-5.0, 4.0, 6.0), (0.0, 0.0, 0.0), (60, 63)),
])
def test_block_stacks_equal_oracle(oracle, name, w, h, eye, target, largest):
    sc = _scene(name)
    smp = scenes.barrel_samples(w, h)
    xf = scenes.camera_transform(eye, target)
    rc, cam = render_gpu(sc, smp, w, h, 1, xf)
    fo = render_oracle(oracle, sc, smp, w, h, 1, xf)
    sizes, entries = cam.block_stacks()
    assert largest[0] <= sizes.max() <= largest[1]
    assert np.array_equal(sizes, fo.block_sizes) and np.array_equal(entries, fo.block_entries)
    rc.close()
