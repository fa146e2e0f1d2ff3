"""The intersect's direct path for short lists (at most 32 entries and 8 subsamples) and its border with the
bounded one: hit IDs and depths equal the oracle's bit for bit where lists have none, one, an odd number,
32 and more entries, with coincident triangles (decided by list order), in both arithmetic modes."""
import numpy as np
import pytest

import hvvr_b200 as hv
from hvvr_b200 import scenes

from helpers import render_gpu, render_oracle

pytestmark = pytest.mark.gpu


def _scene(quads, boxes, doubled):
    sc = scenes.make_scene(quads, boxes, seed=6)
    sc.tri_shade = np.concatenate([sc.tri_shade, sc.tri_shade[:1]])  # (an odd number of triangles)
    if doubled:
        sc.tri_shade = np.concatenate([sc.tri_shade, sc.tri_shade])
    return hv.generate_topology(sc)


# longest: the range of the view's longest list, so that the case stays what it is for
@pytest.mark.parametrize("fp_mode", [hv.HVVR_FP_FMA, hv.HVVR_FP_STRICT])
@pytest.mark.parametrize("quads,boxes,doubled,w,h,msaa,longest", [
    (1, 0, False, 67, 45, 1, (1, 3)),
    (1, 1, False, 320, 200, 8, (2, 32)),
    (1, 1, True, 320, 200, 4, (3, 32)),
    (4, 3, False, 257, 129, 2, (5, 64)),
    (8, 20, False, 400, 300, 1, (33, 200)),
    (8, 20, True, 400, 300, 8, (33, 300)),
    (12, 40, False, 640, 400, 2, (33, 200)),
    (12, 40, False, 320, 200, 16, (33, 300)),  # (16 subsamples: always the bounded path)
])
def test_short_lists_change_no_hit(oracle, quads, boxes, doubled, w, h, msaa, longest, fp_mode):
    sc = _scene(quads, boxes, doubled)
    smp = scenes.barrel_samples(w, h)
    xf = scenes.camera_transform((2.0, 2.0, 8.0), (0.0, 0.0, 0.0))
    rc, cam = render_gpu(sc, smp, w, h, msaa, xf, fp_mode)
    counts, _ = cam.tile_lists()
    assert longest[0] <= counts.max() <= longest[1], counts.max()
    if longest[1] > 64:
        assert ((counts >= 1) & (counts <= 32)).any() and (counts > 32).any()
    ids, depth = cam.hits()
    fo = render_oracle(oracle, sc, smp, w, h, msaa, xf, fp_mode)
    assert np.array_equal(ids, fo.hit_ids)
    assert np.array_equal(depth.view(np.uint32), fo.depth.view(np.uint32))
    d = np.abs(cam.sample_colors().view(np.uint8).astype(int) - fo.colors.view(np.uint8).astype(int))
    assert d.max() <= 1
    assert (ids != 0xFFFFFFFF).any()
    rc.close()
