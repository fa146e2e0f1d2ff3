"""The breadth-first cull's order among components whose sort keys are all equal: a root whose own key
exceeds every key below it holds the largest key on every path, and what comes first is then decided
component by component. One root of a whole tree in one tile, with a key above and one below all others:
the lists are the same (a root alone is popped first whatever its key), and the ties' order costs no
multiple of the cull."""
import ctypes as C

import numpy as np
import pytest
import torch

import hvvr_b200 as hv
from hvvr_b200 import _abi, scenes

from helpers import render_gpu

pytestmark = pytest.mark.gpu
W, H, TILES = 64, 48, 64


# components in one run: within a warp's store, just above the counted runs' length, in a CTA's and an SM's store
@pytest.mark.parametrize("grid,boxes", [(20, 30), (28, 60), (40, 160), (84, 100), (150, 600)])
def test_one_run_of_ties(oracle, grid, boxes):
    sc = hv.generate_topology(scenes.make_scene(grid, boxes, seed=3))
    smp = scenes.grid_samples(W, H)
    xf = scenes.camera_transform((0.0, 900.0, 1500.0), (0.0, 0.0, 0.0))
    rc, cam = render_gpu(sc, smp, W, H, 1, xf, capture=False)
    counts, _ = cam.tile_lists()
    tile = int(np.argmax(counts))
    assert counts[tile] == sc.tri_count  # the whole tree passes this tile's tests
    rays = oracle.render(sc, smp, xf, scenes.viewport_for(W, H), W, H, 1, want=("tile_rays",)).tile_rays
    rays = np.repeat(np.asarray(rays)[tile:tile + 1], TILES, 0)
    nodes = rc.scene_nodes()

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).copy()).cuda()

    total = int(counts[tile]) * TILES
    d_nodes, d_rays, d_sizes = dev(nodes), dev(rays), dev(np.ones(TILES // 64, np.uint32))
    lists, times = [], []
    for key in (-1e9, 1e9):
        stacks = np.zeros((TILES // 64, 64, 3), np.uint32)
        stacks[:, 0, 0] = np.float32(key).view(np.uint32)
        d_stacks = dev(stacks)
        d_counts = torch.zeros(TILES, dtype=torch.int32, device="cuda")
        d_idx = torch.zeros(total, dtype=torch.int32, device="cuda")
        args = _abi.TileCullArgs(d_nodes.data_ptr(), len(nodes), d_rays.data_ptr(), TILES, d_stacks.data_ptr(),
                                 d_sizes.data_ptr(), xf)
        n = C.c_uint64(0)
        ms = []
        for _ in range(9):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            start.record()
            assert hv.lib().hvvr_tile_cull_static(C.c_void_p(C.addressof(args)), C.c_void_p(d_counts.data_ptr()),
                                                  C.c_void_p(d_idx.data_ptr()), total, C.byref(n), None) == 0
            end.record()
            torch.cuda.synchronize()
            ms.append(start.elapsed_time(end))
        assert n.value == total
        lists.append(d_idx.cpu().numpy())
        times.append(sorted(ms)[len(ms) // 2])
    assert np.array_equal(lists[0], lists[1])
    assert np.array_equal(np.sort(lists[0][:sc.tri_count]), np.arange(sc.tri_count))
    assert times[1] < 2.5 * times[0]
    rc.close()
