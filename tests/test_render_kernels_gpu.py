"""GPU: the ray marcher over every kind of brick edge, against the oracle's scalar march."""
import math

import numpy as np
import pytest

from csvb200.camera import SLOT_DTYPE, SLOT_EMPTY, SLOT_MISSING, camera_uniform, orbit

pytestmark = pytest.mark.gpu


# edge 1 (one voxel, no steps inside), the decoder's edges, the largest whose voxels all have a Morton neighbour in
# 32 bits, and 1024, which has not; bricks at several LODs, some empty, some missing
@pytest.mark.parametrize("brick", [1, 2, 16, 64, 128, 512, 1024])
def test_march_by_brick_edge(codec, oracle, brick):
    import torch
    rng = np.random.default_rng(brick)
    bpa, top = 4, brick.bit_length() - 1
    n, grid = bpa ** 3, float(bpa * brick)
    lods = rng.integers(0, min(top, 5) + 1, n).astype(np.uint32)
    sizes = 8 ** lods.astype(np.uint64)
    offs = np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.uint64)
    keys = np.unique(rng.integers(1, 2 ** 62, 40, dtype=np.uint64))
    pool = np.concatenate([np.zeros(60, np.uint64), keys, keys[:3] + np.uint64(1)])  # mostly 0, some labels not in the table
    labels = pool[rng.integers(0, len(pool), int(sizes.sum()))]
    slots = np.zeros(n, SLOT_DTYPE)
    slots["offset"], slots["lod"] = offs, lods
    slots["flags"] = np.where(rng.random(n) < 0.15, SLOT_EMPTY, np.where(rng.random(n) < 0.15, SLOT_MISSING, 0))
    cols = oracle.transfer_function(keys)
    d_slots = torch.from_numpy(slots.view(np.uint8).copy()).cuda()
    d_labels = torch.from_numpy(labels.view(np.int64)).cuda()
    d_keys, d_cols = torch.from_numpy(keys.view(np.int64)).cuda(), torch.from_numpy(cols.view(np.int32)).cuda()
    W, H = 75, 50
    out = torch.empty(W * H, dtype=torch.int64, device="cuda")
    dep = torch.empty(W * H, dtype=torch.float32, device="cuda")
    img = torch.empty(W * H, dtype=torch.int32, device="cuda")
    for r, yaw, pitch in ((1.4, 0.7, 0.3), (0.3, -2.0, -0.4), (2.0, 3.5, 1.3)):
        pos, d = orbit((grid / 2,) * 3, r * grid, yaw, pitch)
        cam = camera_uniform(pos, d, math.pi / 3)
        codec.render(cam, W, H, grid, brick, bpa, d_slots, d_labels, out, dep)
        ref_l, ref_d, _ = oracle.render(cam, W, H, grid, brick, bpa, slots, labels)
        assert np.array_equal(out.cpu().numpy().view(np.uint64).reshape(H, W), ref_l)
        assert np.array_equal(dep.cpu().numpy().view(np.uint32).reshape(H, W), ref_d.view(np.uint32))
        light = codec.lighting()
        codec.render_rgba(cam, W, H, grid, brick, bpa, d_slots, d_labels, d_keys, d_cols, light, img)
        ref = oracle.render_rgba(cam, W, H, grid, brick, bpa, slots, labels, keys, cols, light.as_array())
        a = img.cpu().numpy().view(np.uint8).reshape(H, W, 4).astype(int)
        b = ref.view(np.uint8).reshape(H, W, 4).astype(int)
        # powf and expf are the device's: as in the colour tests, two counts on all but one pixel in 200
        assert (np.abs(a - b).max(axis=2) <= 2).mean() >= 0.995
