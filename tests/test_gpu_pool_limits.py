"""A voxel-block pool that is too small for the scene: the blocks that it holds
are integrated as in a roomy one, and nothing beyond its last slot is touched.

The device counter of handed-out slots keeps counting requests once the pool is
full; the capacities here are no multiple of the 256 slots that a CTA of the
visit list takes, so that its last CTA has threads beyond the pool."""
import numpy as np
import pytest

from mid_fusion_b200 import build
from mid_fusion_b200.capi import STATUS_POOL_FULL, Context
from mid_fusion_b200.scene import generalize_masks, make_scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def _run(s, pool, frames=3):
    ctx = Context(s.width, s.height, k=s.k, pool_blocks=pool)
    inst = s.instances[0]
    ctx.add_instance(inst.size, inst.dim, np.eye(4), inst.label)
    ctx.set_camera_pose(s.cam_poses[0])
    d, rgb, lab = s.render(0)
    ctx.upload(d, rgb, generalize_masks(lab, [inst.label]))
    visited = []
    for _ in range(frames):
        ctx.integrate([0])
        visited.append(ctx.frame_stats())
    keys, coords, active, vox = ctx.blocks(0)
    status = ctx.status()
    ctx.close()
    return keys, active, vox, status, visited


@pytest.mark.parametrize("pool", [1, 44, 255, 257, 300])
def test_full_pool_keeps_to_its_slots(pool):
    s = make_scene("room", 160, 120, n_frames=1, seed=4, bg_size=256, noise=False)
    keys, active, vox, status, _ = _run(s, 1 << 13)
    assert status == 0 and len(keys) > 320
    k, a, v, st, stats = _run(s, pool)
    assert st & STATUS_POOL_FULL
    assert len(k) == pool and len(np.unique(k)) == pool
    assert stats[0]["visited_blocks"] == pool   # a new block is active
    for f in stats:
        assert f["pool_blocks"] == pool and f["visited_blocks"] <= pool
    at = {int(x): i for i, x in enumerate(keys)}
    where = np.array([at[int(x)] for x in k])   # every held block is one of the roomy pool's
    assert np.array_equal(a, active[where])
    for f in ("x", "y", "r", "g", "b", "c", "fg", "w"):
        assert np.array_equal(v[f], vox[f][where]), f
