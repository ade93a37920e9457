"""Edges of the kernels' tiles, rows and lists on the GPU.

* The one-launch GN against the host-driven loop (whose steps run on the host):
  the same poses bit for bit, at frame sizes that tiles, 32-pixel segments and
  rows of CTAs do not divide, from fewer tiles than CTAs to several per CTA,
  with one to many objects (also one that is out of view), every row set and
  one to four pyramid levels.
* Allocation, integration and raycast against the oracle, bit for bit: volumes
  from the smallest size up, one ray sample and many, rays that leave the
  volume.
* The mesh's block list and offsets over block tables of one and of many
  chunks, against the exported voxels' own block order.
"""
import numpy as np
import pytest

import _oracle as O
from mid_fusion_b200 import build
from mid_fusion_b200.capi import Context
from mid_fusion_b200.scene import generalize_masks, make_scene
from test_gpu_volume import _assert_volume_equal

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def _track(s, frames, batched, move=None, **kw):
    ctx = Context(s.width, s.height, k=s.k, pool_blocks=1 << 15, batched=batched, **kw)
    for i, (inst, T) in enumerate(zip(s.instances, s.volume_poses(0))):
        T = np.array(T)
        if i == move:   # out of view from the start
            T[:3, 3] += 30.0
        ctx.add_instance(inst.size, inst.dim, T, inst.label)
    ctx.set_camera_pose(s.cam_poses[0])
    n = len(s.instances)
    out = []
    for f, (d, rgb, lab) in enumerate(frames):
        ctx.upload(d, rgb)
        ctx.upload_labels(lab)
        ctx.preprocess()
        if f:
            ctx.track_camera(list(range(1, n)))
            if n > 1:
                ctx.track_objects(list(range(1, n)))
        ctx.integrate(list(range(n)))
        ctx.raycast()
        ctx.set_ref_from_current()
        out.append([ctx.camera_pose()] + [ctx.instance_pose(i) for i in range(n)])
    assert ctx.status() & 32 == 0   # no barrier timed out
    sums = [ctx.track_info(i)[1][:, :29] for i in range(n)]
    ctx.close()
    return np.array(out), sums


@pytest.mark.parametrize("W,H,objects,move,kw", [
    (41, 31, 1, None, dict(robust="none")),
    (97, 65, 2, None, dict(robust="huber", use_rgb=False)),
    (161, 119, 3, 2, dict(robust="tukey")),
    (319, 241, 5, None, dict(robust="cauchy", use_icp=False)),
    (333, 250, 4, None, dict(robust="huber", gn_iterations=(4, 3, 3, 2))),
    (640, 97, 3, None, dict(robust="huber", gn_iterations=(3,))),
    (801, 601, 2, None, dict(robust="huber", gn_iterations=(2, 2))),
])
def test_one_launch_gn_equals_host_loop(W, H, objects, move, kw):
    s = make_scene("multi", W, H, n_frames=3, seed=13, bg_size=128, obj_size=64,
                   n_objects=objects)
    frames = [s.render(f) for f in range(3)]
    a, sa = _track(s, frames, True, move, **kw)
    b, sb = _track(s, frames, False, move, **kw)
    assert np.array_equal(a, b, equal_nan=True)
    for x, y in zip(sa, sb):
        assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("size,dim,mu,offset", [
    (16, 5.12, 0.1, 0.0),      # two blocks per side, one sample per ray
    (32, 1.28, 0.1, 1.5),      # the surface leaves the volume
    (64, 5.12, 0.02, 0.0),
    (256, 1.28, 0.1, 1.9),     # 40 samples per ray, many rays leave
    (512, 2.56, 0.2, 1.0),     # 80 samples per ray
    (1024, 5.12, 0.1, 0.0),
])
def test_allocation_edges_match_oracle(size, dim, mu, offset):
    s = make_scene("multi", 75, 53, n_frames=2, seed=4, n_objects=0)
    T_w_o = np.eye(4, dtype=np.float32)
    T_w_o[:3, 3] = offset
    orc = O.oracle()
    ctx = Context(s.width, s.height, k=s.k, pool_blocks=1 << 15, mu=mu)
    ctx.add_instance(size, dim, T_w_o, 0)
    vol = orc.volume(size, dim)
    for f in range(2):
        depth, rgb, lab = s.render(f)
        masks = generalize_masks(lab, [0])
        T = s.cam_poses[f].astype(np.float32)
        ctx.set_camera_pose(T)
        ctx.upload(depth, rgb, masks)
        ctx.integrate([0])
        vol.integrate(depth, rgb.astype(np.float32) / np.float32(255.0), masks[0], T, T_w_o, s.k,
                      mu)
    assert ctx.status() & 1 == 0   # the pool was not full
    _assert_volume_equal(ctx, 0, vol)


@pytest.mark.parametrize("size", [32, 256, 1024])
def test_mesh_block_order(size):
    """Triangles come in Morton order of their blocks, whatever the number of
    chunks that the block table is listed in, and in device memory too."""
    s = make_scene("multi", 160, 120, n_frames=1, seed=4, n_objects=0)
    ctx = Context(s.width, s.height, k=s.k, pool_blocks=1 << 15)
    ctx.add_instance(size, 5.12, np.eye(4, dtype=np.float32), 0)
    d, rgb, lab = s.render(0)
    ctx.set_camera_pose(s.cam_poses[0])
    ctx.upload(d, rgb, generalize_masks(lab, [0]))
    for _ in range(5):
        ctx.integrate([0])
    tri = ctx.mesh(0, float_bounds=True)
    assert np.array_equal(tri, ctx.mesh(0, float_bounds=True))
    keys, coords, _, _ = ctx.blocks(0, with_voxels=False)
    if size > 32:
        assert len(tri) > 100
    # the block of a triangle's cell: floor of its smallest corner
    vox = np.floor(tri.min(1).astype(np.float64) * (size / 5.12) + 1e-4).astype(np.int64) // 8
    where = {tuple(c // 8): i for i, c in enumerate(coords)}
    order = np.array([where.get(tuple(v), -1) for v in vox])
    known = order[order >= 0]
    assert len(known) >= 0.9 * len(tri)
    assert np.mean(np.diff(known) >= 0) > 0.98   # up to corners on a block's face


def _half(a):
    """The reference's robust half-sampling in float32, element by element in
    its order (centre, right, below, diagonal)."""
    h, w = a.shape[0] // 2, a.shape[1] // 2
    c = a[0:2 * h:2, 0:2 * w:2]
    s = np.zeros_like(c)
    t = np.zeros_like(c)
    for dy in (0, 1):
        for dx in (0, 1):
            v = a[dy:2 * h:2, dx:2 * w:2]
            near = np.abs(v - c) < np.float32(np.float32(0.1) * 3)
            s = np.where(near, s + np.float32(1), s)
            t = np.where(near, t + v, t)
    return t / s


@pytest.mark.parametrize("W,H,levels", [(17, 19, 2), (97, 65, 3), (161, 119, 4), (350, 267, 4),
                                        (64, 48, 1)])
def test_pyramid_levels_at_ragged_sizes(W, H, levels):
    """Every level of depth and intensity is the half-sampled finer level bit
    for bit, and the vertex planes (live and rendered reference) have the
    depth as z where there is one, at sizes that the 16 x 16 tiles do not
    divide."""
    s = make_scene("multi", W, H, n_frames=2, seed=5, n_objects=0)
    ctx = Context(W, H, k=s.k, pool_blocks=1 << 14, gn_iterations=(2,) * levels)
    ctx.add_instance(128, 5.12, np.eye(4, dtype=np.float32), 0)
    ctx.set_camera_pose(s.cam_poses[0])
    for f in range(2):
        d, rgb, lab = s.render(f)
        d = np.array(d, np.float32)
        d[H // 3:H // 3 + 3, :W // 2] = 0   # missing depths
        ctx.upload(d, rgb)
        ctx.upload_labels(lab)
        ctx.preprocess()
        if f:
            ctx.track_camera([])
        ctx.integrate([0])
        ctx.raycast()
        if f == 0:
            ctx.set_ref_from_current()
    for which in (0, 1):
        for l in range(1, levels):
            fine = ctx.pyramid(l - 1, which)
            got = ctx.pyramid(l, which)
            assert np.array_equal(got, _half(fine)[:got.shape[0], :got.shape[1]]), (which, l)
    ref = ctx.pyramid(0, 7)[..., 2]
    for l in range(levels):
        d = ctx.pyramid(l, 0)
        assert np.array_equal(ctx.pyramid(l, 2)[..., 2], np.where(d > 0, d, np.float32(0)))
        if l:
            ref = _half(ref)
        got = ctx.pyramid(l, 7)[..., 2]
        assert np.array_equal(got, np.where(ref > 0, ref, np.float32(0))[:got.shape[0],
                                                                        :got.shape[1]]), l
    ctx.close()
