"""The normal equations that tracking itself reduces, on the GPU.

mf_track_eval (compared with the FP64 oracle in test_gpu_track.py) sums whole
tiles in a kernel of its own.  Tracking sums in its one-launch loops, where the
camera's rows are spread over CTAs and an object's pixels are taken in 32-pixel
segments, those left out that cannot hold a valid row.  The last sums of each
level (mf_track_info) are compared here with mf_track_eval at the pose that
they were evaluated at: a tile, segment or row that one of the two loses shows
as another number of rows.

Both evaluate the same FP32 rows and add a thread's rows of a tile in the same
order in FP32; the FP64 additions that follow differ in their order only.  N
additions of terms t in another order differ by at most 2 N 2^-53 sum |t|, and
sum |t| is at most the geometric mean of the two sums of squares (Cauchy); with
N below 10^6 that is 3e-10 of it.
"""
import numpy as np
import pytest

from mid_fusion_b200 import build
from mid_fusion_b200.capi import Context
from mid_fusion_b200.scene import make_scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def _compare(ctx, slot, level, counts):
    """The sums of the problem's last evaluation at `level` against
    mf_track_eval's; returns the number of rows."""
    import torch
    live = ctx.track_info(slot)[1][level].copy()
    codes = torch.empty(2 * ctx.W * ctx.H, dtype=torch.int8, device="cuda")
    pose = ctx.track_results(slot, codes.data_ptr())
    want = ctx.track_eval(slot, level, pose)
    assert live[28] == want[28], (slot, level, live[28], want[28])
    if counts:
        assert np.array_equal(live[29:], want[29:]), (slot, level)
    elif want[28]:
        assert np.all(live[29:] <= want[29:]), (slot, level)
    # sum w e^2 is at most 6 times the sum of the losses (Tukey; 2 for the others)
    diag = np.array([want[7 + i * 6 - i * (i - 1) // 2] for i in range(6)])
    scale = [want[0]] + [np.sqrt(6 * want[0] * d) for d in diag]
    scale += [np.sqrt(diag[i] * diag[j]) for i in range(6) for j in range(i, 6)]
    err = np.abs(live[:28] - want[:28])
    assert np.all(err <= 3e-10 * np.array(scale)), (slot, level, err, scale)
    return int(want[28])


def _second_frame(s, world=np.eye(4), **kw):
    """The context after tracking the second of two frames, every pose given
    in the frame `world`."""
    ctx = Context(s.width, s.height, k=s.k, pool_blocks=1 << 15, **kw)
    n = len(s.instances)
    for inst, T in zip(s.instances, s.volume_poses(0)):
        ctx.add_instance(inst.size, inst.dim, world @ T, inst.label)
    ctx.set_camera_pose(world @ s.cam_poses[0])
    for f in range(2):
        d, rgb, lab = s.render(f)
        ctx.upload(d, rgb)
        ctx.upload_labels(lab)
        ctx.preprocess()
        if f:
            ctx.track_camera(list(range(1, n)))
            if n > 1:
                ctx.track_objects(list(range(1, n)))
            return ctx
        ctx.integrate(list(range(n)))
        ctx.raycast()
        ctx.set_ref_from_current()


@pytest.mark.parametrize("W,H,objects,level,kw", [
    (41, 31, 1, 0, dict(robust="none")),
    (97, 65, 2, 1, dict(robust="huber")),
    (97, 65, 2, 0, dict(robust="huber", use_rgb=False)),
    (161, 119, 3, 3, dict(robust="tukey")),
    (161, 119, 3, 0, dict(robust="tukey")),
    (319, 241, 5, 0, dict(robust="cauchy", use_icp=False)),
    (333, 250, 4, 2, dict(robust="huber")),
    (640, 97, 3, 0, dict(robust="cauchy")),
    (640, 480, 3, 0, dict(robust="huber")),
    (640, 480, 3, 1, dict(robust="huber")),
    (801, 601, 2, 0, dict(robust="cauchy")),
])
def test_live_sums_equal_the_evaluation(W, H, objects, level, kw):
    s = make_scene("multi", W, H, n_frames=2, seed=13, bg_size=128, obj_size=64,
                   n_objects=objects)
    ctx = _second_frame(s, gn_iterations=(0,) * level + (3,), **kw)
    rows = [_compare(ctx, i, level, counts=i == 0) for i in range(objects + 1)]
    assert rows[0] > 0.2 * (W >> level) * (H >> level)
    assert W < 97 or any(rows[1:])
    assert ctx.status() & 32 == 0
    ctx.close()


def _far_wall_to_origin(s, px, normal):
    """The rigid motion of the world that brings the point of the far wall (z =
    room_hi[2]) that frame 1 sees at column px, middle row, to the origin, and
    the wall's normal (facing the room) to `normal` times the x axis."""
    fx, fy, cx, cy = [float(v) for v in s.k]
    T = s.cam_poses[1]
    d = T[:3, :3] @ np.array([(px - cx) / fx, 0.0, 1.0])
    p = T[:3, 3] + d * (s.room_hi[2] - T[2, 3]) / d[2]
    R = np.array([[0, 0, -normal], [0, 1, 0], [normal, 0, 0]], np.float64)
    D = np.eye(4)
    D[:3, :3] = R
    D[:3, 3] = -R @ p
    return D


@pytest.mark.parametrize("fx_sign", [1.0, -1.0])
@pytest.mark.parametrize("normal", [1.0, -1.0])
@pytest.mark.parametrize("level", [0, 1])
def test_pixels_beside_the_object_near_the_world_origin(fx_sign, normal, level):
    """Beside an object its model map holds (0, 0, 0) with an invalid normal,
    whose bilinear interpolation may round to a valid one: a live point within
    10 cm of the world origin then has a row.  Segments there are evaluated for
    either sign of the focal length (x runs from right to left for fx < 0)."""
    W, H = 161, 119
    s = make_scene("multi", W, H, n_frames=2, seed=13, bg_size=128, obj_size=64, n_objects=1)
    s.statics = []
    s.k = s.k * np.array([fx_sign, 1, 1, 1], np.float32)
    _, _, lab = s.render(1)
    # a column away from the object
    px = W - 30 if np.nonzero(lab == 1)[1].mean() < W / 2 else 30
    ctx = _second_frame(s, _far_wall_to_origin(s, px, normal), robust="huber", use_rgb=False,
                        gn_iterations=(0,) * level + (2,))
    for i in range(2):
        _compare(ctx, i, level, counts=i == 0)
    ctx.close()
