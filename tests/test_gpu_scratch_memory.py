"""Device memory that calls keep beyond their return."""
import numpy as np
import pytest

from mid_fusion_b200 import build
from mid_fusion_b200.capi import Context
from mid_fusion_b200.scene import generalize_masks, make_scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _pair(W, H):
    """A context with a reference frame and a preprocessed live one, and the
    live pose."""
    s = make_scene("multi", W, H, n_frames=2, seed=3, bg_size=128, n_objects=0)
    ctx = Context(W, H, k=s.k, pool_blocks=1 << 13, max_instances=1, robust="huber")
    ctx.add_instance(128, 5.12, np.eye(4, dtype=np.float32), 0)
    ctx.set_camera_pose(s.cam_poses[0])
    for f in range(2):
        d, rgb, lab = s.render(f)
        ctx.upload(d, rgb, generalize_masks(lab, [0]))
        ctx.preprocess()
        if f == 0:
            ctx.integrate([0])
            ctx.set_ref_from_current()
    return ctx, s.cam_poses[1]


def test_cost_without_a_gradient_keeps_no_gradient_scratch():
    """The raycast's winner planes (17 B per pixel) serve the TSDF gradient:
    they are allocated by the first call that asks for one."""
    import torch
    W, H = 1280, 720
    small, T = _pair(160, 120)
    grad = torch.zeros(small.pool_tsdf()[1], dtype=torch.float32, device="cuda")
    small.camera_cost(T, grad.data_ptr())   # the driver's own memory for these kernels' stacks
    small.close()
    ctx, T = _pair(W, H)
    a = ctx.camera_cost(T)
    before = _free()
    b = ctx.camera_cost(T, grad.data_ptr())
    taken = before - _free()
    assert taken >= 17 * W * H
    c = ctx.camera_cost(T, grad.data_ptr())
    assert before - _free() == taken   # the first one only
    assert a[0] == b[0] == c[0] and a[2] == b[2] > 0
    assert float(grad.abs().max()) > 0
    ctx.close()


def test_a_large_mesh_is_given_back():
    """Up to 64 MiB of triangles on their way to host memory stay with the
    context for the next call; more is freed before the call returns."""
    s = make_scene("multi", 640, 480, n_frames=1, seed=4, n_objects=0, noise=False)
    ctx = Context(640, 480, k=s.k, mu=0.02, pool_blocks=1 << 17, max_instances=1)
    ctx.add_instance(2048, 5.12, np.eye(4, dtype=np.float32), 0)
    d, rgb, lab = s.render(0)
    ctx.set_camera_pose(s.cam_poses[0])
    ctx.upload(d, rgb, generalize_masks(lab, [0]))
    for _ in range(5):
        ctx.integrate([0])
    before = _free()
    tri = ctx.mesh(0, float_bounds=True)
    kept = before - _free()
    assert tri.nbytes > 72 << 20, tri.nbytes
    # next to the triangles the call keeps its block list and offsets: 16 B per
    # block of the pool (and what the driver rounds up to)
    assert kept <= 8 << 20, kept
    assert np.array_equal(tri, ctx.mesh(0, float_bounds=True))
    ctx.close()
