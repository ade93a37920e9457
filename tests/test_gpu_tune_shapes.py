"""What the numbers of the launch shapes stand for in a context."""
import numpy as np
import pytest

from mid_fusion_b200 import build, capi
from mid_fusion_b200.capi import Context
from mid_fusion_b200.scene import make_scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def _frames(ctx, s, first, n):
    for f in range(first, first + n):
        d, rgb, lab = s.render(f)
        ctx._check(ctx.lib.mf_process_frame(
            ctx.h, capi._ptr(np.ascontiguousarray(d), np.float32),
            capi._ptr(np.ascontiguousarray(rgb), np.uint8),
            capi._ptr(np.ascontiguousarray(lab.astype(np.uint16)), np.uint16)))
    ctx.synchronize()


def _context(s, **kw):
    ctx = Context(s.width, s.height, k=s.k, pool_blocks=1 << 15, robust="huber", **kw)
    for inst, T in zip(s.instances, s.volume_poses(0)):
        ctx.add_instance(inst.size, inst.dim, T, inst.label)
    ctx.set_camera_pose(s.cam_poses[0])
    return ctx


def test_setting_the_shape_in_use_changes_nothing():
    """mf_tune_set(stage, mf_tune_get(stage)), as a program that saves and
    restores the choice does, leaves an untuned context's overlapped frames
    with the launches that they had."""
    s = make_scene("multi", 160, 120, n_frames=7, seed=11, n_objects=2, bg_size=128, obj_size=64)
    ctx = _context(s)
    _frames(ctx, s, 0, 3)   # both reference parities captured
    before = ctx.frame_stats()["graph_kernels"]
    for stage in (capi.TUNE_RAYCAST, capi.TUNE_INTEGRATE):
        assert ctx.tune_get(stage) == 0
        ctx.tune_set(stage, ctx.tune_get(stage))
    _frames(ctx, s, 3, 2)
    assert ctx.frame_stats()["graph_kernels"] == before > 0
    # so does any other number: overlapped frames march per instance
    for v in range(capi.tune_candidates(capi.TUNE_RAYCAST)):
        ctx.tune_set(capi.TUNE_RAYCAST, v)
        _frames(ctx, s, 5, 2)
        assert ctx.frame_stats()["graph_kernels"] == before, v
    ctx.close()


def test_the_tuner_times_whole_raycasts():
    """Whether frames overlap or not, the tuner's time of a raycast shape is
    that of the whole raycast, as mf_raycast, motion frames, costs and frames
    in order run it.  (Without the background's marches a phased shape takes
    less than half.)"""
    s = make_scene("multi", 640, 480, n_frames=3, seed=11, n_objects=2, bg_size=512,
                   obj_size=128)
    ctx = _context(s)
    _frames(ctx, s, 0, 3)
    us = {}
    for overlap in (-1, 0):
        ctx.set_overlap(overlap)
        us[overlap] = np.array(ctx.autotune(reps=10)["raycast"]["us"])
    phased = [v for v in range(len(us[0]))
              if "phased" in capi.tune_describe(capi.TUNE_RAYCAST, v)]
    # the same launches: run to run a few percent apart
    assert np.all(us[-1][phased] > 0.75 * us[0][phased]), us
    ctx.close()
