"""The Gauss-Newton launches' waits for their own CTAs, on the GPU.

Both launches are cooperative (all CTAs resident) and wait between iterations.
A wait that gives up sets a status flag and leaves the problem's pose as it was;
the calls that would hand out that pose say so.  Two contexts that track at the
same time do not disturb each other."""
import threading

import numpy as np
import pytest

from mid_fusion_b200 import build
from mid_fusion_b200.capi import Context, MfError
from mid_fusion_b200.scene import make_scene

pytestmark = pytest.mark.gpu

GN_TIMEOUT = 32


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def _context(s, **kw):
    ctx = Context(s.width, s.height, k=s.k, pool_blocks=1 << 16, robust="huber", **kw)
    for inst, T in zip(s.instances, s.volume_poses(0)):
        ctx.add_instance(inst.size, inst.dim, T, inst.label)
    ctx.set_camera_pose(s.cam_poses[0])
    return ctx


def _frame(ctx, frame):
    from mid_fusion_b200 import capi
    d, rgb, lab = frame
    ctx._check(ctx.lib.mf_process_frame(
        ctx.h, capi._ptr(np.ascontiguousarray(d), np.float32),
        capi._ptr(np.ascontiguousarray(rgb), np.uint8),
        capi._ptr(np.ascontiguousarray(lab.astype(np.uint16)), np.uint16)))


def _poses(ctx, n):
    return np.array([ctx.camera_pose()] + [ctx.instance_pose(i) for i in range(n)])


def _gave_up(call, *args):
    with pytest.raises(MfError, match="MF_E_TIMEOUT"):
        call(*args)


@pytest.mark.parametrize("batched", [True, False])
def test_a_wait_that_gives_up_is_reported(batched, tmp_path):
    """With no poll allowed, every CTA that is not the last to arrive gives up
    at once (the coarsest level has rows for 5 of the camera's 25 CTAs)."""
    s = make_scene("multi", 160, 120, n_frames=4, seed=11, n_objects=2, bg_size=128, obj_size=64)
    frames = [s.render(f) for f in range(4)]
    n = len(s.instances)
    ctx = _context(s, batched=batched)
    for f in frames[:2]:
        _frame(ctx, f)
    good = _poses(ctx, n)
    assert ctx.status() & GN_TIMEOUT == 0
    ctx.debug_gn_wait(0)
    if batched:
        _frame(ctx, frames[2])   # queued work: the error shows where it is waited for
    else:
        _gave_up(_frame, ctx, frames[2])
    for call in (ctx.camera_pose, ctx.synchronize, lambda: ctx.instance_pose(1),
                 lambda: ctx.track_info(0), lambda: ctx.save_poses(str(tmp_path / "p"), 0)):
        _gave_up(call)
    assert not list(tmp_path.iterdir())
    assert ctx.status() & GN_TIMEOUT
    assert ctx.status() == 0
    # the camera's pose is the one before the frame
    assert np.array_equal(ctx.camera_pose(), good[0])
    # a motion frame decides on poses: it stops before it integrates
    _gave_up(ctx.process_frame_motion, *frames[3])
    assert ctx.status() & GN_TIMEOUT
    # the context goes on
    ctx.debug_gn_wait(1 << 21)
    ctx.set_camera_pose(good[0])
    _frame(ctx, frames[2])
    assert np.all(np.isfinite(_poses(ctx, n)))
    assert not np.array_equal(ctx.camera_pose(), good[0])
    assert ctx.status() & GN_TIMEOUT == 0
    ctx.close()


@pytest.mark.parametrize("a,b", [
    (("multi", 640, 480, 3), ("multi", 640, 480, 3)),
    (("uneven", 640, 480, 12), ("multi", 160, 120, 0)),
    (("multi", 1280, 720, 6), ("multi", 320, 240, 2)),
])
def test_two_contexts_at_once(a, b):
    """Both contexts' frames queued by two threads at the same time: the poses
    of each are those of the context alone, bit for bit."""
    runs = []
    for preset, W, H, objects in (a, b):
        s = make_scene(preset, W, H, n_frames=4, seed=23, n_objects=objects)
        frames = [s.render(f) for f in range(4)]
        # more frames for the smaller one: its launches meet all of the other's
        order = [0, 1, 2, 3, 2, 1] * (2 if W * H > 200000 else 12)
        runs.append((s, [frames[i] for i in order]))

    def run(s, frames, out, start=None):
        ctx = _context(s)
        for f in frames[:2]:
            _frame(ctx, f)   # both reference parities captured
        ctx.synchronize()
        if start:
            start.wait()
        for f in frames[2:]:
            _frame(ctx, f)
        out.append((_poses(ctx, len(s.instances)), ctx.status()))
        ctx.close()

    alone, both = [[], []], [[], []]
    for r, out in zip(runs, alone):
        run(*r, out)
    barrier = threading.Barrier(2, timeout=60)
    threads = [threading.Thread(target=run, args=(*r, out, barrier))
               for r, out in zip(runs, both)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for x, y in zip(alone, both):
        assert len(y) == 1
        assert y[0][1] & (GN_TIMEOUT | 1) == 0   # nor was the pool full
        assert x[0][1] == y[0][1]
        assert np.array_equal(x[0][0], y[0][0], equal_nan=True)
