"""mf_set_gn_persistent selects nothing any more, so it costs nothing either."""
import ctypes as C
import time

import numpy as np
import pytest

from mid_fusion_b200 import build
from mid_fusion_b200.capi import Context
from mid_fusion_b200.scene import make_scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def test_the_call_keeps_the_captured_frames():
    """A frame after the call replays the captured graph: queueing it takes the
    host the time of a launch, not that of a capture (some 30 kernels recorded
    and instantiated again, many times as long)."""
    import torch
    s = make_scene("multi", 160, 120, n_frames=2, seed=11, n_objects=2, bg_size=128, obj_size=64)
    ctx = Context(160, 120, k=s.k, pool_blocks=1 << 14, robust="huber")
    for inst, T in zip(s.instances, s.volume_poses(0)):
        ctx.add_instance(inst.size, inst.dim, T, inst.label)
    ctx.set_camera_pose(s.cam_poses[0])
    inputs = []
    for f in range(2):
        d, rgb, lab = s.render(f)
        inputs.append([torch.from_numpy(np.ascontiguousarray(a)).cuda()
                       for a in (d, rgb, lab.astype(np.int16))])
    torch.cuda.synchronize()

    def queue(f):
        t = time.perf_counter()
        rc = ctx.lib.mf_process_frame_device(ctx.h, *(C.c_void_p(a.data_ptr())
                                                      for a in inputs[f & 1]))
        t = time.perf_counter() - t
        assert rc == 0
        ctx.synchronize()
        return t

    for f in range(4):
        queue(f)
    kept, called = [], []
    for f in range(20):
        kept.append(queue(f))
    for f in range(20):
        ctx.set_gn_persistent(f & 1)
        called.append(queue(f))
    assert min(called) < 3 * min(kept), (min(called), min(kept))
    ctx.close()
