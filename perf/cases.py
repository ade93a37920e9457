"""The work that programs built on this library have it do, as measurable cases.

Every case is one of the kinds below, run through the public entry points
(mid_fusion_b200.capi, mid_fusion_b200.autograd and, where a device destination
is wanted, the C ABI of include/midfusion_b200.h itself):

  frame      the whole per-frame pipeline of a live RGB-D stream: poses, map
             and model maps updated, the poses read back and the model's
             normals rendered for display.  feed "host": mf_process_frame from
             host buffers; "staged": uploads overlapped (mf_frame_stage);
             "device": frames that are on the GPU already.
  motion     the pipeline with motion segmentation (mf_process_frame_motion)
  localise   camera tracking against a fixed map, stage by stage: pyramid,
             Gauss-Newton, row codes, raycast at the tracked pose
  map        mapping with known poses: allocation and integration alone
  render     the shaded view of the map from a free view point
  adjoint    the camera cost and its gradients (twist and TSDF) for an optimiser
  mesh       marching cubes over the background, for export
  interp     field queries at a few thousand points, the smallest calls

The sequences are seeded synthetic scenes (mid_fusion_b200.scene: room, static
furniture, moving boxes, spheres and cylinders), rendered on the GPU here.  A
state walks its frames back and forth; after each walk its poses are put back
to the known ones, as a relocaliser would, so that passes stay alike.
"""
import ctypes
import math

import numpy as np
import torch

from mid_fusion_b200 import capi, scene

FRAMES = 6           # rendered frames of a sequence; walked back and forth
VIEW_BLOCKS = 20480  # blocks that the map and adjoint kinds return, more than their scenes hold
MESH_CAP = 1 << 19   # triangles that the mesh kind's buffer holds
ORDER = list(range(FRAMES)) + list(range(FRAMES - 2, 0, -1))


def listed():
    vga = dict(w=640, h=480, bg=512)
    return [
        # a robot's map queries: a few thousand points of a small volume
        dict(name="interp_4k", kind="interp", n=4096, size=64),
        # the smallest frames: a room on an embedded-sized stream, one octree
        dict(name="frame_room_160", kind="frame", feed="host", w=160, h=120, bg=128, objects=0,
             uneven=False, robust="huber", tuned=False),
        # the single-octree room at 320x240, 256^3
        dict(name="frame_room_320", kind="frame", feed="host", w=320, h=240, bg=256, objects=0,
             uneven=False, robust="cauchy", tuned=False),
        # the headline stream: VGA, 512^3 background and three 256^3 objects
        dict(name="frame_multi_640", kind="frame", feed="device", objects=3, uneven=False,
             robust="huber", tuned=True, **vga),
        # a cluttered table: twelve objects of uneven size, uploads overlapped
        dict(name="frame_uneven_640", kind="frame", feed="staged", objects=12, uneven=True,
             robust="huber", tuned=True, **vga),
        # the largest: 720p, six objects, the reference's default robust kernel
        dict(name="frame_multi_1280", kind="frame", feed="device", w=1280, h=720, bg=512,
             objects=6, uneven=False, robust="cauchy", tuned=False),
        # VGA with motion segmentation, host-driven
        dict(name="motion_640", kind="motion", objects=3, uneven=False, robust="cauchy",
             tuned=False, **vga),
        # tracking against a fixed map on a ragged frame size
        dict(name="localise_637", kind="localise", w=637, h=479, bg=512, objects=0,
             uneven=False, robust="tukey", tuned=False),
        # mapping with external poses
        dict(name="map_640", kind="map", objects=3, uneven=False, robust="huber", tuned=False,
             **vga),
        # a viewer
        dict(name="render_640", kind="render", objects=3, uneven=False, robust="huber",
             tuned=False, **vga),
        # an optimiser over poses and map
        dict(name="adjoint_640", kind="adjoint", objects=3, uneven=False, robust="huber",
             tuned=False, **vga),
        # export of the finished map
        dict(name="mesh_512", kind="mesh", objects=0, uneven=False, robust="huber", tuned=False,
             **vga),
    ]


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["motion", "localise", "localise", "map", "map", "render",
                                       "adjoint", "mesh", "interp"])
    if kind == "interp":
        return dict(kind=kind, n=int(math.exp(rng.uniform(math.log(16), math.log(65536)))),
                    size=rng.choice([32, 64, 128]))
    w = int(math.exp(rng.uniform(math.log(160), math.log(1280))))
    h = int(w * rng.uniform(0.55, 0.76))
    h = min(h, 1280 * 720 // w)
    c = dict(kind=kind, w=w, h=h, bg=rng.choice([128, 256, 512, 512]),
             objects=rng.choice([0, 1, 2, 3, 4]), uneven=False,
             robust=rng.choice(["none", "huber", "tukey", "cauchy"]), tuned=rng.random() < 0.4)
    if kind == "frame":
        c["feed"] = rng.choice(["host", "staged", "device"])
        if rng.random() < 0.3 and w >= 320 and w * h <= 640 * 480:
            c.update(objects=rng.randint(4, 12), uneven=True)
    if kind == "motion":
        c["objects"] = max(1, c["objects"])
    if kind == "localise":
        c["objects"] = 0
    return c


# ---------------------------------------------------------------- scenes
def _scene(case, seed):
    return scene.make_scene("uneven" if case["uneven"] else "multi", case["w"], case["h"],
                            n_frames=FRAMES, seed=int(seed) % (1 << 30),
                            n_objects=case["objects"], bg_size=case["bg"], noise=False,
                            sway=48.0 if case["uneven"] else 0.0)


def _noise(lat, p):
    """scene.ValueNoise on the GPU: two octaves of seeded value noise."""
    n, out = lat.shape[1], 0
    for octave, amp in ((1.0, 0.65), (2.0, 0.35)):
        q = p * (6.0 * octave)
        i0 = torch.floor(q).long()
        f = q - i0
        f = f * f * (3 - 2 * f)
        acc = 0
        for c in range(8):
            d = (c & 1, (c >> 1) & 1, c >> 2)
            i = [(i0[:, k] + d[k]) % n for k in range(3)]
            wgt = 1
            for k in range(3):
                wgt = wgt * (f[:, k] if d[k] else 1 - f[:, k])
            acc = acc + wgt[:, None] * lat[:, i[0], i[1], i[2]].t()
        out = out + amp * acc
    return out


def _hit(sh, o, d):
    """Ray parameter and normal of a primitive in its own frame (scene._intersect_local)."""
    inf = torch.full_like(d[:, 0], math.inf)
    if sh.kind == "box":
        hs = torch.tensor([0.5 * v for v in sh.size], dtype=d.dtype, device=d.device)
        inv = 1.0 / d
        a, b = (-hs - o) * inv, (hs - o) * inv
        lo, hi = torch.minimum(a, b), torch.maximum(a, b)
        tn, ax = lo.max(1)
        ok = (tn <= hi.min(1).values) & (tn > 1e-6)
        nrm = torch.zeros_like(d)
        nrm.scatter_(1, ax[:, None], -torch.sign(d.gather(1, ax[:, None])))
        return torch.where(ok, tn, inf), nrm
    if sh.kind == "sphere":
        r, a, b = sh.size[0], (d * d).sum(1), (o * d).sum(1)
        disc = b * b - a * ((o * o).sum(1) - r * r)
        t = (-b - torch.sqrt(disc.clamp(min=0))) / a
        t = torch.where((disc >= 0) & (t > 1e-6), t, inf)
        return t, (o + torch.where(t < math.inf, t, 0)[:, None] * d) / r
    r, hh = sh.size[0], 0.5 * sh.size[1]
    a = (d[:, 0] ** 2 + d[:, 2] ** 2).clamp(min=1e-12)
    b = o[:, 0] * d[:, 0] + o[:, 2] * d[:, 2]
    disc = b * b - a * (o[:, 0] ** 2 + o[:, 2] ** 2 - r * r)
    t = (-b - torch.sqrt(disc.clamp(min=0))) / a
    ok = (disc >= 0) & (t > 1e-6) & ((o[:, 1] + t * d[:, 1]).abs() <= hh)
    t = torch.where(ok, t, inf)
    p = o + torch.where(ok, t, 0)[:, None] * d
    nrm = torch.stack([p[:, 0], torch.zeros_like(t), p[:, 2]], 1) / r
    for cap in (-hh, hh):
        tc = (cap - o[:, 1]) / d[:, 1]
        q = o + tc[:, None] * d
        ok = (tc > 1e-6) & (q[:, 0] ** 2 + q[:, 2] ** 2 <= r * r) & (tc < t)
        t = torch.where(ok, tc, t)
        cn = torch.tensor([0.0, math.copysign(1.0, cap), 0.0], dtype=d.dtype, device=d.device)
        nrm = torch.where(ok[:, None], cn, nrm)
    return t, nrm


def _render(s, f, lat, gen):
    """Frame f of a scene on the GPU: depth f32 (noisy, 1 % dropouts), rgb u8, labels i16."""
    W, H, dev = s.width, s.height, "cuda"
    t64 = lambda v: torch.as_tensor(np.asarray(v, np.float64), device=dev)  # noqa: E731
    fx, fy, cx, cy = (float(v) for v in s.k)
    T = t64(s.cam_poses[f])
    ys, xs = torch.meshgrid(torch.arange(H, dtype=torch.float64, device=dev),
                            torch.arange(W, dtype=torch.float64, device=dev), indexing="ij")
    dc = torch.stack([(xs - cx) / fx, (ys - cy) / fy, torch.ones_like(xs)], -1).reshape(-1, 3)
    dw = dc @ T[:3, :3].t()
    o = T[:3, 3].expand_as(dw)
    tt = (torch.where(dw > 0, t64(s.room_hi), t64(s.room_lo)) - o) / dw
    tt = torch.where(torch.isfinite(tt) & (tt > 0), tt, math.inf)
    best, ax = tt.min(1)
    nrm = torch.zeros_like(dw)
    nrm.scatter_(1, ax[:, None], -torch.sign(dw.gather(1, ax[:, None])))
    label = torch.zeros(len(best), dtype=torch.int16, device=dev)
    tint = t64([0.8, 0.78, 0.72]).expand_as(dw).clone()
    for sh in list(s.statics) + list(s.movers):
        P = t64(sh.pose_at(f))
        t, nl = _hit(sh, (o - P[:3, 3]) @ P[:3, :3], dw @ P[:3, :3])
        near = t < best
        best = torch.where(near, t, best)
        nrm = torch.where(near[:, None], nl @ P[:3, :3].t(), nrm)
        label = torch.where(near, torch.tensor(sh.label, dtype=torch.int16, device=dev), label)
        tint = torch.where(near[:, None], t64(sh.tint), tint)
    p = o + best[:, None] * dw
    light = t64([0.3, -0.8, -0.5]) / math.sqrt(0.98)
    shade = 0.55 + 0.45 * (nrm @ light).abs()
    rgb = (_noise(lat, p) * tint * shade[:, None] * 1.15).clamp(0, 1)
    rgb = (rgb * 255 + 0.5).to(torch.uint8).reshape(H, W, 3).contiguous()
    sigma = 0.0012 + 0.0019 * (best - 0.4) ** 2
    depth = best + torch.randn(best.shape, generator=gen, device=dev, dtype=torch.float64) * sigma
    depth[torch.rand(best.shape, generator=gen, device=dev) < 0.01] = 0.0
    depth = depth.clamp(min=0).float().reshape(H, W).contiguous()
    return depth, rgb, label.reshape(H, W).contiguous()


def _masks(label, n):
    """Generalised masks (1 inside, 0 on the ring of a 5x5 elliptic dilation, -1 elsewhere)."""
    pool = torch.nn.functional.max_pool2d
    out = []
    for i in range(n):
        m = (label == i).float()[None]
        ring = torch.maximum(pool(m, (3, 5), 1, (1, 2)), pool(m, (5, 1), 1, (2, 0)))
        out.append(torch.where(m > 0, 1.0, torch.where(ring > 0, 0.0, -1.0))[0])
    return torch.stack(out).contiguous()


class _State:
    """A context, its sequence and where the walk over it stands."""

    def __init__(self, case, seed):
        self.case, self.at = case, 0
        s = self.scene = _scene(case, seed)
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        lat = torch.as_tensor(s.albedo.lat.astype(np.float64), device="cuda")
        self.frames = [_render(s, f, lat, gen) for f in range(FRAMES)]
        self.poses = [np.asarray(T, np.float32) for T in s.cam_poses]
        self.volumes = [[np.asarray(T, np.float32) for T in s.volume_poses(f)]
                        for f in range(FRAMES)]
        n = len(s.instances)
        self.ctx = capi.Context(s.width, s.height, k=s.k, pool_blocks=1 << 16,
                                max_instances=max(n, 1), robust=case["robust"])
        for inst, T in zip(s.instances, self.volumes[0]):
            self.ctx.add_instance(inst.size, inst.dim, T, inst.label)
        if case["tuned"]:  # the choice that the autotuner made once on this hardware
            self.ctx.tune_set(capi.TUNE_RAYCAST, 11)
            self.ctx.tune_set(capi.TUNE_INTEGRATE, 5)
        self.stream = torch.cuda.ExternalStream(self.ctx.stream())
        self.out_cam = np.zeros(16, np.float32)
        self.out_vol = np.zeros((n, 16), np.float32)
        self.image = torch.zeros((s.height, s.width, 3), dtype=torch.uint8, device="cuda")
        self.relocate(0)

    def relocate(self, f):
        self.ctx.set_camera_pose(self.poses[f])
        for i, T in enumerate(self.volumes[f]):
            self.ctx.set_instance_pose(i, T)

    def host_frames(self):
        def pin(t):
            return t.cpu().pin_memory().numpy()
        self.host = [(pin(d), pin(c), pin(lab).view(np.uint16)) for d, c, lab in self.frames]

    def next(self):
        f = ORDER[self.at]
        self.at = (self.at + 1) % len(ORDER)
        return f

    def check(self, rc):
        if rc != 0:
            raise RuntimeError(self.ctx.lib.mf_last_error(self.ctx.h).decode())

    def get_poses(self):
        self.check(self.ctx.lib.mf_get_poses(self.ctx.h, _np(self.out_cam), _np(self.out_vol)))
        return self.out_cam.reshape(4, 4).copy(), self.out_vol.reshape(-1, 4, 4).copy()

    def map_frame(self, f):
        """Allocation and integration of frame f at its known poses."""
        c = self.ctx
        d, rgb, _ = self.frames[f]
        m = self.masks[f]
        self.check(c.lib.mf_frame_set_device(c.h, _pt(d), _pt(rgb), _pt(m), len(m)))
        self.relocate(f)
        c.integrate(list(range(c.n_instances)))

    def known_map(self):
        """The map of the whole sequence at its known poses."""
        self.masks = [_masks(fr[2], self.ctx.n_instances) for fr in self.frames]
        torch.cuda.synchronize()
        for f in ORDER:
            self.map_frame(f)
        self.ctx.synchronize()
        slots = self.ctx.pool_slots()
        # the blocks in a fixed order (slots are handed out in any), then unused slots
        perm = np.lexsort((slots[:, 0], slots[:, 1], slots[:, 2], slots[:, 3]))
        perm = np.concatenate([perm, np.arange(len(perm), max(len(perm), VIEW_BLOCKS))])
        self.perm = torch.as_tensor(perm[:VIEW_BLOCKS], device="cuda")


def _pt(t):
    return ctypes.c_void_p(t.data_ptr())


def _np(a):
    return a.ctypes.data_as(ctypes.c_void_p)


# ---------------------------------------------------------------- cases
def prepare(case, seed):
    if case["kind"] == "interp":
        return _Interp(case, seed).open()
    s = _State(case, seed)
    kind = case["kind"]
    if kind in ("frame", "motion"):
        if case.get("feed") != "device":
            s.host_frames()
        torch.cuda.synchronize()
        s.staged = 0
        if case.get("feed") == "staged":
            s.ctx.frame_stage(0, *s.host[s.next()])
        for _ in ORDER:   # a stream that has been running for a while
            run(s)
    else:
        s.known_map()
        if kind == "localise":
            s.codes = torch.zeros((2, case["h"], case["w"]), dtype=torch.int8, device="cuda")
            s.errors = torch.zeros((2, case["h"], case["w"]), device="cuda")
            s.relocate(0)
            d, rgb, _ = s.frames[0]
            s.check(s.ctx.lib.mf_frame_set_device(s.ctx.h, _pt(d), _pt(rgb), None, 0))
            s.ctx.preprocess()
            s.ctx.raycast()
            s.ctx.set_ref_from_current()
            for _ in ORDER:
                run(s)
        elif kind == "render":
            s.view = torch.zeros((case["h"], case["w"], 4), dtype=torch.uint8, device="cuda")
            rng = np.random.default_rng(seed)
            s.views = []
            for f in range(FRAMES):
                T = s.poses[f].astype(np.float64) @ scene.se3_exp(
                    rng.uniform(-1, 1, 6) * [0.15, 0.1, 0.15, 0.08, 0.12, 0.05])
                s.views.append(np.ascontiguousarray(T.astype(np.float32)))
        elif kind == "adjoint":
            from mid_fusion_b200 import autograd
            s.cost = autograd.CameraCost
            c = s.ctx
            for f in (0, 1):
                d, rgb, _ = s.frames[f]
                s.check(c.lib.mf_frame_set_device(c.h, _pt(d), _pt(rgb), None, 0))
                c.preprocess()
                if f == 0:
                    c.set_ref_from_current()
            s.relocate(0)
            s.T0 = s.poses[1].astype(np.float64)
            rng = np.random.default_rng(seed)
            s.twists = [torch.tensor(rng.uniform(-1, 1, 6) * 0.002, dtype=torch.float64)
                        for _ in range(4)]
            s.tsdf = autograd.pool_tsdf_tensor(c)
        elif kind == "mesh":
            s.triangles = torch.zeros((MESH_CAP, 3, 3)).pin_memory().numpy()
            s.count = ctypes.c_longlong()
    s.ctx.synchronize()
    return s


class _Interp:
    """A small volume holding a known field, and the points to query."""

    def __init__(self, case, seed):
        n = self.n = case["size"]
        rng = np.random.default_rng(seed)
        self.field = rng.uniform(-1, 1, (n, n, n)).astype(np.float32)      # [z, y, x]
        self.dim = 0.01 * n
        # inside the last whole cell: every tap is a voxel of the volume
        self.points = rng.uniform(0, 0.01 * (n - 1.001), (case["n"], 3)).astype(np.float32)

    def open(self):
        n, c = self.n, capi.Context(64, 48, pool_blocks=max(64, (self.n // 8) ** 3),
                                    max_instances=1)
        c.add_instance(n, self.dim, np.eye(4, dtype=np.float32), 0)
        b = np.arange((n // 8) ** 3, dtype=np.uint64)
        c.alloc_update(0, (b << np.uint64(9)) | np.uint64(int(math.log2(n)) - 3))
        from mid_fusion_b200 import autograd
        x, y, z = (c.pool_slots()[:, k] // 8 for k in range(3))
        m = n // 8
        blocks = self.field.reshape(m, 8, m, 8, m, 8).transpose(0, 2, 4, 1, 3, 5)[z, y, x]
        pool = autograd.pool_tsdf_tensor(c).view(-1, 512)
        pool[:len(blocks)] = torch.as_tensor(blocks.reshape(-1, 512).copy(), device="cuda")
        torch.cuda.synchronize()
        self.ctx = c
        return self


def run(state):
    if isinstance(state, _Interp):
        return state.ctx.interp(0, state.points, 0)
    c, case = state.ctx, state.case
    kind = case["kind"]
    if kind == "frame":
        feed = case["feed"]
        if feed == "staged":
            slot, state.staged = state.staged, 1 - state.staged
            c.process_staged(slot)
            c.frame_stage(1 - slot, *state.host[state.next()])   # copies while this one runs
        else:
            f = state.next()
            if feed == "host":
                d, rgb, lab = state.host[f]
                rc = c.lib.mf_process_frame(c.h, _np(d), _np(rgb), _np(lab))
            else:
                d, rgb, lab = state.frames[f]
                rc = c.lib.mf_process_frame_device(c.h, _pt(d), _pt(rgb), _pt(lab))
            state.check(rc)
        state.check(c.lib.mf_render_normal(c.h, _pt(state.image)))
        cam, vols = state.get_poses()
        # the frame just processed, once its walk is over
        at = (state.at - (2 if feed == "staged" else 1)) % len(ORDER)
        if at == len(ORDER) - 1:
            state.relocate(ORDER[at])
            c.raycast()
        return cam, vols, state.image
    if kind == "motion":
        f = state.next()
        bits = c.process_frame_motion(*state.host[f])
        state.check(c.lib.mf_render_normal(c.h, _pt(state.image)))
        cam, vols = state.get_poses()
        if state.at == 0:
            state.relocate(f)
            c.raycast()
        return cam, vols, state.image, bits
    if kind == "localise":
        f = state.next()
        d, rgb, _ = state.frames[f]
        state.check(c.lib.mf_frame_set_device(c.h, _pt(d), _pt(rgb), None, 0))
        c.preprocess()
        c.track_camera()
        c.track_results(0, state.codes.data_ptr(), state.errors.data_ptr())
        c.raycast()
        c.set_ref_from_current()
        state.check(c.lib.mf_render_normal(c.h, _pt(state.image)))
        cam = c.camera_pose()
        if state.at == 0:
            c.set_camera_pose(state.poses[f])
            c.raycast()
        return cam, state.codes, state.errors, state.image
    if kind == "map":
        state.map_frame(state.next())
        tsdf = _tsdf(state)
        with torch.cuda.stream(state.stream):
            return tsdf.view(-1, 512).index_select(0, state.perm)
    if kind == "render":
        T = state.views[state.next()]
        state.check(c.lib.mf_render_volume(c.h, _np(T), 1, ctypes.c_float(0.075), None, None, 0,
                                           _pt(state.view)))
        return state.view
    if kind == "adjoint":
        twist = state.twists[state.next() % 4].clone().requires_grad_(True)
        tsdf = state.tsdf.detach().requires_grad_(True)
        e = state.cost.apply(twist, tsdf, c, state.T0)
        e.backward()
        g = tsdf.grad.view(-1, 512).index_select(0, state.perm)
        return e.detach(), twist.grad, g
    state.check(c.lib.mf_mesh(c.h, 0, 0, _np(state.triangles), ctypes.c_longlong(MESH_CAP),
                              ctypes.byref(state.count)))
    return state.triangles, state.count.value


def _tsdf(state):
    if not hasattr(state, "tsdf"):
        from mid_fusion_b200 import autograd
        state.tsdf = autograd.pool_tsdf_tensor(state.ctx)
    return state.tsdf


def _voxels(case):
    """Voxels in the truncation band (0.2 m) of the surfaces in view, roughly: 18 m^2 of room
    at the background's voxel size, and of each object what its volume holds of the band."""
    bg = min(case["bg"] ** 3, 18.0 * 0.2 * (case["bg"] / 5.12) ** 3)
    return bg + case["objects"] * (2e5 if case["uneven"] else 4e5)


def work(case):
    kind = case["kind"]
    if kind == "interp":
        return {"bytes": case["n"] * 16 + 4 * case["size"] ** 3, "flops": 30 * case["n"]}
    px, n = case["w"] * case["h"], 1 + case["objects"]
    iters = 10 + 5 / 4 + 4 / 16          # Gauss-Newton iterations in level-0 images
    fuse = 72 * _voxels(case)            # 36 B of voxel payload read and written
    maps = 28 * px                       # vertex, normal and label of the model
    gn = 500 * iters * px * 1.5          # the camera's rows, and the objects' in view
    cast = 400 * px * n
    if kind in ("frame", "motion"):
        return {"bytes": 9 * px + fuse + maps + 3 * px, "flops": gn + cast + 30 * _voxels(case)}
    if kind == "localise":
        return {"bytes": 7 * px + maps + 13 * px, "flops": gn + cast}
    if kind == "map":
        return {"bytes": px * (7 + 4 * n) + fuse, "flops": 30 * _voxels(case)}
    if kind == "render":
        return {"bytes": 4 * px + 4 * _voxels(case) / 4, "flops": cast}
    if kind == "adjoint":
        return {"bytes": 2 * maps + 4 * 512 * 65536, "flops": 6 * cast + 2000 * px}
    return {"bytes": 36.0 * _voxels(case), "flops": 40 * _voxels(case)}


def exact(case, seed):
    """Trilinear interpolation in 64 bits.  The other kinds are whole trackers and maps with
    data-dependent decisions (convergence tests, row validity, nearest hits): no value."""
    if case["kind"] != "interp":
        return None
    s = _Interp(case, seed)
    q = s.points.astype(np.float64) * (s.n / np.float64(np.float32(s.dim)))
    i = np.minimum(np.floor(q).astype(np.int64), s.n - 2)
    f, out = q - i, 0.0
    for c in range(8):
        d = np.array([c & 1, (c >> 1) & 1, c >> 2])
        j = i + d
        out = out + s.field[j[:, 2], j[:, 1], j[:, 0]] * np.prod(np.where(d, f, 1 - f), axis=1)
    return out
