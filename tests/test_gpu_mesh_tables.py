"""mf_mesh with triangulation tables of a caller's own, against the oracle's
marching cubes with the same table, bit for bit (NaN included).

mf_mesh_set_triangle_table checks the layout and the edge numbers; which edges
a row lists is the caller's affair.  An edge whose corners are on the same side
of the surface has its vertex outside the edge, possibly outside the volume, or
no finite one where the corners' values are equal."""
import ctypes as C

import numpy as np
import pytest

import _oracle as O
from mid_fusion_b200 import build
from mid_fusion_b200.capi import Context
from mid_fusion_b200.scene import generalize_masks, make_scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def _table(rows):
    t = np.full((256, 16), -1, np.int32)
    for r, edges in enumerate(rows):
        t[r, :len(edges)] = edges
    return t


def _tables():
    rng = np.random.default_rng(3)
    # any edges in any row, row 0 (also the row of cells without valid
    # corners) and row 255 among them
    yield "random", _table([rng.integers(0, 12, 3 * rng.integers(0, 6)) for _ in range(256)])
    # one triangle per row, of edges that the row does cross wherever it can
    corner = [(0, 1), (1, 2), (2, 3), (0, 3), (4, 5), (5, 6), (6, 7), (4, 7), (0, 4), (1, 5),
              (2, 6), (3, 7)]
    crossed = [[e for e, (a, b) in enumerate(corner) if (r >> a & 1) != (r >> b & 1)][:3]
               for r in range(256)]
    yield "crossed", _table(crossed)
    # the same with one uncrossed edge in every row that has one
    for r in range(256):
        other = [e for e in range(12) if e not in crossed[r] and
                 (r >> corner[e][0] & 1) == (r >> corner[e][1] & 1)]
        if crossed[r] and other:
            crossed[r][r % 3] = other[r % len(other)]
    yield "one uncrossed", _table(crossed)
    yield "empty", _table([[]] * 256)


def test_callers_tables_match_oracle():
    s = make_scene("room", 160, 120, n_frames=5, seed=4, bg_size=128)
    inst = s.instances[0]
    ctx = Context(160, 120, k=s.k, pool_blocks=1 << 13)
    ctx.add_instance(inst.size, inst.dim, np.eye(4), inst.label)
    orc = O.oracle()
    vol = orc.volume(inst.size, inst.dim)
    for f in range(5):
        d, rgb, lab = s.render(f)
        m = generalize_masks(lab, [inst.label])
        T = s.cam_poses[f].astype(np.float32)
        ctx.set_camera_pose(T)
        ctx.upload(d, rgb, m)
        ctx.integrate([0])
        vol.integrate(d, rgb.astype(np.float32) / np.float32(255), m[0], T, np.eye(4), s.k, 0.1)
    lib = orc.lib
    lib.or_mesh_set_table.argtypes = [C.c_void_p]
    try:
        for name, t in _tables():
            ctx.set_triangle_table(t)
            lib.or_mesh_set_table(t.ctypes.data_as(C.c_void_p))
            for fb in (False, True):
                got, want = ctx.mesh(0, float_bounds=fb), O.mesh(orc, vol, float_bounds=fb)
                assert len(got) == len(want), (name, fb, len(got), len(want))
                assert np.array_equal(got, want, equal_nan=True), (name, fb)
            assert name == "empty" or len(want) > 1000, name
    finally:
        lib.or_mesh_set_table(None)
    assert ctx.status() == 0
    ctx.close()
