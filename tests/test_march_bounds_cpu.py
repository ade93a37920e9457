"""Bounds that the allocation march rests on (alloc_mark_kernel,
mid_fusion_b200/csrc/mf_volume.cu), on the CPU in float32.

A ray's samples are `band / ceil(band / voxel)` apart: half a voxel to a voxel.
The march counts the samples of a run through one block in five bits, lists the
blocks that 24 samples leave in a list of 14, and leaves out the range test
where both ends of the ray are two voxels inside the volume."""
import numpy as np
import pytest

F = np.float32
MARK_STEPS, RUN_LIST, RUN_MAX = 24, 14, 31


def _rays(rng, size, dim, mu, n):
    """Surface points in and around the volume and directions through them:
    any, along an axis, along diagonals, and next to both; block corners too."""
    d = rng.normal(size=(n, 3))
    d[::5] = rng.choice([-1.0, 0.0, 1.0], (len(d[::5]), 3))
    d[1::5] = rng.choice([-1.0, 1.0], (len(d[1::5]), 3)) + rng.normal(size=(len(d[1::5]), 3)) * 1e-6
    d[2::5] = np.eye(3)[rng.integers(0, 3, len(d[2::5]))] + rng.normal(size=(len(d[2::5]), 3)) * 1e-6
    d[~d.any(axis=1)] = (0, 0, 1)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    p = rng.uniform(-0.1, 1.1, (n, 3)) * dim
    # a few ends just inside and outside the two-voxel margin, and on corners
    vox = dim / size
    p[3::7] = rng.integers(0, size // 8 + 1, (len(p[3::7]), 3)) * 8 * vox
    p[4::7] = rng.choice([2.0, 2.001, 1.999, size - 2.0, size - 2.001], (len(p[4::7]), 3)) * vox
    return p.astype(F), d.astype(F)


@pytest.mark.parametrize("size", [16, 64, 512, 4096])
@pytest.mark.parametrize("mu_voxels", [0.1, 0.5, 0.50001, 0.75, 1.0, 1.00001, 2.6, 10.0, 51.3])
def test_runs_lists_and_the_range_test(size, mu_voxels):
    rng = np.random.default_rng(size + int(1000 * mu_voxels))
    for dim in (0.512, 5.12, 37.7):
        dim = F(dim)
        vs = dim / F(size)
        inv_voxel = F(1) / vs
        mu = F(mu_voxels) * vs
        band = F(2) * mu
        steps = int(np.ceil(band * inv_voxel))
        p, d = _rays(rng, size, float(dim), float(mu), 3000)
        pos = p - (band * F(0.5)) * d
        step = (d * band) / F(steps)
        end = pos + F(steps) * step
        lo, hi = F(2), F(size) - F(2)

        def inside(q):
            f = q * inv_voxel
            return np.all((f > lo) & (f < hi), axis=1)
        all_in = inside(pos) & inside(end)
        n = len(p)
        key = np.full((n, 3), -1, np.int64)
        run = np.zeros(n, np.int64)
        listed = np.zeros(n, np.int64)
        for i in range(steps):
            if i % MARK_STEPS == 0:
                listed[:] = 0
            f = pos * inv_voxel
            ok = np.all((f < F(size)) & (f >= 0), axis=1)
            assert np.all(ok | ~all_in)
            k = np.where(ok[:, None], np.floor(np.where(ok[:, None], f, 0) / 8).astype(np.int64),
                         key)
            new = ok & np.any(k != key, axis=1)
            listed += new & (run > 0)
            run = np.where(new, 0, run) + ok
            key = k
            assert run.max() <= RUN_MAX
            assert listed.max() + (i == steps - 1) <= RUN_LIST
            pos = pos + step
