"""Device arithmetic that stands in for costlier formulas gives their bits.

* exp_nearest and div_e2 (mf_exp.cuh): the double exponential rounded to float,
  for every float at most 0.
* robust (mf_robust.cuh): the double weights and losses of the four robust
  kernels rounded to float, for every float.
* inverse_warp and inverse (mf_warp.cuh, mf_common.cuh): Gaussian elimination
  with plain divisions, for poses, ill-scaled and pivoting matrices, singular
  ones and ones that are not finite.
* solve6_eigen_warp: the host's truncated solve, where rotation angles are so
  small that the square roots are left out."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from mid_fusion_b200 import build
from mid_fusion_b200.capi import Context

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("device") / "identities.so"
    subprocess.run([os.environ.get("NVCC", "nvcc"), *build.NVCC_FLAGS, "-I",
                    os.path.join(build.HERE, "csrc"), "-I", os.path.join(build.ROOT, "include"),
                    os.path.join(HERE, "device_identities.cu"), "-o", str(so)], check=True)
    return C.CDLL(str(so))


def _run(fn, *args):
    bad, first = np.zeros(2, np.uint64), np.zeros(2, np.float32)
    rc = fn(*args, bad.ctypes.data_as(C.c_void_p), first.ctypes.data_as(C.c_void_p))
    assert rc == 0, rc
    return bad.tolist(), first.tolist()


def test_exponential_of_every_float(lib):
    assert _run(lib.check_exp) == ([0, 0], [0.0, 0.0])


@pytest.mark.parametrize("kind", [0, 1, 2, 3])
def test_robust_weight_and_loss_of_every_float(lib, kind):
    assert _run(lib.check_robust, kind) == ([0, 0], [0.0, 0.0])


def _matrices():
    rng = np.random.default_rng(5)
    f = np.float32
    out = []
    n = 20000
    # rotations and translations of every size
    q = rng.normal(size=(n, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    P = np.zeros((n, 4, 4))
    P[:, 0] = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                        rng.normal(size=n) * 10.0 ** rng.uniform(-6, 6, n)], 1)
    P[:, 1] = np.stack([2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                        rng.normal(size=n)], 1)
    P[:, 2] = np.stack([2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y),
                        rng.normal(size=n)], 1)
    P[:, 3, 3] = 1
    out.append(P)
    # signed permutations: exact zeros and pivots in every order
    S = np.zeros((n, 4, 4))
    for i in range(n):
        S[i, np.arange(3), rng.permutation(3)] = rng.choice([-1.0, 1.0, 0.5], 3)
    S[:, :3, 3] = rng.integers(-2, 3, (n, 3))
    S[:, 3, 3] = 1
    out.append(S)
    # affine matrices of any scale, rows scaled apart, some entries zero
    A = rng.normal(size=(n, 4, 4)) * 2.0 ** rng.uniform(-70, 70, (n, 1, 1))
    A *= 2.0 ** rng.uniform(-20, 20, (n, 4, 1))
    A[rng.random((n, 4, 4)) < 0.2] = 0
    A[:, 3] = (0, 0, 0, 1)
    out.append(A)
    # small whole numbers: ties between pivots, singular ones among them
    Z = rng.integers(-2, 3, (n, 4, 4)).astype(float)
    Z[::2, 3] = (0, 0, 0, 1)
    out.append(Z)
    # general last rows, negative zeros there, infinities and NaN
    G = P.copy()
    G[:, 3] = rng.normal(size=(n, 4))
    G[::3, 3] = (-0.0, 0.0, 0.0, 1.0)
    G[1::3, 3] = (0, 0, 0, 2.0)
    out.append(G)
    N = P.copy()
    i = rng.integers(0, 3, n), rng.integers(0, 4, n)
    N[np.arange(n), i[0], i[1]] = rng.choice([np.inf, -np.inf, np.nan, 1e38, 1e-44], n)
    out.append(N)
    with np.errstate(over="ignore"):
        return np.ascontiguousarray(np.concatenate(out).astype(f).reshape(-1, 16))


def test_inverse_of_any_matrix(lib):
    A = _matrices()
    bad, first = _run(lib.check_inverse, A.ctypes.data_as(C.c_void_p), len(A))
    assert bad == [0, 0], (bad, [A[int(i)] for i in first])


def test_truncated_solve_of_nearly_diagonal_systems():
    """Off-diagonal terms from 1 down to the smallest doubles: rotation angles
    below 2^-28 (the square roots are exact there) and quotients whose square
    overflows.  The steps are small: their pose update has no sine or cosine
    (which round differently on the host), and on the identity it shows every
    bit of the solution."""
    build.build()
    rng = np.random.default_rng(9)
    n = 400
    state, sums = np.zeros((n, 36)), np.zeros((n, 32))
    state[:, 0:16] = state[:, 16:32] = np.eye(4).reshape(16)
    state[:, 32] = np.inf
    state[:, 33] = np.arange(n) % 2
    sums[:, 0] = 1.0
    sums[:, 28] = 1000
    for m in range(n):
        A = np.diag(10.0 ** rng.uniform(-3, 3, 6))
        dead = rng.integers(0, 6, rng.integers(1, 3))
        A[dead, dead] = rng.choice([0.0, 1e-30, 1e-12])   # dropped by the truncation
        lo = rng.choice([-308.0, -160.0, -20.0, -9.0])
        for i in range(6):
            for j in range(i):
                v = rng.normal() * 10.0 ** rng.uniform(lo, -6) * (rng.random() < 0.6)
                A[i, j] = A[j, i] = v
        sums[m, 7:28] = [A[i, j] for i in range(6) for j in range(i, 6)]
        sums[m, 1:7] = rng.normal(size=6) * 1e-10
    ctx = Context(64, 48, robust="huber")
    dev, host = ctx.debug_gn_step(state, sums)
    ctx.close()
    for m in range(n):
        assert np.array_equal(dev[m], host[m], equal_nan=True), m
    assert np.count_nonzero(host[:, 34]) > 0.9 * n   # the truncated solve
