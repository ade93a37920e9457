"""Arithmetic identities the CUDA kernels rely on to match the reference,
checked on the CPU in float32.

Allocation marking (alloc_mark_kernel, mid_fusion_b200/csrc/mf_volume.cu):
the reference floors p = pos / voxel and tests 0 <= floor(p) < size before
converting to int (alloc_impl.hpp:121-191).  The kernel tests 0 <= p < size
and truncates.  For an integer size both tests accept the same p, NaN and
infinities included, and on the accepted p truncation equals the floor."""
import numpy as np
import pytest


def _reference(p, size):
    s = np.floor(p)
    ok = (s < np.float32(size)) & (s >= 0)
    return ok, np.where(ok, s, 0).astype(np.int64)


def _kernel(p, size):
    ok = (p < np.float32(size)) & (p >= 0)
    return ok, np.where(ok, np.trunc(np.where(ok, p, 0)), 0).astype(np.int64)


@pytest.mark.parametrize("size", [32, 64, 256, 512, 1024, 4096])
def test_floor_test_equals_range_test_and_truncation(size):
    f = np.float32
    ints = np.arange(-3, size + 4, dtype=np.float64)
    vals = [ints.astype(f)]
    # the float32 neighbours of every integer boundary
    for k in (1, 2, 3):
        up, dn = ints.astype(f), ints.astype(f)
        for _ in range(k):
            up = np.nextafter(up, f(np.inf))
            dn = np.nextafter(dn, f(-np.inf))
        vals += [up, dn]
    rng = np.random.default_rng(size)
    vals.append(rng.uniform(-2.0, size + 2.0, 200000).astype(f))
    vals.append(np.array([0.0, -0.0, np.nan, -np.nan, np.inf, -np.inf, 1e-45, -1e-45,
                          np.finfo(f).max, -np.finfo(f).max, 1e30, -1e30], f))
    p = np.concatenate(vals).astype(f)
    ok_r, v_r = _reference(p, size)
    ok_k, v_k = _kernel(p, size)
    assert np.array_equal(ok_r, ok_k)
    assert np.array_equal(v_r[ok_r], v_k[ok_k])
    assert np.all((v_k[ok_k] >= 0) & (v_k[ok_k] < size))



def test_block_index_is_the_morton_index():
    """spread3_10 / block_index (mf_common.cuh) against the bit-by-bit Morton
    code, every coordinate below 1024."""
    def spread(v):
        v = v.astype(np.uint32)
        v = (v | v << np.uint32(16)) & np.uint32(0x030000ff)
        v = (v | v << np.uint32(8)) & np.uint32(0x0300f00f)
        v = (v | v << np.uint32(4)) & np.uint32(0x030c30c3)
        return (v | v << np.uint32(2)) & np.uint32(0x09249249)
    v = np.arange(1024, dtype=np.uint32)
    want = sum(((v >> np.uint32(b)) & 1).astype(np.uint32) << np.uint32(3 * b) for b in range(10))
    assert np.array_equal(spread(v), want)


def test_length_threshold_without_the_square_root():
    """sqrtf(x) > 0.1f exactly when x > 0x1.47ae16p-7f (longer_than_10cm)."""
    t = np.float32(float.fromhex("0x1.47ae16p-7"))
    assert np.sqrt(t) <= np.float32(0.1) < np.sqrt(np.nextafter(t, np.float32(1)))
    rng = np.random.default_rng(1)
    x = np.abs(t + rng.standard_normal(1 << 20).astype(np.float32) * np.float32(1e-6))
    assert np.array_equal(np.sqrt(x) > np.float32(0.1), x > t)


def test_float_quotient_equals_the_rounded_double_quotient():
    """(float)(1.0 / (double)s) == 1.0f / s for normal results (inv_sigma)."""
    rng = np.random.default_rng(2)
    s = np.exp(rng.uniform(-60, 60, 1 << 21)).astype(np.float32)
    assert np.array_equal((1.0 / s.astype(np.float64)).astype(np.float32), np.float32(1) / s)


def test_huber_inlier_loss_in_float():
    """0.5f * (e * e) is the double loss 0.5 e^2 rounded once, up to the largest
    float that is at most 1.345 (mf_robust.cuh)."""
    k = np.float32(float.fromhex("0x1.5851eap+0"))
    assert float(k) <= 1.345 < float(np.nextafter(k, np.float32(2)))
    e = np.random.default_rng(3).uniform(-1, 1, 1 << 21).astype(np.float32) * k
    e = np.concatenate([e, np.float32([0, 1e-15, -1e-15]), k[None], -k[None]])
    want = (0.5 * e.astype(np.float64) ** 2).astype(np.float32)
    assert np.array_equal(np.float32(0.5) * (e * e), want)


def test_constant_division_with_one_correction():
    """div_e2 (mf_track.cu): x / 0.02f as q = x rc; q += rc (x - q b), both
    multiply-adds rounded once, equals the IEEE quotient for every mantissa."""
    b = np.float32(np.float32(0.1) * np.float32(0.1)) * np.float32(2)
    rc = np.float32(1) / b
    assert float(b).hex() == "0x1.47ae160000000p-6" and float(rc).hex() == "0x1.8ffffe0000000p+5"
    x = ((np.uint32(127) << np.uint32(23)) | np.arange(1 << 23, dtype=np.uint32)).view(np.float32)
    q = x * rc
    # q b has 48 bits and x - q b cancels: exact in double, as in the fma
    r = (x.astype(np.float64) - q.astype(np.float64) * np.float64(b)).astype(np.float32)
    got = (r.astype(np.longdouble) * np.longdouble(rc) + q).astype(np.float32)
    assert np.array_equal(got, x / b)


def test_block_coordinate_by_a_round_down_addition():
    """f + (2^26 + 2^25) rounded towards minus infinity is a multiple of 8: its
    low bits are floor(f / 8) for 0 <= f < 4096 (alloc_mark_kernel)."""
    rng = np.random.default_rng(4)
    f = rng.uniform(0, 4096, 1 << 20).astype(np.float32)
    f = np.concatenate([f, np.arange(0, 4096, 8, dtype=np.float32),
                        np.nextafter(np.arange(8, 4097, 8, dtype=np.float32), np.float32(0)),
                        np.float32([0.0, -0.0, 4095.9998])])
    big = np.float64(2 ** 26 + 2 ** 25)
    down = (np.floor((f.astype(np.float64) + big) / 8) * 8).astype(np.float32)
    bits = down.view(np.uint32) - np.uint32(0x4cc00000)
    assert np.array_equal(bits, (f.astype(np.int64) >> 3).astype(np.uint32))


def test_cheap_robust_weights_equal_the_double_formulas(tmp_path):
    """robust_fast (mf_robust.cuh), compiled for the host, returns the floats of
    the double formulas, or leaves the residual to them: thresholds, residuals
    across each kernel's range, extremes, infinities and NaN."""
    import ctypes as C
    import os
    import subprocess
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                        "mid_fusion_b200", "csrc")
    src = tmp_path / "r.cpp"
    src.write_text('#include "mf_robust.cuh"\n'
                   'extern "C" void run(int kind, const float* e, int n, float* w, float* l, '
                   'int* fast) { for (int i = 0; i < n; ++i) '
                   'fast[i] = mf::robust_fast(e[i], kind, w[i], l[i]); }\n')
    so = tmp_path / "r.so"
    subprocess.run(["g++", "-O2", "-std=c++14", "-ffp-contract=off", "-fPIC", "-shared", "-I",
                    csrc, "-o", str(so), str(src)], check=True)
    lib = C.CDLL(str(so))
    rng = np.random.default_rng(6)
    e = np.concatenate([
        rng.normal(scale=s, size=200000) for s in (1e-3, 0.5, 3.0, 50.0)] + [
        np.exp(rng.uniform(-80, 80, 100000)),
        [0.0, 1.345, 4.6851, 2.3849, 1e-30, 1e-45, 3e38, np.inf, np.nan]]).astype(np.float32)
    e = np.concatenate([e, -e, np.nextafter(np.float32([1.345, 4.6851]), np.float32(9))])
    w, loss = np.zeros_like(e), np.zeros_like(e)
    fast = np.zeros(e.size, np.int32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    r = e.astype(np.float64)
    a = np.abs(r)
    with np.errstate(all="ignore"):
        x2 = (r / 2.3849) * (r / 2.3849)
        u = 1.0 - r * r / (4.6851 * 4.6851)
        v = 1.0 - (r / 4.6851) * (r / 4.6851)
        want = {1: (1.345 / a, 1.345 * (a - 0.5 * 1.345), a > 1.345),
                2: (u * u, 4.6851 * 4.6851 / 6.0 * (1.0 - v * v * v), a <= 4.6851),
                3: (1 / (1 + x2), 0.5 * 2.3849 * 2.3849 * np.log(1.0 + x2), a < 1e15)}
        for kind, (ww, ll, domain) in want.items():
            lib.run(kind, p(e), e.size, p(w), p(loss), p(fast))
            on = fast != 0
            assert not np.any(on & ~domain)
            assert np.count_nonzero(on) > 0.999 * np.count_nonzero(domain & (a < 1e14))
            assert np.array_equal(w[on], ww[on].astype(np.float32)), kind
            assert np.array_equal(loss[on], ll[on].astype(np.float32)), kind
