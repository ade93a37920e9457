// 4x4 float matrices by the lanes of one warp, with the bits of the serial
// forms in mf_common.cuh.
#pragma once
#include "mf_common.cuh"

namespace mf {

// inverse(M4) by one warp, the same operations on the same values (so the
// same bits): every lane eliminates A on its own registers (the row swaps are
// uniform branches, rarely taken) and carries one column of the identity,
// lane & 3.  A is read from memory by all lanes: `A` is its 16 floats, row-
// major.  Returns element (lane & 15) of the inverse.
static __device__ __noinline__ float inverse_warp_general(const float* A, int lane) {
  float a[4][4], b[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
#pragma unroll
    for (int k = 0; k < 4; ++k) a[r][k] = A[4 * r + k];
    b[r] = r == (lane & 3) ? 1.f : 0.f;
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    int p = c;
    float best = fabsf(a[c][c]);
#pragma unroll
    for (int r = c + 1; r < 4; ++r)
      if (fabsf(a[r][c]) > best) { best = fabsf(a[r][c]); p = r; }
#pragma unroll
    for (int r = c + 1; r < 4; ++r) {
      if (p == r) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float t = a[c][k]; a[c][k] = a[r][k]; a[r][k] = t;
        }
        const float t = b[c]; b[c] = b[r]; b[r] = t;
      }
    }
#pragma unroll
    for (int r = c + 1; r < 4; ++r) {
      const float f = div0(a[r][c], a[c][c]);
#pragma unroll
      for (int k = c + 1; k < 4; ++k) a[r][k] -= f * a[c][k];  // column c is not read again
      b[r] -= f * b[c];
    }
  }
  float R[4];
#pragma unroll
  for (int r = 3; r >= 0; --r) {
    float s = b[r];
#pragma unroll
    for (int k = r + 1; k < 4; ++k) s -= a[r][k] * R[k];
    R[r] = div0(s, a[r][r]);
  }
  const int i = (lane >> 2) & 3;   // lane's own column is lane & 3, its element's row i
  return i == 0 ? R[0] : i == 1 ? R[1] : i == 2 ? R[2] : R[3];
}

// n / d rounded to float for the d whose reciprocal y is given: n * y is within
// 2^-52 of the quotient, and the quotient of two floats is no closer than
// 2^-49 to the middle between two floats (a middle m has 25 bits, so
// |n - m d| >= 1 in units of the last places, against m d < 2^49).
// For n and d within [2^-60, 2^60], and n = 0 (div_range).
__device__ __forceinline__ float div_by(float n, double y) { return (float)((double)n * y); }
__device__ __forceinline__ bool div_range(float n) {
  return n == 0.f || (fabsf(n) >= 0x1p-60f && fabsf(n) <= 0x1p60f);
}
// 1 / d up to 2^-53: y (1 + e + e^2) with y the approximate float reciprocal.
__device__ __forceinline__ double recip(float d) {
  const double y = __fdividef(1.f, d), e = fma(-(double)d, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// inverse(M4) by one warp for a matrix whose last row is 0 0 0 1, as every
// pose's: with the same bits, since the elimination then subtracts zeros from
// that row, and (general) for any other.  Returns element (lane & 15).
// Bound by the latency of the dependent quotients: as the general elimination
// it was 2.1 k of the GN step's 6.8 k cycles (ten divisions one after the
// other, each with a branch to a slow path); the three pivots' reciprocals are
// taken once here, in double, and serve the back substitution as well, and
// rows swap by selection: an iteration is 1.2 k cycles shorter (camera launch
// 160x120 96 -> 89 us, 640x480 185 -> 175).
__device__ __forceinline__ float inverse_warp(const float* A, int lane) {
  float a[3][4], b[3];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
#pragma unroll
    for (int k = 0; k < 4; ++k) a[r][k] = A[4 * r + k];
    b[r] = r == (lane & 3) ? 1.f : 0.f;
  }
  bool ok = __float_as_int(A[12]) == 0 && __float_as_int(A[13]) == 0 &&
            __float_as_int(A[14]) == 0 && A[15] == 1.f;
  double y[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    int p = c;
    float best = fabsf(a[c][c]);
#pragma unroll
    for (int r = c + 1; r < 3; ++r)
      if (fabsf(a[r][c]) > best) { best = fabsf(a[r][c]); p = r; }
    ok = ok && best >= 0x1p-60f && best <= 0x1p60f;
#pragma unroll
    for (int k = c; k < 5; ++k) {
      const float t = k < 4 ? a[c][k & 3] : b[c];
      float u = t;
#pragma unroll
      for (int r = c + 1; r < 3; ++r) {
        const float s = k < 4 ? a[r][k & 3] : b[r];
        u = p == r ? s : u;
        if (k < 4) a[r][k & 3] = p == r ? t : s;
        else b[r] = p == r ? t : s;
      }
      if (k < 4) a[c][k & 3] = u;
      else b[c] = u;
    }
    y[c] = recip(a[c][c]);
#pragma unroll
    for (int r = c + 1; r < 3; ++r) {
      ok = ok && div_range(a[r][c]);
      const float f = div_by(a[r][c], y[c]);
#pragma unroll
      for (int k = c + 1; k < 4; ++k) a[r][k] -= f * a[c][k];  // column c is not read again
      b[r] -= f * b[c];
    }
  }
  float R[4];
  R[3] = (lane & 3) == 3 ? 1.f : 0.f;
#pragma unroll
  for (int r = 2; r >= 0; --r) {
    float s = b[r];
#pragma unroll
    for (int k = r + 1; k < 4; ++k) s -= a[r][k] * R[k];
    ok = ok && div_range(s);
    R[r] = div_by(s, y[r]);
  }
  if (!__all_sync(0xffffffffu, ok)) return inverse_warp_general(A, lane);
  const int i = (lane >> 2) & 3;   // lane's own column is lane & 3, its element's row i
  return i == 0 ? R[0] : i == 1 ? R[1] : i == 2 ? R[2] : R[3];
}

// mul(A, B) by the lanes of one warp, element (lane & 15), A and B row-major.
__device__ __forceinline__ float mul_warp(const float* A, const float* B, int lane) {
  const int i = (lane >> 2) & 3, j = lane & 3;
  float s = A[4 * i] * B[j];
#pragma unroll
  for (int k = 1; k < 4; ++k) s += A[4 * i + k] * B[4 * k + j];
  return s;
}

}  // namespace mf
