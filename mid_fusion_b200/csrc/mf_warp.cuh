// 4x4 float matrices by the lanes of one warp, with the bits of the serial
// forms in mf_common.cuh.
#pragma once
#include "mf_common.cuh"

namespace mf {

// inverse(M4) by one warp, the same operations on the same values (so the
// same bits): every lane eliminates A on its own registers (the row swaps are
// uniform branches, rarely taken) and carries one column of the identity,
// lane & 3.  A is read from memory by all lanes: `A` is its 16 floats, row-
// major.  Returns element (lane & 15) of the inverse.  (One column of [A | I]
// per lane, its pivots and factors moved by 40 shuffles, took 2.8 k cycles of
// the GN step's 7.5 k; this form 2.1 k.)
__device__ __forceinline__ float inverse_warp(const float* A, int lane) {
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
      const float f = a[r][c] / a[c][c];
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
    R[r] = s / a[r][r];
  }
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
