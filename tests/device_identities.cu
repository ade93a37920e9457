// Device arithmetic that stands in for costlier formulas, against those
// formulas, on the device: counts the arguments whose results differ in a bit.
// Built and run by test_gpu_device_identities.py.
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>
#include "mf_exp.cuh"
#include "mf_robust.cuh"
#include "mf_warp.cuh"

namespace {

__device__ bool same(float a, float b) {
  return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b);
}

// the bits of every float, 0 .. 2^32 - 1, over the grid
template <typename F>
__device__ void each_float(F f) {
  const unsigned long long n = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long b = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
       b < (1ULL << 32); b += n)
    f(__uint_as_float((unsigned)b));
}

__global__ void exp_kernel(unsigned long long* bad, float* first) {
  __shared__ double tab[64];
  if (threadIdx.x < 64) tab[threadIdx.x] = mf::c_exp2_64[threadIdx.x];
  __syncthreads();
  const float b = 0.1f * 0.1f * 2;
  each_float([&](float x) {
    if (!(x <= 0.f)) return;
    if (!same(mf::exp_nearest(x, tab), (float)exp((double)x))) {
      atomicAdd(bad, 1ULL);
      *first = x;
    }
    if (!same(mf::exp_nearest(mf::div_e2(x), tab), (float)exp((double)(x / b)))) {
      atomicAdd(bad + 1, 1ULL);
      first[1] = x;
    }
  });
}

// Tracking::calc_robust_weight / calc_robust_residual in double, as the kernels'
// general case takes them
__device__ void robust_double(float e, int kind, float& w, float& loss) {
  const double r = e, a = fabs(r), b = 4.6851;
  double wd = 1.0, l = 0.5 * r * r;
  if (kind == 1 && !(a <= 1.345)) {
    wd = 1.345 / a;
    l = 1.345 * (a - 0.5 * 1.345);
  } else if (kind == 2) {
    const double u = 1.0 - r * r / (b * b), v = 1.0 - (r / b) * (r / b);
    wd = a <= b ? u * u : 0;
    l = a <= b ? b * b / 6.0 * (1.0 - v * v * v) : b * b / 6.0;
  } else if (kind == 3) {
    const double q = (r / 2.3849) * (r / 2.3849);
    wd = 1 / (1 + q);
    l = 0.5 * 2.3849 * 2.3849 * log(1.0 + q);
  }
  w = (float)wd;
  loss = (float)l;
}

__global__ void robust_kernel(int kind, unsigned long long* bad, float* first) {
  each_float([&](float e) {
    float w, l, wd, ld;
    mf::robust(e, kind, w, l);
    robust_double(e, kind, wd, ld);
    if (!same(w, wd) || !same(l, ld)) {
      atomicAdd(bad, 1ULL);
      *first = e;
    }
  });
}

// Gaussian elimination with partial pivoting on [A | I], plain divisions
__device__ void inverse_plain(const float* A, float* out) {
  float a[4][8];
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 8; ++j) a[i][j] = j < 4 ? A[4 * i + j] : (i == j - 4 ? 1.f : 0.f);
  for (int c = 0; c < 4; ++c) {
    int p = c;
    float best = fabsf(a[c][c]);
    for (int r = c + 1; r < 4; ++r)
      if (fabsf(a[r][c]) > best) { best = fabsf(a[r][c]); p = r; }
    if (p != c)
      for (int j = 0; j < 8; ++j) { const float t = a[c][j]; a[c][j] = a[p][j]; a[p][j] = t; }
    for (int r = c + 1; r < 4; ++r) {
      const float f = a[r][c] / a[c][c];
      for (int j = c; j < 8; ++j) a[r][j] -= f * a[c][j];
    }
  }
  for (int j = 0; j < 4; ++j) {
    float R[4];
    for (int r = 3; r >= 0; --r) {
      float s = a[r][4 + j];
      for (int k = r + 1; k < 4; ++k) s -= a[r][k] * R[k];
      R[r] = s / a[r][r];
      out[4 * r + j] = R[r];
    }
  }
}

// one warp per matrix: bad[0] inverse_warp, bad[1] the serial inverse
__global__ void inverse_kernel(const float* A, int n, unsigned long long* bad, float* first) {
  const int lane = threadIdx.x & 31;
  for (int m = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; m < n;
       m += (gridDim.x * blockDim.x) >> 5) {
    const float* a = A + 16 * (long long)m;
    const float e = mf::inverse_warp(a, lane);
    if (lane < 16) {
      float want[16];
      inverse_plain(a, want);
      const mf::M4 S = mf::inverse(mf::load_m4(a));
      const float serial = mf::m_at(S, lane >> 2, lane & 3);
      if (!same(e, want[lane])) { atomicAdd(bad, 1ULL); *first = (float)m; }
      if (!same(serial, want[lane])) { atomicAdd(bad + 1, 1ULL); first[1] = (float)m; }
    }
  }
}

struct Result {
  unsigned long long* bad;
  float* first;
  Result() {
    cudaMalloc(&bad, 16);
    cudaMalloc(&first, 8);
    cudaMemset(bad, 0, 16);
    cudaMemset(first, 0, 8);
  }
  int read(unsigned long long* n, float* f) {
    cudaError_t e = cudaMemcpy(n, bad, 16, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(f, first, 8, cudaMemcpyDeviceToHost);
    cudaFree(bad);
    cudaFree(first);
    return (int)e;
  }
};

}  // namespace

extern "C" int check_exp(unsigned long long* bad, float* first) {
  Result r;
  exp_kernel<<<148 * 8, 256>>>(r.bad, r.first);
  return r.read(bad, first);
}
extern "C" int check_robust(int kind, unsigned long long* bad, float* first) {
  Result r;
  robust_kernel<<<148 * 8, 256>>>(kind, r.bad, r.first);
  return r.read(bad, first);
}
extern "C" int check_inverse(const float* A, int n, unsigned long long* bad, float* first) {
  Result r;
  float* d = nullptr;
  if (cudaMalloc(&d, 64LL * n) != cudaSuccess) return -1;
  cudaMemcpy(d, A, 64LL * n, cudaMemcpyHostToDevice);
  inverse_kernel<<<148 * 4, 256>>>(d, n, r.bad, r.first);
  const int e = r.read(bad, first);
  cudaFree(d);
  return e;
}
