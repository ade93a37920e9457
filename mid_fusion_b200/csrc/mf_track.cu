// ICP + photometric Gauss-Newton tracking on the device.
//
// Reference: apps/kfusion/src/cpp/tracking/tracking.cpp (Tracking) and
// apps/kfusion/src/cpp/preprocessing/*.  The whole coarse-to-fine GN of a
// stage (the camera, or all moving objects at once) is one launch: per
// iteration its CTAs evaluate the ICP row and the photometric row of every
// pixel of the level, weight them (IRLS), and reduce the 29 sums of the normal
// equations plus the three outlier counts:
//   - per thread in FP32 over at most GN_PIX_MAX pixels (2 rows each), so no
//     FP32 sum runs over more than 2 * GN_PIX_MAX terms,
//   - per warp / block / grid in FP64 (fixed summation order, so results are
//     bitwise reproducible run to run),
// and every CTA of a problem then runs the same GN step on its own copy of the
// problem (cost test, step back, FP64 6x6 solve, SE(3) update, convergence
// test).  The host only launches.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>
#include "mf_exp.cuh"
#include "mf_internal.h"
#include "mf_robust.cuh"
#include "mf_solve.cuh"
#include "mf_warp.cuh"

namespace mf {

constexpr float INVALIDF = -2.f;
constexpr int GN_THREADS = 256;
#ifndef MF_GN_PIX0
#define MF_GN_PIX0 3
#endif
#ifndef MF_GN_MINB
#define MF_GN_MINB 3
#endif
// pixels per thread per iteration at level 0 (1 above): 3 makes the 640x480
// level one wave of 400 CTAs on 148 SMs x 3 resident (2: 600 CTAs in two
// waves, 30.9 us per launch against 24.8 us)
constexpr int GN_PIX_MAX = MF_GN_PIX0;
__host__ __device__ constexpr int gn_pix(int L) { return L == 0 ? GN_PIX_MAX : 1; }

struct GNState {
  double T[16], prevT[16];
  double prev_err;
  int done;
  int kind;          // 0 camera, 1 object
  int label;
  int inst;
  int iters[MAX_PYR];
  int fallback;
  int ticket;
  int pad_;
  // objects: bounding box (x0, y0, x1, y1) of the object's pixels in the
  // full-resolution model label map; empty when x1 < x0
  int box[4];
  M4 Tf, invTf;      // float pose (and inverse) seen by the per-pixel kernels
  M4 evalTf;         // the pose of the last GN evaluation (Tf when gn_step ran)
  M4 T_w_r, inv_T_w_r, view;               // camera: reference pose, K * inverse(T_w_r)
  M4 T_c1_o1, inv_T_c1_o1, inv_T_w_o1, T_w_c2;  // object constants
  M4 T_w_o1;         // object: the volume pose before this frame's tracking
  M4 T_virtual;      // object: virtual camera pose T_w_o1 inverse(T_c2_o2) after tracking
  double sums[MAX_PYR][32];
};

struct PyrPtrs {
  int w[MAX_PYR], h[MAX_PYR];
  float* D[MAX_PYR];
  float* I[2][MAX_PYR];
  F3* V[2][MAX_PYR];
  F3* N[MAX_PYR];
  float* GX[MAX_PYR];
  float* GY[MAX_PYR];
  F3* COV[MAX_PYR];
  uint8_t* MASK[MAX_PYR];
};

struct TrackState {
  int levels = 0;
  PyrPtrs pyr{};
  int cur = 0;                      // live set; 1 - cur holds the reference frame
  bool have_ref = false;
  bool tracked = false;             // the reference pose of this frame is saved
  float* rD[MAX_INSTANCES][MAX_PYR] = {};
  F3* rV[MAX_INSTANCES][MAX_PYR] = {};
  GNState* d_state = nullptr;       // MAX_INSTANCES (slot 0: camera, slot i: object i)
  int slot_kind[MAX_INSTANCES];     // per slot: -1 never set up, else the GNState kind
  unsigned* d_gnbar = nullptr;      // MAX_INSTANCES: each problem's barrier arrivals
  double* d_gnrows = nullptr;       // 2 x GN_CAM_ROWS x 32 partial sums of the camera's GN
  int coop_blocks = 0, obj_blocks = 0;  // co-resident CTAs of gn_camera_kernel, gn_objects_kernel
  double* d_objrows = nullptr;      // 2 x max_instances x max_tiles x 32 tile sums of the objects
  uint8_t* d_objlive = nullptr;     // 2 x max_instances x max_tiles
  double* d_partials = nullptr;     // max_tiles x 32 (one evaluation at a time)
  int max_tiles = 0;
  float2* d_zr = nullptr;           // MAX_PYR x max_tiles live depth range per CTA tile
  float2* d_zs = nullptr;           // MAX_PYR x max_segs, per 32-pixel segment
  int max_segs = 0;
  float* d_Twc_prev = nullptr;      // camera pose of the previous frame
  uint8_t* d_mask0 = nullptr;       // full-resolution ICP outlier mask
  float gaussian[5];
  std::vector<void*> allocs;
  // camera cost and adjoint (allocated on first use)
  double* d_gmodel = nullptr;       // 2 x 3 x W x H: dE/d model vertex, dE/d model normal
  double* d_cost_part = nullptr;    // per-CTA partials of the cost rows, 8 each
  double* d_cost = nullptr;         // 8: cost, dE/d twist (6), rows
  F4* d_win_hit = nullptr;          // W x H: the hit of the raycast's winner per pixel (for
  uint8_t* d_win = nullptr;         // TSDF gradients), and behind them the winners
  int cost_blocks = 0;
  // motion residuals (allocated on first use)
  int8_t* d_mres = nullptr;         // 2 x W x H result codes: ICP rows, then photometric
  float* d_merr = nullptr;          // 2 x W x H errors
  F3* d_lvert = nullptr;            // model raycast at the live pose: vertex, normal, label
  F3* d_lnorm = nullptr;
  int* d_llabel = nullptr;
  int* d_mcount = nullptr;          // 2 x MAX_INSTANCES: object pixels, inliers
};

// ------------------------------------------------------------------ preprocessing
struct Gauss25 { float g[25]; };   // g[5 * i + j] = gaussian[i] * gaussian[j]

// bilateralFilterKernel, preprocessing.cpp:11-50 (e_d = 0.1, r = 2) on the
// intensity (z = 0) and the depth (z = 1).  Neighbour coordinates clamp to the
// image (the reference's host clamp on unsigned values goes through int min/max,
// utils/cutil_math.h:51-57, 987-989).  The range weight is the reference's
// expf of the same float argument, rounded to the nearest float
// (exp_nearest), as the host's expf is in all but rare cases (measured on a
// 640x480 frame: 99.94 % of the filtered pixels equal the reference's bit for
// bit, against 72 % with the single-precision expf, whose results differ from
// the nearest float by up to 2 ulp); every later stage inherits the
// difference.
// Bound by instruction issue, the FP64 of the 25 weights above all.  A CTA
// stages its 32 x 8 pixels and their border in shared memory (the taps' index
// arithmetic and bounds go with it).  640x480, both planes: 52 us with the general
// double exp and loads from global memory, now 32; 1280x720 144, now 85.
constexpr int BIL_W = 32, BIL_H = 8;
__global__ void __launch_bounds__(BIL_W * BIL_H)
bilateral_kernel(const float* __restrict__ grey, const float* __restrict__ depth,
                 float* __restrict__ out_i, float* __restrict__ out_d, int W, int H, Gauss25 gs) {
  __shared__ float tile[BIL_H + 4][BIL_W + 4];
  __shared__ double tab[64];
  const float* in = blockIdx.z == 0 ? grey : depth;
  float* out = blockIdx.z == 0 ? out_i : out_d;
  const int x0 = blockIdx.x * BIL_W, y0 = blockIdx.y * BIL_H;
  if (threadIdx.x < 64) tab[threadIdx.x] = c_exp2_64[threadIdx.x];
  for (int i = threadIdx.x; i < (BIL_W + 4) * (BIL_H + 4); i += BIL_W * BIL_H) {
    const int tx = i % (BIL_W + 4), ty = i / (BIL_W + 4);
    const int cx = imn(imx(x0 + tx - 2, 0), W - 1), cy = imn(imx(y0 + ty - 2, 0), H - 1);
    tile[ty][tx] = in[cx + cy * W];
  }
  __syncthreads();
  const int lx = threadIdx.x % BIL_W, ly = threadIdx.x / BIL_W;
  const int x = x0 + lx, y = y0 + ly;
  if (x >= W || y >= H) return;
  const float center = tile[ly + 2][lx + 2];
  float sum = 0.0f, t = 0.0f;
  if (center != 0) {
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        const float cur = tile[ly + j][lx + i];
        if (cur > 0) {
          const float mod = sq(cur - center);
          const float factor = gs.g[5 * i + j] * exp_nearest(div_e2(-mod), tab);
          t += factor * cur;
          sum += factor;
        }
      }
  }
  out[x + y * W] = center == 0 ? 0.f : t / sum;
}

// halfSampleRobustImageKernel, preprocessing.cpp:161-196 (e_d = 0.3, r = 1), on
// the 2 x 2 pixels `at(dx, dy)` of the finer level.
template <typename At>
__device__ __forceinline__ float half_sampled(At at, float e_d) {
  const float center = at(0, 0);
  float sum = 0.0f, t = 0.0f;
#pragma unroll
  for (int i = 0; i <= 1; ++i)
#pragma unroll
    for (int j = 0; j <= 1; ++j) {
      const float cur = at(j, i);
      if (fabsf(cur - center) < e_d) { sum += 1.0f; t += cur; }
    }
  return div0(t, sum);
}

// Levels 2 and up of a HALF_T x HALF_T tile of level 1 that the CTA's threads
// have just computed, through shared memory; out(level, x, y, value) for each
// pixel.  Tiles start at multiples of HALF_T, so a pixel's 2 x 2 is in its tile.
constexpr int HALF_T = 16;
template <typename Out>
__device__ __forceinline__ void half_sample_tile(float (*tile)[HALF_T][HALF_T], float mine,
                                                 const int* w, const int* h, int levels,
                                                 float e_d, Out out) {
  const int tx = threadIdx.x % HALF_T, ty = threadIdx.x / HALF_T;
  tile[0][ty][tx] = mine;
#pragma unroll
  for (int l = 2; l < MAX_PYR; ++l) {
    if (l >= levels) break;
    __syncthreads();
    const int side = HALF_T >> (l - 1);
    const int x = blockIdx.x * side + tx, y = blockIdx.y * side + ty;
    if (tx < side && ty < side && x < w[l] && y < h[l]) {
      const float v = half_sampled(
          [&](int dx, int dy) { return tile[l & 1][2 * ty + dy][2 * tx + dx]; }, e_d);
      tile[(l & 1) ^ 1][ty][tx] = v;
      out(l, x, y, v);
    }
  }
}

// Every level of the pyramid of intensity (z = 0) and depth (z = 1) in one
// launch (640x480, three levels: 7.1 us by level, now 4.1 and a launch less).
struct HalfLevels {
  const float* in[2];
  float* out[2][MAX_PYR];
  int w[MAX_PYR], h[MAX_PYR];
  int levels;
};
__global__ void __launch_bounds__(HALF_T * HALF_T)
half_sample_levels_kernel(const __grid_constant__ HalfLevels m, float e_d) {
  __shared__ float tile[2][HALF_T][HALF_T];
  const int x = blockIdx.x * HALF_T + threadIdx.x % HALF_T;
  const int y = blockIdx.y * HALF_T + threadIdx.x / HALF_T;
  const int plane = blockIdx.z;
  const float* in = m.in[plane];
  float mine = 0.f;
  if (x < m.w[1] && y < m.h[1]) {
    mine = half_sampled(
        [&](int dx, int dy) { return in[2 * x + dx + (2 * y + dy) * m.w[0]]; }, e_d);
    m.out[plane][1][x + y * m.w[1]] = mine;
  }
  half_sample_tile(tile, mine, m.w, m.h, m.levels, e_d, [&](int l, int px, int py, float v) {
    m.out[plane][l][px + py * m.w[l]] = v;
  });
}

// depth2vertexKernel, preprocessing.cpp:52-71.
__device__ __forceinline__ F3 depth2vertex_at(float d, int x, int y, const M4& invK) {
  return d > 0 ? d * rotate(invK, mk3((float)x, (float)y, 1.f)) : mk3(0.f);
}

// The planes of every level of the live pyramid; the level kernels below take
// the level from blockIdx.y, so one launch covers all levels.
struct LevelMaps {
  const float* D[MAX_PYR];
  F3* V[MAX_PYR];
  const float* I[MAX_PYR];
  F3* N[MAX_PYR];
  float* GX[MAX_PYR];
  float* GY[MAX_PYR];
  F3* COV[MAX_PYR];
  uint8_t* MASK[MAX_PYR];
  int w[MAX_PYR], h[MAX_PYR];
  M4 invK[MAX_PYR];
  float focal[MAX_PYR];
  int negy;             // fy < 0 (the ICL-NUIM convention): up and down swap
};

// vertex2normalKernel<SDF, NegY> (preprocessing.h:39-81; NegY when fy < 0,
// tracking.cpp:805-810), gradientsKernel (preprocessing.cpp:235-246, borders
// untouched) and calc_icp_cov (tracking.cpp:845-871, sigma_xy = sigma_disp = 1,
// baseline 0.075).
__device__ __forceinline__ void normal_grad_cov_px(F3* __restrict__ V,
                                                   const float* __restrict__ I,
                                                   const float* __restrict__ D,
                                                   F3* __restrict__ N, float* __restrict__ GX,
                                                   float* __restrict__ GY, F3* __restrict__ COV,
                                                   int w, int h, const M4& invK, float focal,
                                                   int negy, int p) {
  const int x = p % w, y = p / w;
  const int xl = imx(x - 1, 0), xr = imn(x + 1, w - 1);
  const int ylo = imx(y - 1, 0), yhi = imn(y + 1, h - 1);
  const int yd = negy ? yhi : ylo, yu = negy ? ylo : yhi;
  const float d = D[p];
  const F3 left = depth2vertex_at(D[xl + w * y], xl, y, invK);
  const F3 right = depth2vertex_at(D[xr + w * y], xr, y, invK);
  const F3 down = depth2vertex_at(D[x + w * yd], x, yd, invK);
  const F3 up = depth2vertex_at(D[x + w * yu], x, yu, invK);
  V[p] = depth2vertex_at(d, x, y, invK);
  if (left.z == 0 || right.z == 0 || up.z == 0 || down.z == 0) {
    N[p].x = INVALIDF;  // the other components keep their previous values
  } else {
    N[p] = normalize(cross(up - down, right - left));
  }
  if (x >= 1 && y >= 1 && x < w - 1 && y < h - 1) {
    GX[p] = (I[p + 1] - I[p - 1]) * 0.5f;
    GY[p] = (I[p + w] - I[p - w]) * 0.5f;
  }
  F3 c;
  c.x = (d / focal) * 1.0f;
  c.y = (d / focal) * 1.0f;
  c.z = (d * d * 1.0f) / (focal * 0.075f);
  c.x = c.x * c.x; c.y = c.y * c.y; c.z = c.z * c.z;
  COV[p] = c;
}

// normal_grad_cov_px on every level (vertices included: a pixel's neighbours
// are recomputed from their depths, as cheap as loading them and a launch less:
// 640x480 4.9 + 9.1 us, now 11.4); it also clears the level's ICP outlier
// mask (no pixel is masked until the camera track sets one) unless MASK is
// null (the mask is then written whole by the camera's mask kernel).
__global__ void normal_grad_cov_levels_kernel(LevelMaps m) {
  const int l = blockIdx.y;
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= m.w[l] * m.h[l]) return;
  normal_grad_cov_px(m.V[l], m.I[l], m.D[l], m.N[l], m.GX[l], m.GY[l], m.COV[l], m.w[l],
                     m.h[l], m.invK[l], m.focal[l], m.negy, p);
  if (m.MASK[l]) m.MASK[l][p] = 0;
}

struct SlotPtrs { float* D[MAX_INSTANCES]; };

// vertex2depth (preprocessing.cpp:292-309) of the model vertex map -- for an
// object, its own map: the composite where label == object, 0 elsewhere
// (rendering.cpp:153-178) -- seen from the reference camera (T_w_r for the
// camera problem, T_w_c1 for an object; its inverse is kept in inv_T_w_r).
// For an object it also gathers the bounding box of the object's pixels in the
// label map (warp-reduced atomics); the object rows use it to skip gathers that
// can only find other labels.
__global__ void render_depth_kernel(const F3* __restrict__ vertex, const int* __restrict__ label,
                                    GNState* __restrict__ st, IdList slots, SlotPtrs sp,
                                    int W, int WH) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  GNState& S = st[slots.v[blockIdx.y]];
  bool mine = false;
  if (p < WH) {
    F3 v = vertex[p];
    if (S.kind == 1) {
      mine = label[p] == S.label;
      if (!mine) v = mk3(0.f);
    }
    sp.D[blockIdx.y][p] = v.z > 0.0 ? xform(S.inv_T_w_r, v).z : 0.f;
  }
  if (S.kind != 1) return;
  const int x = mine ? p % W : INT_MAX, y = mine ? p / W : INT_MAX;
  const int x0 = __reduce_min_sync(0xffffffffu, x), y0 = __reduce_min_sync(0xffffffffu, y);
  const int x1 = __reduce_max_sync(0xffffffffu, mine ? x : -1);
  const int y1 = __reduce_max_sync(0xffffffffu, mine ? y : -1);
  if ((threadIdx.x & 31) == 0 && x1 >= 0) {
    atomicMin(&S.box[0], x0); atomicMin(&S.box[1], y0);
    atomicMax(&S.box[2], x1); atomicMax(&S.box[3], y1);
  }
}

// The rendered reference depth and vertex planes of every slot at every level,
// from the rendered depth D[0], in one launch (640x480: 11.5 us by level and
// kernel in three launches, now 6.5).  A thread takes 2 x 2 pixels of level 0 and theirs of level 1.
struct SlotLevels {
  float* D[MAX_PYR][MAX_INSTANCES];
  F3* V[MAX_PYR][MAX_INSTANCES];
  int w[MAX_PYR], h[MAX_PYR];
  int levels;
  M4 invK[MAX_PYR];
};
__global__ void __launch_bounds__(HALF_T * HALF_T)
reference_levels_kernel(const __grid_constant__ SlotLevels sl, float e_d) {
  __shared__ float tile[2][HALF_T][HALF_T];
  const int x = blockIdx.x * HALF_T + threadIdx.x % HALF_T;
  const int y = blockIdx.y * HALF_T + threadIdx.x / HALF_T;
  const int s = blockIdx.z, w0 = sl.w[0], h0 = sl.h[0];
  const float* D0 = sl.D[0][s];
  F3* V0 = sl.V[0][s];
  float d[2][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int px = 2 * x + j, py = 2 * y + i;
      if (px < w0 && py < h0) {
        d[i][j] = D0[px + py * w0];
        V0[px + py * w0] = depth2vertex_at(d[i][j], px, py, sl.invK[0]);
      }
    }
  if (sl.levels < 2) return;
  float mine = 0.f;
  if (x < sl.w[1] && y < sl.h[1]) {
    mine = half_sampled([&](int dx, int dy) { return d[dy][dx]; }, e_d);
    sl.D[1][s][x + y * sl.w[1]] = mine;
    sl.V[1][s][x + y * sl.w[1]] = depth2vertex_at(mine, x, y, sl.invK[1]);
  }
  half_sample_tile(tile, mine, sl.w, sl.h, sl.levels, e_d, [&](int l, int px, int py, float v) {
    sl.D[l][s][px + py * sl.w[l]] = v;
    sl.V[l][s][px + py * sl.w[l]] = depth2vertex_at(v, px, py, sl.invK[l]);
  });
}

// ------------------------------------------------------------------ GN setup
// retrack: the second trackLiveFrame of a frame (kfusion.cpp:370-373), from
// the tracked pose against the same reference pose, which stays saved.
__global__ void setup_camera_kernel(GNState* st, const float* __restrict__ Twc,
                                    float* __restrict__ Twc_prev, F4 k, int retrack,
                                    unsigned* __restrict__ bar) {
  // one warp, element `lane` of the matrices per lane (one thread: 6.2 us,
  // the inverses' serial chains; now 3.9)
  const int lane = threadIdx.x, e = lane & 15;
  __shared__ float sT[16], sR[16], sI[16], sK[16];
  GNState& S = st[0];
  const float t = Twc[e];
  const float tr = retrack ? Twc_prev[e] : t;
  const M4 K = camera_matrix(k);
  if (lane < 16) {
    if (!retrack) Twc_prev[e] = t;
    sT[e] = t;
    sR[e] = tr;
    sK[e] = m_at(K, e >> 2, e & 3);
    S.T[e] = S.prevT[e] = (double)t;
  }
  if (lane == 0) {
    *bar = 0;   // the grid barrier of this problem's GN launch
    S.kind = 0; S.label = 0; S.inst = 0; S.done = 0; S.ticket = 0; S.fallback = 0;
    for (int l = 0; l < MAX_PYR; ++l) S.iters[l] = 0;
  }
  __syncwarp();
  const float ir = inverse_warp(sR, lane), it = inverse_warp(sT, lane);
  if (lane < 16) sI[e] = ir;
  __syncwarp();
  const float view = mul_warp(sK, sI, lane);  // tracking.cpp:258
  if (lane < 16) {
    reinterpret_cast<float*>(&S.T_w_r)[e] = tr;
    reinterpret_cast<float*>(&S.inv_T_w_r)[e] = ir;
    reinterpret_cast<float*>(&S.view)[e] = view;
    reinterpret_cast<float*>(&S.Tf)[e] = t;
    reinterpret_cast<float*>(&S.invTf)[e] = it;
    reinterpret_cast<float*>(&S.evalTf)[e] = t;
  }
}

// trackEachObject setup, tracking.cpp:586-593: T_c1_o1 = inverse(T_w_c1) T_wo1,
// T_c2_o2 = inverse(T_w_c2) T_wo1 with T_w_c2 the freshly tracked camera.
// The part that does not need T_w_c2 (the previous camera pose, the object's
// last pose, the rendered reference's label box) and the part that does.
__device__ void setup_object_post(GNState& S, const M4& T_w_c2) {
  S.T_w_c2 = T_w_c2;
  const M4 T0 = mul(inverse(T_w_c2), S.T_w_o1);
  for (int i = 0; i < 16; ++i) {
    S.T[i] = (double)m_at(T0, i / 4, i % 4);
    S.prevT[i] = S.T[i];
  }
  S.Tf = T0;
  S.invTf = inverse(T0);
  S.evalTf = T0;
}

__global__ void setup_objects_pre_kernel(GNState* st, unsigned* __restrict__ bar, IdList slots,
                                         const float* __restrict__ Twc1,
                                         const float* __restrict__ Two,
                                         const int* __restrict__ inst_label) {
  // one warp per object, element `lane` of the matrices per lane (one thread
  // per object: 8.4 us for three; now 4.6)
  const int lane = threadIdx.x & 31, e = lane & 15, w = threadIdx.x >> 5;
  const int t = blockIdx.x * (blockDim.x >> 5) + w;
  if (t >= slots.n) return;
  const int s = slots.v[t];
  __shared__ float sm[4][4][16];
  float *c1 = sm[w][0], *o1 = sm[w][1], *ic1 = sm[w][2], *c1o1 = sm[w][3];
  GNState& S = st[s];
  const float two = Two[16 * s + e];
  if (lane < 16) {
    c1[e] = Twc1[e];
    o1[e] = two;
  }
  if (lane == 0) {
    bar[s] = 0;   // the barrier of this problem's CTAs
    S.kind = 1; S.inst = s; S.label = inst_label[s]; S.done = 0; S.ticket = 0; S.fallback = 0;
    for (int l = 0; l < MAX_PYR; ++l) S.iters[l] = 0;
    S.box[0] = S.box[1] = INT_MAX;
    S.box[2] = S.box[3] = -1;
  }
  __syncwarp();
  const float ir = inverse_warp(c1, lane), io = inverse_warp(o1, lane);
  if (lane < 16) ic1[e] = ir;
  __syncwarp();
  const float m = mul_warp(ic1, o1, lane);
  if (lane < 16) c1o1[e] = m;
  __syncwarp();
  const float im = inverse_warp(c1o1, lane);
  if (lane < 16) {
    reinterpret_cast<float*>(&S.inv_T_w_r)[e] = ir;
    reinterpret_cast<float*>(&S.T_c1_o1)[e] = m;
    reinterpret_cast<float*>(&S.inv_T_c1_o1)[e] = im;
    reinterpret_cast<float*>(&S.inv_T_w_o1)[e] = io;
    reinterpret_cast<float*>(&S.T_w_o1)[e] = two;
  }
}
__global__ void setup_objects_post_kernel(GNState* st, IdList slots, const float* __restrict__ Twc2) {
  const int t = threadIdx.x;
  if (t >= slots.n) return;
  setup_object_post(st[slots.v[t]], load_m4(Twc2));
}

__global__ void finalize_camera_kernel(const GNState* st, float* __restrict__ Twc) {
  store_m4(Twc, to_m4f(st[0].T));
}

// volume_pose_ = T_w_c2 * T_c2_o2, tracking.cpp:695.
// trackEachObject's outputs, tracking.cpp:695-696: the volume pose
// T_w_c2 T_c2_o2 and the virtual camera pose T_w_o1 inverse(T_c2_o2).
__global__ void finalize_objects_kernel(GNState* st, IdList slots, float* __restrict__ Two) {
  const int t = threadIdx.x;
  if (t >= slots.n) return;
  const int s = slots.v[t];
  const M4 Tco = to_m4f(st[s].T);
  store_m4(Two + 16 * s, mul(st[s].T_w_c2, Tco));
  st[s].T_virtual = mul(st[s].T_w_o1, inverse(Tco));
}

// ------------------------------------------------------------------ GN step
// One GN iteration's decision logic (tracking.cpp:287-335, objects :657-686):
// cost test with step back, solve, convergence test, left-multiplied update.
MF_HD void gn_step(GNState& S, const double* s, int level) {
  // work on register copies; one copy-out at the end
  double T[16], P[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) { T[i] = S.T[i]; P[i] = S.prevT[i]; }
  S.evalTf = S.Tf;   // the rows just summed were evaluated here
  const double prev_err = S.prev_err;
  const double err = s[0] / s[28];
  int done = 0, fallback = 0;
  if (S.kind == 1 && s[28] == 0) {  // no valid row: the object loop stops (:674-676)
    S.done = 1;
    S.iters[level] += 1;
    return;
  }
  if (err > prev_err) {
#pragma unroll
    for (int i = 0; i < 16; ++i) T[i] = P[i];
    done = 1;
  } else {
    S.prev_err = err;
    double A[6][6], b[6], x[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) b[i] = s[1 + i];
    make_jtj(s + 7, A);
    if (solve6(A, b, x)) fallback = 1;
    double nx = 0;
#pragma unroll
    for (int i = 0; i < 6; ++i) nx += x[i] * x[i];
    if (sqrt(nx) < (double)1e-05f && sqrt(s[0] / s[28]) < 2e-3) {
      done = 1;
    } else {
      double E[16], R[16];
      se3_exp(x, E);
      mul4d(E, T, R);
#pragma unroll
      for (int i = 0; i < 16; ++i) { P[i] = T[i]; T[i] = R[i]; }
    }
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) { S.T[i] = T[i]; S.prevT[i] = P[i]; }
  S.done = done;
  if (fallback) S.fallback = 1;
  S.iters[level] += 1;
  const M4 Tf = to_m4f(T);
  S.Tf = Tf;
  S.invTf = inverse(Tf);
}

// gn_step by one whole warp (every lane of the calling warp, converged), with
// the same operations in the same order on every value, so the results equal
// the serial gn_step's bit for bit.  The serial step holds the 6x6 system, the
// poses and the update in one thread and spills at the GN kernels' register
// budget; here lane i < 6 holds row i of the system, lane l < 16 element l of
// the poses, and values move by shuffles.
// first: the level's first iteration (prev_err starts at infinity).
constexpr unsigned FULL_MASK = 0xffffffffu;

// A[i][j] of the symmetric normal matrix from the 21 packed sums (makeJTJ).
__device__ __forceinline__ double jtj_at(const double* v21, int i, int j) {
  const int a = i < j ? i : j, b = i < j ? j : i;
  return v21[a * 6 - a * (a - 1) / 2 + (b - a)];
}

// solve6_eigen by one warp, the same operations on the same values (so the same
// bits): the rotation's coefficients on every lane, its three loops over k on
// lanes (columns of A and V at once, then the rows of A), the projections and
// the result's components on lanes.  x on all lanes.  On one lane with the
// matrices in local memory an iteration that needed it took some 250 us longer
// (frames with such an object: 1.95 ms of object GN against 0.93).
__device__ __noinline__ void solve6_eigen_warp(const double* s, int lane, double condition,
                                               double x[6]) {
  __shared__ double A[6][6], V[6][6], coef[6], xs[6];
  for (int e = lane; e < 36; e += 32) {
    const int i = e / 6, j = e % 6;
    A[i][j] = jtj_at(s + 7, i, j);
    V[i][j] = i == j ? 1.0 : 0.0;
  }
  __syncwarp();
  for (int sweep = 0; sweep < 60; ++sweep) {
    double off = 0;
    for (int p = 0; p < 6; ++p)
      for (int q = p + 1; q < 6; ++q) off += A[p][q] * A[p][q];
    if (off < 1e-300) break;
    for (int p = 0; p < 6; ++p)
      for (int q = p + 1; q < 6; ++q) {
        const double apq = A[p][q];
        if (apq == 0) continue;
        const double theta = (A[q][q] - A[p][p]) / (2 * apq);
        const double ta = fabs(theta);
        double t, c;
        if (ta > 0x1p28) {
          // theta^2 + 1 rounds to theta^2 and t^2 + 1 to 1, so both square
          // roots are exact: t = 1 / (2 |theta|) (0 once theta^2 overflows)
          t = ta > 0x1.fffffffffffffp511 ? 0.0 : 1.0 / (ta + ta);
          t = theta >= 0 ? t : -t;
          c = 1.0;
        } else {
          t = (theta >= 0 ? 1.0 : -1.0) / (ta + sqrt(theta * theta + 1));
          c = 1 / sqrt(t * t + 1);
        }
        const double sn = t * c;
        __syncwarp();
        if (lane < 12) {
          double(*M)[6] = lane < 6 ? A : V;
          const int k = lane < 6 ? lane : lane - 6;
          const double mp = M[k][p], mq = M[k][q];
          M[k][p] = c * mp - sn * mq;
          M[k][q] = sn * mp + c * mq;
        }
        __syncwarp();
        if (lane < 6) {
          const double ap = A[p][lane], aq = A[q][lane];
          A[p][lane] = c * ap - sn * aq;
          A[q][lane] = sn * ap + c * aq;
        }
        __syncwarp();
      }
  }
  double smax = 0;
#pragma unroll
  for (int i = 0; i < 6; ++i) smax = fmax(smax, fabs(A[i][i]));
  const int k = lane < 6 ? lane : 5;
  const double sk = fabs(A[k][k]);
  const bool use = sk > smax / condition && sk != 0;
  double vb = 0;
#pragma unroll
  for (int i = 0; i < 6; ++i) vb += V[i][k] * s[1 + i];
  if (lane < 6) coef[lane] = vb / A[lane][lane];
  const unsigned used = __ballot_sync(FULL_MASK, use);
  __syncwarp();
  double xi = 0;
  for (int j = 0; j < 6; ++j)
    if ((used >> j) & 1u) xi += coef[j] * V[k][j];
  if (lane < 6) xs[lane] = xi;
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 6; ++i) x[i] = xs[i];
  __syncwarp();
}

// solve6 with row i of the eliminated system on lane i < 6 (lanes 6..31
// repeat row 5): the pivot row reaches every lane by shuffles; x (all lanes)
// and the fallback flag as solve6 gives them.
__device__ __forceinline__ bool solve6_warp(const double* s, int lane, double x[6]) {
  const double* v21 = s + 7;
  const int r = lane < 6 ? lane : 5;
  double a[6], c = s[1 + r];
#pragma unroll
  for (int k = 0; k < 6; ++k) a[k] = jtj_at(v21, r, k);
  double piv[6], pmax = 0;
  bool ok = true;
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    double pr[6];
#pragma unroll
    for (int k = j; k < 6; ++k) pr[k] = __shfl_sync(FULL_MASK, a[k], j);
    const double pc = __shfl_sync(FULL_MASK, c, j);
    piv[j] = pr[j];
    pmax = fmax(pmax, pr[j]);
    ok = ok && (pr[j] > 0);
    const double f = a[j] / pr[j];
#pragma unroll
    for (int k = j; k < 6; ++k) a[k] = r != j ? a[k] - f * pr[k] : a[k];
    c = r != j ? c - f * pc : c;
  }
#pragma unroll
  for (int j = 0; j < 6; ++j) ok = ok && (piv[j] > 1e-5 * pmax);
  if (!ok) {  // the truncated eigen solve
    solve6_eigen_warp(s, lane, 1e6, x);
    return true;
  }
  const double xr = c / a[r];
#pragma unroll
  for (int i = 0; i < 6; ++i) x[i] = __shfl_sync(FULL_MASK, xr, i);
  return false;
}

__device__ __noinline__ void gn_step_warp(GNState* Sp, const double* s, int level, int first) {
  GNState& S = *Sp;
  const int lane = threadIdx.x & 31;
  const int e = lane & 15;                 // pose element of this lane
  const int kind = S.kind;
  const double prev_err = first ? INFINITY : S.prev_err;
  const double err = s[0] / s[28];
  const float tf_old = reinterpret_cast<const float*>(&S.Tf)[e];
  double Tl = S.T[e], Pl = S.prevT[e];
  __syncwarp();
  if (lane < 16) reinterpret_cast<float*>(&S.evalTf)[e] = tf_old;
  if (kind == 1 && s[28] == 0) {  // no valid row: the object loop stops (:674-676)
    if (lane == 0) {
      S.prev_err = prev_err;
      S.done = 1;
      S.iters[level] += 1;
    }
    __syncwarp();
    return;
  }
  int done = 0, fallback = 0;
  double new_err = prev_err;
  if (err > prev_err) {
    Tl = Pl;
    done = 1;
  } else {
    new_err = err;
    double x[6];
    if (solve6_warp(s, lane, x)) fallback = 1;
    double nx = 0;
#pragma unroll
    for (int i = 0; i < 6; ++i) nx += x[i] * x[i];
    // sqrt(nx) < (double)1e-05f without the square root: the smallest double
    // whose root is not below is 0x1.b7cdfc28ae3ffp-34
    if (nx < 0x1.b7cdfc28ae3ffp-34 && sqrt(s[0] / s[28]) < 2e-3) {
      done = 1;
    } else {
      // se3_exp(x): element (i, j) of the update on lane 4 i + j
      const double w0 = x[3], w1 = x[4], w2 = x[5];
      const double th2 = w0 * w0 + w1 * w1 + w2 * w2;
      double A, B, C;
      if (th2 < 1e-10) {
        A = 1 - th2 / 6; B = 0.5 - th2 / 24; C = 1.0 / 6 - th2 / 120;
      } else {
        const double th = sqrt(th2);
        double sn, cs;
        sincos(th, &sn, &cs);
        A = sn / th; B = (1 - cs) / th2; C = (1 - A) / th2;
      }
      // every lane evaluates se3_exp's elements in its order (no divergence)
      // and keeps element (i, j)
      const int i = e >> 2, j = e & 3;
      const double W[3][3] = {{0, -w2, w1}, {w2, 0, -w0}, {-w1, w0, 0}};
      double El = (i == 3 && j == 3) ? 1.0 : 0.0;
#pragma unroll
      for (int ii = 0; ii < 3; ++ii) {
        double t = 0;
#pragma unroll
        for (int jj = 0; jj < 3; ++jj) {
          const double W2 = W[ii][0] * W[0][jj] + W[ii][1] * W[1][jj] + W[ii][2] * W[2][jj];
          const double I = ii == jj ? 1.0 : 0.0;
          const double v = I + A * W[ii][jj] + B * W2;
          if (ii == i && jj == j) El = v;
          t += (I + B * W[ii][jj] + C * W2) * x[jj];
        }
        if (ii == i && j == 3) El = t;
      }
      // R = E T (mul4d)
      double R = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        R += __shfl_sync(FULL_MASK, El, 4 * i + k) * __shfl_sync(FULL_MASK, Tl, 4 * k + j);
      Pl = Tl;
      Tl = R;
    }
  }
  if (lane < 16) {
    S.T[e] = Tl;
    S.prevT[e] = Pl;
    reinterpret_cast<float*>(&S.Tf)[e] = (float)Tl;
  }
  __syncwarp();
  const float itf = inverse_warp(reinterpret_cast<const float*>(&S.Tf), lane);
  if (lane < 16) reinterpret_cast<float*>(&S.invTf)[e] = itf;
  if (lane == 0) {
    S.prev_err = new_err;
    S.done = done;
    if (fallback) S.fallback = 1;
    S.iters[level] += 1;
  }
  __syncwarp();
}

// ------------------------------------------------------------------ residuals
struct GNArgs {
  PyrPtrs pyr;
  int cur;              // live set index
  int W, H;             // full-resolution model maps
  const F3* mvertex; const F3* mnormal; const int* mlabel;  // composite model maps
  F3* rV[MAX_PYR][MAX_INSTANCES];  // rendered reference vertex of each slot, by level
  GNState* st;
  double* partials;
  int max_tiles;
  const float2* zr;     // live depth range of each CTA tile, [level][tile]
  const float2* zs;     // and of each 32-pixel segment, [level][segment]
  int max_segs;
  F4 kL[MAX_PYR];       // intrinsics by level
  F4 k0;                // full resolution
  float inv_cov_rgb;
  int robust;
  int use_icp, use_rgb;
};

// The planes of one level.  Selected by comparing the level with constants:
// indexing the parameter arrays with it would copy them to local memory.
struct GNView {
  int w, h;
  const F3* V; const F3* Vref; const F3* N; const F3* COV;
  const float* I; const float* Iref; const float* GX; const float* GY;
  const uint8_t* MASK;
  F4 kL;
};
__device__ __forceinline__ GNView gn_view(const GNArgs& a, int L) {
  GNView v;
#pragma unroll
  for (int l = 0; l < MAX_PYR; ++l) {
    if (l != L) continue;
    v.w = a.pyr.w[l]; v.h = a.pyr.h[l];
    v.V = a.cur ? a.pyr.V[1][l] : a.pyr.V[0][l];
    v.Vref = a.cur ? a.pyr.V[0][l] : a.pyr.V[1][l];
    v.I = a.cur ? a.pyr.I[1][l] : a.pyr.I[0][l];
    v.Iref = a.cur ? a.pyr.I[0][l] : a.pyr.I[1][l];
    v.N = a.pyr.N[l]; v.COV = a.pyr.COV[l];
    v.GX = a.pyr.GX[l]; v.GY = a.pyr.GY[l];
    v.MASK = a.pyr.MASK[l];
    v.kL = a.kL[l];
  }
  return v;
}
__device__ __forceinline__ const F3* gn_ref_vertex(const GNArgs& a, int L, int s) {
  const F3* r = nullptr;
#pragma unroll
  for (int l = 0; l < MAX_PYR; ++l)
    if (l == L) r = a.rV[l][s];
  return r;
}

struct Row { int result; float e; float J[6]; };

// length(v) > 0.1f without the square root: the square root is monotone, so
// the test holds exactly when dot(v, v) exceeds the largest float whose square
// root is at most 0.1f (NaN fails both).
__device__ __forceinline__ bool longer_than_10cm(F3 v) { return dot(v, v) > 0x1.47ae16p-7f; }

// sqrtf((float)(1.0 / (double)sig)): a quotient of floats rounded to double and
// then to float equals the float quotient (53 >= 2 * 24 + 2 bits; Figueroa,
// "When is double rounding innocuous?", 1995).
__device__ __forceinline__ float inv_sigma(float sig) { return sqrtf(1.0f / sig); }

// rotate(camera_matrix(k), v): the products with the matrix's zeros only add
// +-0, or turn a coordinate that is out of the image anyway into NaN, which is
// out of the image too.
__device__ __forceinline__ F3 project(const F4& k, F3 v) {
  return mk3(k.x * v.x + k.z * v.z, k.y * v.y + k.w * v.z, v.z);
}
__device__ __forceinline__ bool in_image(float px, float py, int w, int h) {
  return !(px < 1 || px > (float)(unsigned)(w - 2) || py < 1 || py > (float)(unsigned)(h - 2) ||
           isnan(px) || isnan(py));
}

// The four taps and fractions of a bilinear lookup; without a lookup (`in`
// false) every tap is element 0.
struct Cell { int b, dx, dy; float fx, fy; };
__device__ __forceinline__ Cell cell_at(bool in, float px, float py, int w) {
  Cell c;
  const float fx0 = floorf(px), fy0 = floorf(py);
  c.b = in ? (int)fx0 + (int)fy0 * w : 0;
  c.dx = in ? 1 : 0;
  c.dy = in ? w : 0;
  c.fx = px - fx0;
  c.fy = py - fy0;
  return c;
}
__device__ __forceinline__ float bil4(float t00, float t10, float t01, float t11, float fx,
                                      float fy) {
  return t00 * (1.f - fx) * (1.f - fy) + t10 * (1.f - fy) * fx + t01 * (1.f - fx) * fy +
         t11 * fx * fy;
}
__device__ __forceinline__ float bil(const float* img, int w, float px, float py) {
  const Cell c = cell_at(true, px, py, w);
  return bil4(img[c.b], img[c.b + 1], img[c.b + w], img[c.b + w + 1], c.fx, c.fy);
}

// The rows of one pixel.  Both rows are written as one straight line: the
// loads that do not depend on the pose, both projections, every gather (at a
// harmless address where a test failed), then both rows.  A pixel then waits
// for memory twice, and the two rows' arithmetic overlaps; as two functions
// with early returns a pixel's chain was 6.7 k cycles long and a level-0
// evaluation at 640x480 12.6 us; now 3.6 k, and 12.0 us (1280x720: 45 against
// 46, 160x120: 5.7 against 10.4).
// A term that is off leaves result 0.

// The photometric row once its taps are there: trackRGB (tracking.cpp:
// 1023-1111, warp :1114-1121, rgb_jacobian :1123-1150) and
// track_obj_RGB_kernel (:491-578, obj_rgb_jacobian :1152-1178).
template <int KIND>
__device__ __forceinline__ void rgb_finish(const GNState& S, const F4& k, float ic, float residual,
                                           float gx, float gy, F3 wv, F3 live, Row& r) {
  // in a flat patch the numerator is 0
  F3 Jt = (1.f / live.z) * mk3(gx * k.x, gy * k.y,
                               div0(-(gx * live.x * k.x + gy * live.y * k.y), live.z));
  F3 Jr;
  if (KIND == 0) {
    Jt = -1.f * rotate(S.Tf, Jt);  // rotate(Jtrans, transpose(T_w_l))
    Jr = cross(wv, Jt);
  } else {
    Jr = cross(live, Jt);
  }
  r.J[0] = ic * Jt.x; r.J[1] = ic * Jt.y; r.J[2] = ic * Jt.z;
  r.J[3] = ic * Jr.x; r.J[4] = ic * Jr.y; r.J[5] = ic * Jr.z;
  r.e = ic * residual;
}

// track_ICP_Kernel (tracking.cpp:923-1020) and trackRGB.  The photometric
// outlier mask of the reference is all zero.
template <bool ICP, bool RGB>
__device__ __forceinline__ void camera_rows(const GNArgs& a, const GNView& lv, const GNState& S,
                                            const F3* rV, int p, Row& ri, Row& rr) {
  uint8_t mask;
  F3 n, vl, P, rv, rl;
  float i_ref;
  if (ICP) { mask = lv.MASK[p]; n = lv.N[p]; vl = lv.V[p]; P = lv.COV[p]; }
  if (RGB) { rv = rV[p]; rl = lv.Vref[p]; i_ref = lv.Iref[p]; }
  // projections
  F3 pv, wv, live;
  bool in_i, in_r;
  int q = 0;
  Cell c;
  if (ICP) {
    pv = xform(S.Tf, vl);
    const F3 pp = xform(S.view, pv);
    const float px = pp.x / pp.z, py = pp.y / pp.z;
    in_i = in_image(px, py, a.W, a.H);
    ri.result = mask ? -6 : n.x == INVALIDF ? -1 : in_i ? 0 : -2;
    q = ri.result == 0 ? (int)px + (int)py * a.W : 0;
  }
  if (RGB) {
    wv = xform(S.T_w_r, rv);
    live = xform(S.invTf, wv);
    const F3 pr = project(lv.kL, live);
    const float px = pr.x / pr.z, py = pr.y / pr.z;
    in_r = in_image(px, py, lv.w, lv.h);
    rr.result = (rv.z <= 0.f || rv.z == INVALIDF) ? -1
                : (longer_than_10cm(rv - rl) && rl.z > 0.f) ? -3 : in_r ? 0 : -2;
    c = cell_at(rr.result == 0, px, py, lv.w);
  }
  // gathers
  F3 rn, rm;
  float t[12];
  if (ICP) { rn = a.mnormal[q]; rm = a.mvertex[q]; }
  if (RGB) {
    const int b1 = c.b + c.dx, b2 = c.b + c.dy, b3 = b2 + c.dx;
    t[0] = lv.I[c.b]; t[1] = lv.I[b1]; t[2] = lv.I[b2]; t[3] = lv.I[b3];
    t[4] = lv.GX[c.b]; t[5] = lv.GX[b1]; t[6] = lv.GX[b2]; t[7] = lv.GX[b3];
    t[8] = lv.GY[c.b]; t[9] = lv.GY[b1]; t[10] = lv.GY[b2]; t[11] = lv.GY[b3];
  }
  if (ICP) {
    const F3 diff = rm - pv;
    const F3 pn = rotate(S.Tf, n);
    if (ri.result == 0)
      ri.result = rn.x == INVALIDF ? -3 : longer_than_10cm(diff) ? -4 : dot(pn, rn) < 0.8f ? -5 : 1;
    // a row that is not used has sig = 1: a zero would take the general
    // quotient's slow path, and the warp with it
    const float sig = ri.result == 1 ? rn.x * rn.x * P.x + rn.y * rn.y * P.y + rn.z * rn.z * P.z
                                     : 1.f;
    const float ic = inv_sigma(sig);
    ri.e = ic * dot(rn, diff);
    const F3 j1 = ic * cross(pv, rn);
    ri.J[0] = ic * rn.x; ri.J[1] = ic * rn.y; ri.J[2] = ic * rn.z;
    ri.J[3] = j1.x; ri.J[4] = j1.y; ri.J[5] = j1.z;
  } else {
    ri.result = 0;
  }
  if (RGB) {
    const float residual = i_ref - bil4(t[0], t[1], t[2], t[3], c.fx, c.fy);
    const float gx = bil4(t[4], t[5], t[6], t[7], c.fx, c.fy);
    const float gy = bil4(t[8], t[9], t[10], t[11], c.fx, c.fy);
    rgb_finish<0>(S, lv.kL, a.inv_cov_rgb, residual, gx, gy, wv, live, rr);
    if (rr.result == 0) rr.result = 1;
  } else {
    rr.result = 0;
  }
}

// Object model maps derived from the composite maps and labels: the composite
// where label == object, (0, INVALID normal) elsewhere.
__device__ __forceinline__ void obj_maps(const GNArgs& a, int idx, bool in, int label, F3& v,
                                         F3& n) {
  // all three loaded before the label is looked at
  const int l = a.mlabel[idx];
  const F3 mv = a.mvertex[idx], mn = a.mnormal[idx];
  const bool mine = in && l == label;
  v = mk3(mine ? mv.x : 0.f, mine ? mv.y : 0.f, mine ? mv.z : 0.f);
  n = mk3(mine ? mn.x : INVALIDF, mine ? mn.y : 0.f, mine ? mn.z : 0.f);
}
__device__ __forceinline__ F3 bil4(F3 t0, F3 t1, F3 t2, F3 t3, float fx, float fy) {
  const float A = 1.f - fx, B = 1.f - fy;
  return mk3(t0.x * A * B + t1.x * B * fx + t2.x * A * fy + t3.x * fx * fy,
             t0.y * A * B + t1.y * B * fx + t2.y * A * fy + t3.y * fx * fy,
             t0.z * A * B + t1.z * B * fx + t2.z * A * fy + t3.z * fx * fy);
}

// track_Obj_ICP_Kernel (tracking.cpp:392-486, object outlier mask all zero) and
// track_obj_RGB_kernel.
template <bool ICP, bool RGB>
__device__ __forceinline__ void object_rows(const GNArgs& a, const GNView& lv, const GNState& S,
                                            const F3* rV, int L, int p, Row& ri, Row& rr) {
  F3 cn, cv, P, rv, rl;
  float i_ref;
  if (ICP) { cn = lv.N[p]; cv = lv.V[p]; P = lv.COV[p]; }
  if (RGB) { rv = rV[p]; rl = lv.Vref[p]; i_ref = lv.Iref[p]; }
  F3 o2v, live;
  Cell ci, c;
  bool cell_in = false;
  if (ICP) {
    o2v = xform(S.invTf, cv);
    const F3 c1v = xform(S.T_c1_o1, o2v);
    const F3 pr = project(a.k0, c1v);
    const float px = pr.x / pr.z, py = pr.y / pr.z;
    ri.result = cn.x == INVALIDF || (cv.x == 0 && cv.y == 0 && cv.z == 0) ? -1
                : in_image(px, py, a.W, a.H) ? 0 : -2;
    ci = cell_at(ri.result == 0, px, py, a.W);
    // a 2x2 cell outside the object's label box holds only other labels: its
    // taps are (0, INVALID normal) without reading the maps
    const int bx = (int)floorf(px), by = (int)floorf(py);
    cell_in = ri.result == 0 && !(bx + 1 < S.box[0] || bx > S.box[2] || by + 1 < S.box[1] ||
                                  by > S.box[3]);
    if (!cell_in) ci.b = ci.dx = ci.dy = 0;
  }
  if (RGB) {
    const F3 o1v = xform(S.inv_T_c1_o1, rv);
    live = xform(S.Tf, o1v);
    const F3 pr = project(lv.kL, live);
    const float px = pr.x / pr.z, py = pr.y / pr.z;
    // an object's rendered reference is valid only inside its label box,
    // halved per pyramid level (half-sampling never widens it)
    const int x = p % lv.w, y = p / lv.w;
    const bool boxed = !(x < (S.box[0] >> L) || x > (S.box[2] >> L) || y < (S.box[1] >> L) ||
                         y > (S.box[3] >> L));
    rr.result = !boxed || rv.z <= 0.f || rv.z == INVALIDF ? -1
                : (longer_than_10cm(rv - rl) && rl.z > 0.f) ? -3
                : in_image(px, py, lv.w, lv.h) ? 0 : -2;
    c = cell_at(rr.result == 0, px, py, lv.w);
  }
  F3 v0, v1, v2, v3, n0, n1, n2, n3;
  float t[12];
  if (ICP) {
    obj_maps(a, ci.b, cell_in, S.label, v0, n0);
    obj_maps(a, ci.b + ci.dx, cell_in, S.label, v1, n1);
    obj_maps(a, ci.b + ci.dy, cell_in, S.label, v2, n2);
    obj_maps(a, ci.b + ci.dx + ci.dy, cell_in, S.label, v3, n3);
  }
  if (RGB) {
    const int b1 = c.b + c.dx, b2 = c.b + c.dy, b3 = b2 + c.dx;
    t[0] = lv.I[c.b]; t[1] = lv.I[b1]; t[2] = lv.I[b2]; t[3] = lv.I[b3];
    t[4] = lv.GX[c.b]; t[5] = lv.GX[b1]; t[6] = lv.GX[b2]; t[7] = lv.GX[b3];
    t[8] = lv.GY[c.b]; t[9] = lv.GY[b1]; t[10] = lv.GY[b2]; t[11] = lv.GY[b3];
  }
  if (ICP) {
    const F3 wrv = bil4(v0, v1, v2, v3, ci.fx, ci.fy), wrn = bil4(n0, n1, n2, n3, ci.fx, ci.fy);
    const F3 o2n = rotate(S.invTf, cn);
    const F3 o1rv = xform(S.inv_T_w_o1, wrv);
    const F3 o1rn = rotate(S.inv_T_w_o1, wrn);
    const F3 diff = o2v - o1rv;
    const float residual = dot(o1rn, diff);
    if (ri.result == 0)
      ri.result = wrn.x == INVALIDF ? -3 : longer_than_10cm(diff) ? -4
                  : dot(o2n, o1rn) < 0.8f ? -5 : 1;
    const float sig = ri.result == 1
        ? o1rn.x * o1rn.x * P.x + o1rn.y * o1rn.y * P.y + o1rn.z * o1rn.z * P.z : 1.f;
    const float ic = inv_sigma(sig);
    ri.e = ic * residual;
    const F3 Jt = rotate(S.Tf, o1rn);
    const float c0 = -1.0f * ic * -1.0f;
    const F3 j1 = ic * cross(cv, Jt);
    ri.J[0] = c0 * Jt.x; ri.J[1] = c0 * Jt.y; ri.J[2] = c0 * Jt.z;
    ri.J[3] = j1.x; ri.J[4] = j1.y; ri.J[5] = j1.z;
  } else {
    ri.result = 0;
  }
  if (RGB) {
    const float residual = i_ref - bil4(t[0], t[1], t[2], t[3], c.fx, c.fy);
    const float gx = bil4(t[4], t[5], t[6], t[7], c.fx, c.fy);
    const float gy = bil4(t[8], t[9], t[10], t[11], c.fx, c.fy);
    rgb_finish<1>(S, lv.kL, a.inv_cov_rgb, residual, gx, gy, mk3(0.f), live, rr);
    if (rr.result == 0) rr.result = 1;
  } else {
    rr.result = 0;
  }
}

// Both rows of a pixel with the terms that the context uses (at least one).
template <int KIND>
__device__ __forceinline__ void gn_rows(const GNArgs& a, const GNView& lv, const GNState& S,
                                        const F3* rV, int L, int p, Row& ri, Row& rr) {
  if (a.use_icp && a.use_rgb) {
    if (KIND == 0) camera_rows<true, true>(a, lv, S, rV, p, ri, rr);
    else object_rows<true, true>(a, lv, S, rV, L, p, ri, rr);
  } else if (a.use_icp) {
    if (KIND == 0) camera_rows<true, false>(a, lv, S, rV, p, ri, rr);
    else object_rows<true, false>(a, lv, S, rV, L, p, ri, rr);
  } else {
    if (KIND == 0) camera_rows<false, true>(a, lv, S, rV, p, ri, rr);
    else object_rows<false, true>(a, lv, S, rV, L, p, ri, rr);
  }
}

// Index of J_i J_j (i <= j) among the 21 upper-triangle terms, row-major
// (reduce, tracking.cpp:1279-1311).
__host__ __device__ constexpr int jtj_index(int i, int j) { return 7 + i * 6 - i * (i - 1) / 2 + (j - i); }

__device__ __forceinline__ void accumulate(float* acc, int* cnt, const Row& r, int kind) {
  if (r.result < 1) {
    cnt[0] += r.result == -4;
    cnt[1] += r.result == -5;
    cnt[2] += r.result > -4;
    return;
  }
  float w, loss;
  robust(r.e, kind, w, loss);
  acc[0] += loss;
  const float we = w * r.e;
#pragma unroll
  for (int i = 0; i < 6; ++i) acc[1 + i] += we * r.J[i];
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    const float wj = w * r.J[i];
#pragma unroll
    for (int j = i; j < 6; ++j) acc[jtj_index(i, j)] += wj * r.J[j];
  }
  acc[28] += 1.f;
}

// Range of live depths over the pixels of each GN tile and of each 32-pixel
// segment (a warp's pixels of one step through its tile) whose ICP row gets
// past the validity checks (valid normal, nonzero vertex), by level.
__global__ void __launch_bounds__(GN_THREADS)
tile_depth_range_kernel(PyrPtrs pyr, int cur, float2* __restrict__ zr, int max_tiles,
                        float2* __restrict__ zs, int max_segs) {
  const int L = blockIdx.y;
  const int w = pyr.w[L], n = w * pyr.h[L];
  const int ppt = gn_pix(L);
  const int p0 = blockIdx.x * GN_THREADS * ppt;
  if (p0 >= n) return;
  float lo = INFINITY, hi = -INFINITY;
  for (int k = 0; k < ppt; ++k) {
    const int p = p0 + k * GN_THREADS + threadIdx.x;
    float l = INFINITY, h = -INFINITY;
    if (p < n && pyr.N[L][p].x != INVALIDF) {
      const F3 v = pyr.V[cur][L][p];
      if (!(v.x == 0 && v.y == 0 && v.z == 0)) { l = fminf(l, v.z); h = fmaxf(h, v.z); }
    }
    for (int o = 16; o > 0; o >>= 1) {
      l = fminf(l, __shfl_xor_sync(0xffffffffu, l, o));
      h = fmaxf(h, __shfl_xor_sync(0xffffffffu, h, o));
    }
    if ((threadIdx.x & 31) == 0 && p < n) zs[(size_t)L * max_segs + (p >> 5)] = make_float2(l, h);
    lo = fminf(lo, l);
    hi = fmaxf(hi, h);
  }
  __shared__ float2 sw[GN_THREADS / 32];
  if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = make_float2(lo, hi);
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < GN_THREADS / 32; ++i) { lo = fminf(lo, sw[i].x); hi = fmaxf(hi, sw[i].y); }
    zr[L * max_tiles + blockIdx.x] = make_float2(lo, hi);
  }
}

// Can any pixel of tile `tile` at level L give an object problem a valid row?
// A `false` answer is exact for the 29 normal-equation sums (the tile's pixels
// all end in a negative result code); only the diagnostic outlier counts
// (sums 29-31, which the reference computes and never reads) then leave the
// tile out.
//  - photometric rows need the object's rendered reference: inside its label
//    box, halved per level;
//  - an ICP row needs a model tap with the object's label, i.e. a projection
//    into the label box: the tile's live points lie in the frustum spanned by
//    its pixel rectangle and depth range, whose projection lies in the hull
//    of its 8 projected corners (2 px of slack for rounding);
//  - or, with no such tap, the blended model vertex is 0, the world origin:
//    rows then need a live point within 0.1 m of it (in object coordinates).
// Called by a whole warp: lane l projects frustum corner l & 7 and the warp
// combines the corners with shuffles (every lane gets the answer).  A corner
// behind camera 1 or a NaN projection makes the answer true, as the first such
// corner did in a sequential loop; otherwise no NaN reaches the minima and
// maxima, so their order does not matter.
__device__ bool object_tile_live(const GNArgs& a, const F4& kL, const GNState& S, int L,
                                 int tile, int w, int n) {
  const int ppt = gn_pix(L);
  const int p0 = tile * GN_THREADS * ppt, p1 = min(n, p0 + GN_THREADS * ppt);
  const int ya = p0 / w, yb = (p1 - 1) / w;
  const int xa = ya == yb ? p0 % w : 0, xb = ya == yb ? (p1 - 1) % w : w - 1;
  const bool has_box = S.box[2] >= S.box[0];
  if (a.use_rgb && has_box &&
      !(xb < (S.box[0] >> L) || xa > (S.box[2] >> L) || yb < (S.box[1] >> L) ||
        ya > (S.box[3] >> L)))
    return true;
  if (!a.use_icp) return false;
  const float2 zr = a.zr[L * a.max_tiles + tile];
  if (!(zr.x <= zr.y)) return false;  // no pixel of the tile reaches the projection
  const M4 iK = inverse_camera_matrix(kL), K0 = camera_matrix(a.k0);
  const int c = threadIdx.x & 7;
  const float x = (float)((c & 1) ? xb : xa), y = (float)((c & 2) ? yb : ya);
  const float z = (c & 4) ? zr.y : zr.x;
  const F3 o2v = xform(S.invTf, z * rotate(iK, mk3(x, y, 1.f)));
  F3 lo = o2v, hi = o2v;
  const F3 c1v = xform(S.T_c1_o1, o2v);
  bool unbounded = !(c1v.z > 0.f);  // the frustum reaches behind camera 1: no bound
  float qx0 = 0.f, qy0 = 0.f;
  if (!unbounded) {
    const F3 pr = rotate(K0, c1v);
    qx0 = pr.x / pr.z;
    qy0 = pr.y / pr.z;
    unbounded = isnan(qx0) || isnan(qy0);
  }
  if (__any_sync(0xffffffffu, unbounded)) return true;
  float qx1 = qx0, qy1 = qy0;
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    qx0 = fminf(qx0, __shfl_xor_sync(0xffffffffu, qx0, o));
    qx1 = fmaxf(qx1, __shfl_xor_sync(0xffffffffu, qx1, o));
    qy0 = fminf(qy0, __shfl_xor_sync(0xffffffffu, qy0, o));
    qy1 = fmaxf(qy1, __shfl_xor_sync(0xffffffffu, qy1, o));
    lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, o));
    lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, o));
    lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, o));
    hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, o));
    hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, o));
    hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, o));
  }
  if (has_box && floorf(qx1) + 3.f >= (float)S.box[0] && floorf(qx0) - 2.f <= (float)S.box[2] &&
      floorf(qy1) + 3.f >= (float)S.box[1] && floorf(qy0) - 2.f <= (float)S.box[3])
    return true;
  const F3 o = get_translation(S.inv_T_w_o1);
  const float dx = fmaxf(fmaxf(lo.x - o.x, o.x - hi.x), 0.f);
  const float dy = fmaxf(fmaxf(lo.y - o.y, o.y - hi.y), 0.f);
  const float dz = fmaxf(fmaxf(lo.z - o.z, o.z - hi.z), 0.f);
  return dx * dx + dy * dy + dz * dz <= 0.101f * 0.101f;
}

// The warp's sum of value `lane` (29 sums, then the 3 counts) in FP64: every
// lane stores its FP32 partials in shared memory (rows padded to 33 words, so
// the column reads hit 32 banks) and lane i adds column i over the 32 lanes in
// lane order.  A shuffle tree would take 10 shuffles per double and 320 per
// warp; with one problem per grid row and many problems per launch that tree
// dominated the launch.
__device__ __forceinline__ double warp_sum_fp64(const float* acc, const int* cnt,
                                                float (*red)[33], int lane) {
#pragma unroll
  for (int i = 0; i < 29; ++i) red[lane][i] = acc[i];
#pragma unroll
  for (int i = 0; i < 3; ++i) red[lane][29 + i] = (float)cnt[i];  // small, exact
  __syncwarp();
  double v = 0;
#pragma unroll 8
  for (int j = 0; j < 32; ++j) v += (double)red[j][lane];
  return v;
}

// The FP64 sums of one tile (CTA) of a problem at level L: every thread
// evaluates the ICP and photometric rows of its pixels, weights them and
// accumulates in FP32 (at most 6 rows per thread); the sums are FP64 from the
// warp level up, in a fixed order.  Thread i < 32 returns sum i (29 sums, then
// the 3 counts).  Object problems skip a tile that cannot hold a valid row.
template <int KIND>
__device__ __forceinline__ double gn_tile_sums(const GNArgs& a, const GNState& S, int s, int L,
                                               int tile, double (*sh)[32],
                                               float (*red)[32][33]) {
  const GNView lv = gn_view(a, L);
  const int w = lv.w, n = w * lv.h;
  bool live = true;
  if (KIND == 1) {
    __shared__ int s_live;
    if (threadIdx.x < 32) {
      const bool tl = object_tile_live(a, lv.kL, S, L, tile, w, n);
      if (threadIdx.x == 0) s_live = tl ? 1 : 0;
    }
    __syncthreads();
    live = s_live != 0;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (live) {
    float acc[29];
#pragma unroll
    for (int i = 0; i < 29; ++i) acc[i] = 0.f;
    int cnt[3] = {0, 0, 0};
    const F3* rV = gn_ref_vertex(a, L, s);
    const int ppt = gn_pix(L);
#pragma unroll 1
    for (int k = 0; k < ppt; ++k) {
      const int p = tile * (GN_THREADS * ppt) + k * GN_THREADS + threadIdx.x;
      if (p >= n) break;
      Row ri, rr;
      gn_rows<KIND>(a, lv, S, rV, L, p, ri, rr);
      if (a.use_icp) accumulate(acc, cnt, ri, a.robust);
      if (a.use_rgb) accumulate(acc, cnt, rr, a.robust);
    }
    sh[warp][lane] = warp_sum_fp64(acc, cnt, red[warp], lane);
  } else {
    sh[warp][lane] = 0.0;
  }
  __syncthreads();
  double v = 0;
  if (threadIdx.x < 32) {
#pragma unroll
    for (int wi = 0; wi < GN_THREADS / 32; ++wi) v += sh[wi][threadIdx.x];
  }
  return v;
}

// The 32 sums of a problem over its `ntiles` tile partials, in a fixed order,
// by the whole CTA (the last CTA of the problem): tot[i] = sum i.  The loads
// of 16 tiles are issued before their in-order additions, so the tail waits on
// about ntiles / 128 L2 round trips instead of ntiles / 64.
__device__ __forceinline__ void gn_tail_sums(const GNArgs& a, int ntiles,
                                             double (*sh)[32], double* tot) {
  constexpr int G = GN_THREADS / 32, U = 16;
  {
    const int i = threadIdx.x & 31, g = threadIdx.x >> 5;  // 8 groups of tiles
    const double* col = a.partials + i;
    double v = 0;
    int b = g;
    for (; b + (U - 1) * G < ntiles; b += U * G) {
      double t[U];
#pragma unroll
      for (int u = 0; u < U; ++u) t[u] = __ldcg(col + (size_t)(b + u * G) * 32);
#pragma unroll
      for (int u = 0; u < U; ++u) v += t[u];
    }
    for (; b < ntiles; b += G) v += __ldcg(col + (size_t)b * 32);
    sh[g][i] = v;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = 0;
#pragma unroll
    for (int g = 0; g < G; ++g) v += sh[g][threadIdx.x];
    tot[threadIdx.x] = v;
  }
  __syncthreads();
}

// One evaluation of the normal equations of the problem in slot s: the rows of
// every tile, the tile partials, and in the CTA that finishes last (ticket
// counter) the sum over the tiles.
template <int KIND>
__global__ void __launch_bounds__(GN_THREADS, MF_GN_MINB)
gn_eval_kernel(GNArgs a, int s, int L) {
  GNState& S = a.st[s];
  __shared__ double sh[GN_THREADS / 32][32];
  __shared__ float red[GN_THREADS / 32][32][33];
  const double v = gn_tile_sums<KIND>(a, S, s, L, blockIdx.x, sh, red);
  __shared__ bool last;
  if (threadIdx.x < 32) {
    a.partials[(size_t)blockIdx.x * 32 + threadIdx.x] = v;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int t = atomicAdd(&S.ticket, 1);
    last = (t == (int)gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  __shared__ double tot[32];
  gn_tail_sums(a, (int)gridDim.x, sh, tot);
  if (threadIdx.x < 32) {
    S.sums[L][threadIdx.x] = tot[threadIdx.x];
    if (threadIdx.x == 0) S.ticket = 0;
  }
}

// ------------------------------------------------------------------ whole GN loops
// The coarse-to-fine GN of a stage in one launch.  The pixels of a level stay
// with the same CTA over all its iterations, so the rows' inputs stay in that
// SM's L1; an iteration is the rows of the CTA's tiles, one exchange of the
// CTAs' partial sums, and then every CTA adds the same partials in the same
// order and runs the same step on its own copy of the problem in shared
// memory.  No CTA waits for another one's step, no state travels between
// them, and a problem that stopped ends its level at once.
//
// Sums: FP32 per thread over the rows of its 1 (level > 0) or 3 pixels of a
// tile, FP64 from there on in a fixed order: the warp's lanes, each warp's
// tiles (row, row + R, ...: "row" is a virtual CTA, R a constant), the 16
// warps of the row, the rows.  The order does not depend on the grid or on
// the device, and the plain mode evaluates through the same kernels, so poses
// are the same bit for bit in every mode.
// Tiles in flight per CTA: two teams of 8 warps at 128 registers each.  Three
// at 80 registers spill, and a pixel's chain then takes 5.2 k instead of 3.6 k
// cycles: 160x120 29.2 k against 23.5 k cycles per level-0 iteration, 640x480
// 37.4 k against 36.4 k; only 1280x720, with eight tiles per SM, gains 2 % by
// the third.
constexpr int GN_TEAMS = 2;
constexpr int GN_BLOCK = GN_TEAMS * GN_THREADS;
constexpr int GN_WARPS = GN_BLOCK / 32;
constexpr int GN_CAM_ROWS = 148;                     // one virtual CTA per SM

struct GNShared {
  GNState S;
  GNView lv;         // the level being evaluated
  double sh[GN_WARPS][32];
  double tot[32];
  int flag;
  float red[GN_WARPS][32][17];   // a warp's transposition: 16 values of 32 lanes at a time
};

struct GNLoop {
  int levels;
  int iters[MAX_PYR];
  int only;          // >= 0: one evaluation of this level without a step (sums only)
  double* rows;      // partial sums, alternating by iteration: camera 2 x GN_CAM_ROWS x 32,
                     // objects 2 x slots x max_tiles x 32
  uint8_t* lives;    // objects: the tiles with a sum, 2 x slots x max_tiles
  unsigned* bar;     // barrier arrivals by problem slot
  int slots;         // problem slots (the context's instance capacity)
  unsigned polls;    // of a wait before it gives up
  int* status;
  int* timeout;      // Context::gn_timeout
  float* poses;      // camera: T_w_c; objects: the volume poses
};

// The warp's FP64 sum of value `lane` (29 sums, then the 3 counts).  The lanes'
// FP32 values are transposed through shared memory 16 at a time; the two
// halves of the warp add 16 lanes' values each, in two chains.
__device__ __forceinline__ double gn_warp_sum(const float* acc, const int* cnt, float (*red)[17],
                                              int lane) {
  const int col = lane & 15, half = lane >> 4;
  double out = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      red[lane][i] = 16 * h + i < 29 ? acc[16 * h + i < 29 ? 16 * h + i : 0]
                                     : (float)cnt[16 * h + i < 29 ? 0 : 16 * h + i - 29];  // exact
    __syncwarp();
    double v0 = 0, v1 = 0;
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
      v0 += (double)red[16 * half + j][col];
      v1 += (double)red[16 * half + j + 1][col];
    }
    double v = v0 + v1;
    v += __shfl_xor_sync(FULL_MASK, v, 16);
    if (half == h) out = v;
    __syncwarp();
  }
  return out;
}

// The sum over the CTA's 16 warps of sh[warp][lane], by one warp, in four chains.
__device__ __forceinline__ double gn_sum_warps(const double (*sh)[32], int lane) {
  double c[4] = {0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < GN_WARPS; k += 4)
#pragma unroll
    for (int q = 0; q < 4; ++q) c[q] += sh[k + q][lane];
  return (c[0] + c[1]) + (c[2] + c[3]);
}

// The 32 sums of a row (its tiles row, row + nrows, ...) of level L, by the
// whole CTA: team j of 8 warps takes every second of them.  Returned by lane i
// of warp 0.  Every thread reaches the barrier inside.
template <int KIND>
__device__ __forceinline__ double gn_row_sums(const GNArgs& a, GNShared& sm, int s, int L,
                                              int row, int nrows) {
  const GNView& lv = sm.lv;
  const int n = lv.w * lv.h, ppt = gn_pix(L);
  const int ntiles = (n + GN_THREADS * ppt - 1) / (GN_THREADS * ppt);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int team = warp / (GN_THREADS / 32), wi = warp % (GN_THREADS / 32);
  const GNState& S = sm.S;
  const F3* rV = gn_ref_vertex(a, L, s);
  double v = 0;
#pragma unroll 1
  for (int t = row + nrows * team; t < ntiles; t += GN_TEAMS * nrows) {
    float acc[29];
#pragma unroll
    for (int i = 0; i < 29; ++i) acc[i] = 0.f;
    int cnt[3] = {0, 0, 0};
#pragma unroll 1
    for (int k = 0; k < ppt; ++k) {
      const int p = (t * ppt + k) * GN_THREADS + wi * 32 + lane;
      if (p >= n) break;
      Row ri, rr;
      gn_rows<KIND>(a, lv, S, rV, L, p, ri, rr);
      if (a.use_icp) accumulate(acc, cnt, ri, a.robust);
      if (a.use_rgb) accumulate(acc, cnt, rr, a.robust);
    }
    v += gn_warp_sum(acc, cnt, sm.red[warp], lane);
  }
  sm.sh[warp][lane] = v;
  __syncthreads();
  return warp == 0 ? gn_sum_warps(sm.sh, lane) : 0.0;
}

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Waits until `target` CTAs have arrived at `bar`.  Bounded: after `polls` polls
// (32 ns apart after the first 64: about 1 s) it sets MF_STATUS_GN_TIMEOUT and
// the host's word, which calls that read poses look at, and returns 1; the CTA
// returns then.
__device__ __forceinline__ int gn_wait(const unsigned* bar, unsigned target, const GNLoop& g) {
  for (unsigned spins = 0; ld_acquire_u32(bar) < target; ++spins) {
    if (spins >= g.polls) {
      atomicOr(g.status, MF_STATUS_GN_TIMEOUT);
      *(volatile int*)g.timeout = 1;
      return 1;
    }
    if (spins > 64) __nanosleep(32);
  }
  return 0;
}

__device__ __forceinline__ void gn_copy_state(const GNState* from, GNState* to) {
  static_assert(sizeof(GNState) % 4 == 0, "GNState is copied as words");
  const int* src = reinterpret_cast<const int*>(from);
  int* dst = reinterpret_cast<int*>(to);
  for (int i = threadIdx.x; i < (int)(sizeof(GNState) / 4); i += blockDim.x) dst[i] = src[i];
}

// The camera's GN (trackLiveFrame :240-335): a cooperative launch of one CTA
// per SM (fewer for small frames).  The partial rows are exchanged through L2
// with one grid barrier per iteration.
// What bounds it at 640x480: the evaluation of the rows (instruction issue,
// the FP64 of the weights included), then the serial tail of an iteration
// (barrier, row sums, step).  One launch per iteration, chained by
// programmatic dependent launch, with the step in the CTA that finished last,
// took 342 us for a frame's iterations at 640x480 (ncu, their sum); this launch
// takes 175 (160x120: 19 iterations of 11 us in launches, now 89 in all).
__global__ void __launch_bounds__(GN_BLOCK, 1)
gn_camera_kernel(GNArgs a, GNLoop g) {
  extern __shared__ __align__(16) unsigned char gn_smem[];
  GNShared& sm = *reinterpret_cast<GNShared*>(gn_smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  gn_copy_state(a.st, &sm.S);
  __syncthreads();
  unsigned target = 0;
  int par = 0;
  for (int L = g.only >= 0 ? g.only : g.levels - 1; L >= (g.only >= 0 ? g.only : 0); --L) {
    if (threadIdx.x == 0) sm.lv = gn_view(a, L);
    __syncthreads();
    const int n = sm.lv.w * sm.lv.h, tp = GN_THREADS * gn_pix(L);
    const int nrows = min((n + tp - 1) / tp, GN_CAM_ROWS);
    int iters = 1;
    if (g.only < 0) {
#pragma unroll
      for (int l = 0; l < MAX_PYR; ++l)
        if (l == L) iters = g.iters[l];
    }
    for (int it = 0; it < iters; ++it) {
      double* rows = g.rows + (size_t)par * GN_CAM_ROWS * 32;
      for (int row = blockIdx.x; row < nrows; row += gridDim.x) {
        const double v = gn_row_sums<0>(a, sm, 0, L, row, nrows);
        if (warp == 0) __stcg(rows + row * 32 + lane, v);
        if (row + (int)gridDim.x < nrows) __syncthreads();  // sh is written again
      }
      if (warp == 0) {
        __threadfence();
        __syncwarp();
        if (lane == 0) {
          atomicAdd(g.bar, 1u);
          target += gridDim.x;
          sm.flag = gn_wait(g.bar, target, g);
        }
      }
      __syncthreads();
      if (sm.flag) return;
      // every load in flight before the first addition
      constexpr int U = (GN_CAM_ROWS + GN_WARPS - 1) / GN_WARPS;
      double part[U], v = 0;
#pragma unroll
      for (int u = 0; u < U; ++u)
        part[u] = warp + u * GN_WARPS < nrows ? __ldcg(rows + (warp + u * GN_WARPS) * 32 + lane)
                                              : 0.0;
#pragma unroll
      for (int u = 0; u < U; ++u) v += part[u];
      sm.sh[warp][lane] = v;
      __syncthreads();
      if (warp == 0) {
        const double t = gn_sum_warps(sm.sh, lane);
        sm.tot[lane] = t;
        sm.S.sums[L][lane] = t;
        __syncwarp();
        if (g.only < 0) gn_step_warp(&sm.S, sm.tot, L, it == 0);
      }
      __syncthreads();
      par ^= 1;
      if (sm.S.done && g.only < 0) break;
    }
  }
  if (blockIdx.x != 0) return;
  gn_copy_state(&sm.S, a.st);
  if (g.only < 0 && threadIdx.x < 16) g.poses[threadIdx.x] = (float)sm.S.T[threadIdx.x];
}

// ------------------------------------------------------------------ objects
// The objects' GN (trackEachObject :629-694): one cooperative launch whose
// CTAs are shared out among the objects, one or more each in proportion to
// the objects' label boxes.  The CTAs of an object run its whole loop and
// wait for each other only (one barrier per object and iteration), so a small
// object never waits for a large one.
//
// An object covers a few percent of the frame.  Each iteration first lists
// the CTA's tasks -- (tile, warp of the tile) pairs with a 32-pixel segment
// that can hold a valid row (object_segment_live) -- one thread per pair, and
// the warps then take the listed tasks in turn.  A tile is 768 consecutive
// pixels, more than one image row of a 640-pixel frame: with whole tiles as
// the unit, six of seven evaluated pixels lay beside the object.
//
// The object problems can be so poorly conditioned that the last bit of a sum
// shows in the pose, so the order of the FP64 sums is fixed whatever the
// number of CTAs: the lanes of a warp in order, the 8 warps of a tile, the
// tiles g, g + 8, ... of column g in order, the 8 columns.  Warps and tiles
// without a live segment would add exact zeros and are left out.
//
// Measured on one B200 (ncu, a frame's launches of 19 iterations against this
// one): three objects at 640x480 383 -> 226 us, six at 1280x720 869 -> 308,
// twelve of uneven size at 640x480 1178 -> 522.
constexpr int GO_WARPS = 16, GO_BLOCK = 32 * GO_WARPS;
constexpr int GO_CHUNK = 32;               // tiles listed at a time
constexpr int GO_TASKS = 8 * GO_CHUNK;

struct GOShared {
  GNState S;
  GNView lv;
  double sh[8][32];              // the columns' sums
  double tot[32];
  double ws[GO_TASKS][32];       // warp sums of the listed tasks
  float red[GO_WARPS][32][33];
  int list[GO_TASKS];            // task | live segments << 16
  int live[GO_TASKS];            // task -> its live segments
  short slot[GO_TASKS];          // task -> its place in the list, or -1
  int pick[GO_WARPS][32];        // the live ones of 32 tiles of a column
  int ntask, flag;
  int obj, rank, size;           // this CTA's place: list position, rank among its CTAs, their number
  M4 M;                          // T_c1_o1 inverse(T): live camera -> reference camera, its x
                                 // and y rows taken through the intrinsics
  float ifx, ify;                // 1 / focal lengths of the level
  F3 origin;                     // the world origin's image in the live camera
};

// object_tile_live for one 32-pixel segment, by one thread.  The bounds only
// have to hold up to its slack (2 pixels, 1 mm), so the frustum's corners are
// taken through one product matrix (its rows scaled by the intrinsics), the
// quotients are approximate ones, and the distance to the world origin is
// taken in the live camera's frame.
__device__ __forceinline__ bool object_segment_live(const GNArgs& a, const GOShared& sm, int L,
                                                    int p0, int n) {
  const GNState& S = sm.S;
  const int w = sm.lv.w, p1 = min(n, p0 + 32) - 1;
  const int ya = p0 / w, xe = p0 - ya * w + (p1 - p0);   // xe: the last pixel's x in row ya
  const bool one_row = xe < w;
  const int yb = one_row ? ya : p1 / w;
  const int xa = one_row ? p0 - ya * w : 0, xb = one_row ? xe : w - 1;
  const bool has_box = S.box[2] >= S.box[0];
  if (a.use_rgb && has_box &&
      !(xb < (S.box[0] >> L) || xa > (S.box[2] >> L) || yb < (S.box[1] >> L) ||
        ya > (S.box[3] >> L)))
    return true;
  if (!a.use_icp) return false;
  const float2 zr = a.zs[(size_t)L * a.max_segs + (p0 >> 5)];
  if (!(zr.x <= zr.y)) return false;  // no pixel of the segment reaches the projection
  float qx0 = INFINITY, qx1 = -INFINITY, qy0 = INFINITY, qy1 = -INFINITY;
  bool unbounded = false;   // behind camera 1, or NaN
  const float xs[2] = {((float)xa - sm.lv.kL.z) * sm.ifx, ((float)xb - sm.lv.kL.z) * sm.ifx};
  const float ys[2] = {((float)ya - sm.lv.kL.w) * sm.ify, ((float)yb - sm.lv.kL.w) * sm.ify};
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    if (c >= 2 && one_row) continue;   // one image row: its two ends
    const float dx = xs[c & 1], dy = ys[c >> 1];
    const F3 D = rotate(sm.M, mk3(dx, dy, 1.f));
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float z = e ? zr.y : zr.x;
      const F3 q = z * D + get_translation(sm.M);
      const float px = __fdividef(q.x, q.z), py = __fdividef(q.y, q.z);
      unbounded |= !(q.z > 0.f) || isnan(px) || isnan(py);
      qx0 = fminf(qx0, px); qx1 = fmaxf(qx1, px);
      qy0 = fminf(qy0, py); qy1 = fmaxf(qy1, py);
    }
  }
  if (unbounded) return true;
  if (has_box && floorf(qx1) + 3.f >= (float)S.box[0] && floorf(qx0) - 2.f <= (float)S.box[2] &&
      floorf(qy1) + 3.f >= (float)S.box[1] && floorf(qy0) - 2.f <= (float)S.box[3])
    return true;
  // the frustum's box in the live camera: x and y reach z times the directions
  // (which run from right to left, or from below, for a negative focal length)
  const float xlo = fminf(xs[0], xs[1]), xhi = fmaxf(xs[0], xs[1]);
  const float x0 = fminf(zr.x * xlo, zr.y * xlo), x1 = fmaxf(zr.x * xhi, zr.y * xhi);
  const float ylo = fminf(ys[0], ys[1]), yhi = fmaxf(ys[0], ys[1]);
  const float y0 = fminf(zr.x * ylo, zr.y * ylo), y1 = fmaxf(zr.x * yhi, zr.y * yhi);
  const float ox = fmaxf(fmaxf(x0 - sm.origin.x, sm.origin.x - x1), 0.f);
  const float oy = fmaxf(fmaxf(y0 - sm.origin.y, sm.origin.y - y1), 0.f);
  const float oz = fmaxf(fmaxf(zr.x - sm.origin.z, sm.origin.z - zr.y), 0.f);
  // a NaN origin bounds nothing
  return !(ox * ox + oy * oy + oz * oz > 0.101f * 0.101f);
}

// The share of CTA `b` of `nb`: every object one CTA, the others in proportion
// to the 32-pixel segments that their label boxes meet (in pixels).  With
// fewer CTAs than objects CTA b takes objects b, b + nb, ...
__device__ void gn_share(const GNState* __restrict__ st, const IdList& slots, int b, int nb,
                         GOShared& sm) {
  long long area[MAX_INSTANCES], total = 0;
  for (int i = 0; i < slots.n; ++i) {
    const GNState& S = st[slots.v[i]];
    const long long w = S.box[2] - S.box[0] + 1, h = S.box[3] - S.box[1] + 1;
    area[i] = (S.box[2] >= S.box[0] ? (w + 48) * h : 0) + GN_THREADS * GN_PIX_MAX;
    total += area[i];
  }
  const int spare = nb - slots.n;
  sm.obj = b;
  sm.rank = 0;
  sm.size = 1;
  if (spare <= 0) return;
  long long sum = 0;
  int first = 0;
  for (int i = 0; i < slots.n; ++i) {
    // the cumulative share rounded down, so that the shares add up to nb
    sum += area[i];
    const int next = (int)(spare * sum / total) + i + 1;
    if (b < next) {
      sm.obj = i;
      sm.rank = b - first;
      sm.size = next - first;
      return;
    }
    first = next;
  }
}

__global__ void __launch_bounds__(GO_BLOCK, 1)
gn_objects_kernel(GNArgs a, GNLoop g, IdList slots, const float* __restrict__ Twc2) {
  extern __shared__ __align__(16) unsigned char gn_smem[];
  GOShared& sm = *reinterpret_cast<GOShared*>(gn_smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) gn_share(a.st, slots, blockIdx.x, gridDim.x, sm);
  __syncthreads();
  const int rank = sm.rank, size = sm.size;
  GNState& S = sm.S;
  for (int obj = sm.obj; obj < slots.n; obj += size == 1 ? (int)gridDim.x : slots.n) {
    const int s = slots.v[obj];
    __syncthreads();
    gn_copy_state(a.st + s, &S);
    __syncthreads();
    if (g.only < 0 && warp == 0) {
      // setup_object_post: the start pose inverse(T_w_c2) T_w_o1
      float* c2 = reinterpret_cast<float*>(&S.T_w_c2);
      float* tmp = reinterpret_cast<float*>(&sm.M);
      if (lane < 16) c2[lane] = Twc2[lane];
      __syncwarp();
      const float ie = inverse_warp(c2, lane);
      if (lane < 16) tmp[lane] = ie;
      __syncwarp();
      const float t0 = mul_warp(tmp, reinterpret_cast<const float*>(&S.T_w_o1), lane);
      float* Tf = reinterpret_cast<float*>(&S.Tf);
      if (lane < 16) {
        Tf[lane] = t0;
        reinterpret_cast<float*>(&S.evalTf)[lane] = t0;
        S.T[lane] = S.prevT[lane] = (double)t0;
      }
      __syncwarp();
      const float it0 = inverse_warp(Tf, lane);
      if (lane < 16) reinterpret_cast<float*>(&S.invTf)[lane] = it0;
    }
    unsigned* bar = g.bar + s;
    unsigned target = 0;
    int par = 0;
    for (int L = g.only >= 0 ? g.only : g.levels - 1; L >= (g.only >= 0 ? g.only : 0); --L) {
      if (threadIdx.x == 0) sm.lv = gn_view(a, L);
      __syncthreads();
      const GNView& lv = sm.lv;
      const int n = lv.w * lv.h, ppt = gn_pix(L);
      const int ntiles = (n + GN_THREADS * ppt - 1) / (GN_THREADS * ppt);
      const int U = (ntiles - rank + size - 1) / size;   // this CTA's tiles: rank, rank + size, ...
      const F3* rV = gn_ref_vertex(a, L, s);
      int iters = 1;
      if (g.only < 0) {
#pragma unroll
        for (int l = 0; l < MAX_PYR; ++l)
          if (l == L) iters = g.iters[l];
      }
      for (int it = 0; it < iters; ++it) {
        if (warp == 0) {
          const float m = mul_warp(reinterpret_cast<const float*>(&S.T_c1_o1),
                                   reinterpret_cast<const float*>(&S.invTf), lane);
          // row i < 2: f_i times itself plus c_i times row 2
          const float m2 = __shfl_sync(FULL_MASK, m, 8 + (lane & 3));
          const int i = (lane >> 2) & 3;
          const float mk = i == 0 ? a.k0.x * m + a.k0.z * m2
                           : i == 1 ? a.k0.y * m + a.k0.w * m2 : m;
          if (lane < 16) reinterpret_cast<float*>(&sm.M)[lane] = mk;
          if (lane == 0) {
            sm.origin = xform(S.Tf, get_translation(S.inv_T_w_o1));
            sm.ifx = 1.f / lv.kL.x;
            sm.ify = 1.f / lv.kL.y;
          }
        }
        // this iteration's tile sums and live flags (alternating, so that a
        // slow CTA still reads the last ones)
        const size_t base = ((size_t)par * g.slots + s) * a.max_tiles;
        double* rows = g.rows + base * 32;
        uint8_t* lives = g.lives + base;
        for (int u0 = 0; u0 < U; u0 += GO_CHUNK) {
          const int nt = min(GO_CHUNK, U - u0);
          if (threadIdx.x == 0) sm.ntask = 0;
          __syncthreads();
          if (threadIdx.x < nt * 8) sm.live[threadIdx.x] = 0;
          __syncthreads();
          for (int i = threadIdx.x; i < nt * 8 * ppt; i += GO_BLOCK) {
            // segment k of task i / ppt
            const int task = ppt == 1 ? i : i / GN_PIX_MAX, k = ppt == 1 ? 0 : i % GN_PIX_MAX;
            const int t = rank + size * (u0 + (task >> 3));
            const int p0 = (t * ppt + k) * GN_THREADS + (task & 7) * 32;
            if (p0 < n && object_segment_live(a, sm, L, p0, n)) atomicOr(&sm.live[task], 1 << k);
          }
          __syncthreads();
          if (threadIdx.x < nt * 8) {
            const int live = sm.live[threadIdx.x];
            int q = -1;
            if (live) {
              q = atomicAdd(&sm.ntask, 1);
              sm.list[q] = threadIdx.x | live << 16;
            }
            sm.slot[threadIdx.x] = (short)q;
          }
          __syncthreads();
          for (int q = warp; q < sm.ntask; q += GO_WARPS) {
            const int task = sm.list[q] & 0xffff, live = sm.list[q] >> 16;
            const int t = rank + size * (u0 + (task >> 3));
            float acc[29];
#pragma unroll
            for (int i = 0; i < 29; ++i) acc[i] = 0.f;
            int cnt[3] = {0, 0, 0};
#pragma unroll 1
            for (int k = 0; k < ppt; ++k) {
              const int p = (t * ppt + k) * GN_THREADS + (task & 7) * 32 + lane;
              if (!((live >> k) & 1) || p >= n) continue;
              Row ri, rr;
              gn_rows<1>(a, lv, S, rV, L, p, ri, rr);
              if (a.use_icp) accumulate(acc, cnt, ri, a.robust);
              if (a.use_rgb) accumulate(acc, cnt, rr, a.robust);
            }
            __syncwarp();
            sm.ws[q][lane] = warp_sum_fp64(acc, cnt, sm.red[warp], lane);
            __syncwarp();
          }
          __syncthreads();
          for (int u = warp; u < nt; u += GO_WARPS) {
            const int t = rank + size * (u0 + u);
            double sum = 0;
            int any = 0;
#pragma unroll
            for (int wi = 0; wi < 8; ++wi) {
              const int q = sm.slot[8 * u + wi];
              any |= q >= 0;
              sum += q >= 0 ? sm.ws[q][lane] : 0.0;
            }
            if (any) __stcg(rows + (size_t)t * 32 + lane, sum);
            if (lane == 0) __stcg(lives + t, (uint8_t)any);
          }
          __syncthreads();
        }
        if (threadIdx.x == 0) {
          __threadfence();
          atomicAdd(bar, 1u);
          target += size;
          sm.flag = gn_wait(bar, target, g);
        }
        __syncthreads();
        if (sm.flag) return;
        // column g by warps g and g + 8: 32 tiles of the column at a time, the
        // live ones' sums fetched into ws, half of them by each warp, then
        // added in order by warp g
        {
          const int g8 = warp & 7;
          double v = 0;
          for (int b0 = g8; b0 - g8 < ntiles; b0 += 8 * 32) {
            const int t = b0 + 8 * lane;
            const bool on = t < ntiles && __ldcg(lives + t) != 0;
            const unsigned m = __ballot_sync(FULL_MASK, on);
            const int cnt = __popc(m), mid = (cnt + 1) / 2;
            const int q0 = warp < 8 ? 0 : mid, q1 = warp < 8 ? mid : cnt;
            if (on) sm.pick[warp][__popc(m & ((1u << lane) - 1))] = t;
            __syncwarp();
            double c[16];
#pragma unroll
            for (int q = 0; q < 16; ++q)
              if (q0 + q < q1)
                c[q] = __ldcg(rows + (size_t)sm.pick[warp][q0 + q] * 32 + lane);
#pragma unroll
            for (int q = 0; q < 16; ++q)
              if (q0 + q < q1) sm.ws[g8 * 32 + q0 + q][lane] = c[q];
            __syncthreads();
            if (warp < 8) {
#pragma unroll 8
              for (int q = 0; q < cnt; ++q) v += sm.ws[g8 * 32 + q][lane];
            }
            __syncthreads();
          }
          if (warp < 8) sm.sh[warp][lane] = v;
        }
        __syncthreads();
        if (warp == 0) {
          double t = 0;
#pragma unroll
          for (int q = 0; q < 8; ++q) t += sm.sh[q][lane];
          sm.tot[lane] = t;
          S.sums[L][lane] = t;
          __syncwarp();
          if (g.only < 0) gn_step_warp(&S, sm.tot, L, it == 0);
        }
        __syncthreads();
        par ^= 1;
        if (S.done && g.only < 0) break;
      }
    }
    if (rank != 0) return;
    if (g.only < 0 && warp == 0) {
      // finalize_objects: the volume pose and the virtual camera pose
      // (tracking.cpp:695-696); (float)T is the last Tf
      float* Tco = reinterpret_cast<float*>(&S.Tf);
      float* Tv = reinterpret_cast<float*>(&S.T_virtual);
      float* tmp = reinterpret_cast<float*>(&sm.M);
      float* pose = g.poses + 16 * s;
      const float two = mul_warp(reinterpret_cast<const float*>(&S.T_w_c2), Tco, lane);
      const float it = inverse_warp(Tco, lane);
      if (lane < 16) {
        pose[lane] = two;
        tmp[lane] = it;
      }
      __syncwarp();
      const float tv = mul_warp(reinterpret_cast<const float*>(&S.T_w_o1), tmp, lane);
      if (lane < 16) Tv[lane] = tv;
    }
    __syncthreads();
    gn_copy_state(&S, a.st + s);
  }
}

// ------------------------------------------------------------------ host side
static int div_up(long long a, int b) { return (int)((a + b - 1) / b); }

template <typename T>
static int talloc(Context* ctx, T** p, size_t n) {
  if (cudaMalloc((void**)p, sizeof(T) * (n ? n : 1)) != cudaSuccess) {
    ctx->last_error = "tracking buffer allocation failed";
    return MF_E_CUDA;
  }
  ctx->track->allocs.push_back(*p);
  MF_CUDA(cudaMemsetAsync(*p, 0, sizeof(T) * (n ? n : 1), ctx->stream));
  return MF_OK;
}

int track_init(Context* ctx) {
  if (ctx->track) return MF_OK;
  TrackState* ts = new TrackState;
  ctx->track = ts;
  for (int i = 0; i < MAX_INSTANCES; ++i) ts->slot_kind[i] = -1;
  ts->levels = std::max(1, std::min(ctx->cfg.pyramid_levels, MAX_PYR));
  PyrPtrs& P = ts->pyr;
  for (int l = 0; l < ts->levels; ++l) {
    P.w[l] = ctx->W >> l;
    P.h[l] = ctx->H >> l;
    const size_t n = (size_t)P.w[l] * P.h[l];
    int rc = 0;
    rc |= talloc(ctx, &P.D[l], n);
    rc |= talloc(ctx, &P.I[0][l], n);
    rc |= talloc(ctx, &P.I[1][l], n);
    rc |= talloc(ctx, &P.V[0][l], n);
    rc |= talloc(ctx, &P.V[1][l], n);
    rc |= talloc(ctx, &P.N[l], n);
    rc |= talloc(ctx, &P.GX[l], n);
    rc |= talloc(ctx, &P.GY[l], n);
    rc |= talloc(ctx, &P.COV[l], n);
    rc |= talloc(ctx, &P.MASK[l], n);
    for (int s = 0; s < ctx->cfg.max_instances; ++s) {
      rc |= talloc(ctx, &ts->rD[s][l], n);
      rc |= talloc(ctx, &ts->rV[s][l], n);
    }
    if (rc) return MF_E_CUDA;
  }
  ts->max_tiles = 0;
  for (int l = 0; l < ts->levels; ++l)
    ts->max_tiles = std::max(ts->max_tiles, div_up((long long)P.w[l] * P.h[l], GN_THREADS * gn_pix(l)));
  if (talloc(ctx, &ts->d_state, MAX_INSTANCES)) return MF_E_CUDA;
  if (talloc(ctx, &ts->d_partials, (size_t)ts->max_tiles * 32)) return MF_E_CUDA;
  if (talloc(ctx, &ts->d_zr, (size_t)MAX_PYR * ts->max_tiles)) return MF_E_CUDA;
  ts->max_segs = div_up((long long)ctx->W * ctx->H, 32);
  if (talloc(ctx, &ts->d_zs, (size_t)MAX_PYR * ts->max_segs)) return MF_E_CUDA;
  if (talloc(ctx, &ts->d_Twc_prev, 16)) return MF_E_CUDA;
  if (talloc(ctx, &ts->d_mask0, (size_t)ctx->W * ctx->H)) return MF_E_CUDA;
  if (talloc(ctx, &ts->d_gnbar, MAX_INSTANCES)) return MF_E_CUDA;
  if (talloc(ctx, &ts->d_gnrows, 2 * GN_CAM_ROWS * 32)) return MF_E_CUDA;
  if (talloc(ctx, &ts->d_objrows, (size_t)2 * ctx->cfg.max_instances * ts->max_tiles * 32)) return MF_E_CUDA;
  if (talloc(ctx, &ts->d_objlive, (size_t)2 * ctx->cfg.max_instances * ts->max_tiles)) return MF_E_CUDA;
  // the GN launches need every CTA resident: a grid is at most the SM count
  // times the CTAs one SM holds
  {
    int sms = 0, b = 0;
    MF_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
    MF_CUDA(cudaFuncSetAttribute(gn_camera_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(GNShared)));
    MF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, gn_camera_kernel, GN_BLOCK,
                                                          sizeof(GNShared)));
    ts->coop_blocks = sms * b;
    MF_CUDA(cudaFuncSetAttribute(gn_objects_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(GOShared)));
    MF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, gn_objects_kernel, GO_BLOCK,
                                                          sizeof(GOShared)));
    ts->obj_blocks = sms * b;
  }
  // Tracking::Tracking, tracking.cpp:77-84: gaussian[i] = expf(-(x*x) / (2 delta^2)),
  // x = i - 2, delta = 4 (computed on the host exactly as the reference does).
  for (int i = 0; i < 5; ++i) {
    const int x = i - 2;
    ts->gaussian[i] = expf(-(x * x) / (2 * 4.0f * 4.0f));
  }
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  return MF_OK;
}

void track_free(Context* ctx) {
  if (!ctx->track) return;
  for (void* p : ctx->track->allocs) cudaFree(p);
  delete ctx->track;
  ctx->track = nullptr;
}

static F4 kdiv(const mf_config& c, int l) {
  const float d = float(1 << l);
  return F4{c.k[0] / d, c.k[1] / d, c.k[2] / d, c.k[3] / d};
}

// Tracking::set_params_frame, tracking.cpp:142-171 (buildPyramid :776-818).
int track_preprocess(Context* ctx, bool clear_mask) {
  if (int rc = track_init(ctx)) return rc;
  TrackState& T = *ctx->track;
  PyrPtrs& P = T.pyr;
  const int W = ctx->W, H = ctx->H;
  Gauss25 g;
  for (int i = 0; i < 5; ++i)
    for (int j = 0; j < 5; ++j) g.g[5 * i + j] = T.gaussian[i] * T.gaussian[j];
  bilateral_kernel<<<dim3(div_up(W, BIL_W), div_up(H, BIL_H), 2), BIL_W * BIL_H, 0, ctx->stream>>>(
      ctx->d_grey, ctx->d_depth, P.I[T.cur][0], P.D[0], W, H, g);
  MF_CUDA(cudaGetLastError());
  const float e_d = 0.1f * 3;
  if (T.levels > 1) {
    HalfLevels hl{};
    hl.in[0] = P.I[T.cur][0];
    hl.in[1] = P.D[0];
    for (int l = 0; l < T.levels; ++l) {
      hl.out[0][l] = P.I[T.cur][l];
      hl.out[1][l] = P.D[l];
      hl.w[l] = P.w[l];
      hl.h[l] = P.h[l];
    }
    hl.levels = T.levels;
    half_sample_levels_kernel<<<dim3(div_up(P.w[1], HALF_T), div_up(P.h[1], HALF_T), 2),
                                HALF_T * HALF_T, 0, ctx->stream>>>(hl, e_d);
    MF_CUDA(cudaGetLastError());
  }
  // vertices, normals, gradients, covariances and the cleared outlier masks of
  // every level
  LevelMaps m{};
  for (int l = 0; l < T.levels; ++l) {
    const F4 kl = kdiv(ctx->cfg, l);
    m.D[l] = P.D[l];
    m.V[l] = P.V[T.cur][l];
    m.I[l] = P.I[T.cur][l];
    m.N[l] = P.N[l];
    m.GX[l] = P.GX[l];
    m.GY[l] = P.GY[l];
    m.COV[l] = P.COV[l];
    m.MASK[l] = clear_mask ? P.MASK[l] : nullptr;
    m.w[l] = P.w[l];
    m.h[l] = P.h[l];
    m.invK[l] = inverse_camera_matrix(kl);
    m.focal[l] = kl.x;
  }
  m.negy = ctx->cfg.k[1] < 0.f;
  const dim3 grid(div_up((long long)P.w[0] * P.h[0], 256), T.levels);
  normal_grad_cov_levels_kernel<<<grid, 256, 0, ctx->stream>>>(m);
  MF_CUDA(cudaGetLastError());
  return MF_OK;
}

// Tracking::setRefImgFromCurr, tracking.cpp:1400-1413: the live intensity and
// vertex pyramids become the reference (a buffer swap instead of a copy).
int track_set_ref(Context* ctx) {
  if (int rc = track_init(ctx)) return rc;
  ctx->track->cur = 1 - ctx->track->cur;
  ctx->track->have_ref = true;
  ctx->track->tracked = false;
  return MF_OK;
}

// The camera's ICP outlier mask, trackLiveFrame(..., mask): cv::resize to each
// level: 2x (INTER_AREA) keeps any nonzero of a 2x2 cell, 4x (INTER_LINEAR)
// samples taps 4x+1 and 4x+2 per axis.
struct MaskLevels {
  uint8_t* out[MAX_PYR];
  int w[MAX_PYR], h[MAX_PYR];
};

// One launch for every level (level = blockIdx.y); each level reads m0 only.
__global__ void mask_pyramid_kernel(const uint8_t* __restrict__ m0, MaskLevels ml, int W) {
  const int l = blockIdx.y;
  const int w = ml.w[l], h = ml.h[l];
  uint8_t* __restrict__ out = ml.out[l];
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= w * h) return;
  const int x = p % w, y = p / w;
  uint8_t v;
  if (l == 0) {
    v = m0[p];
  } else {
    const int o = l == 1 ? 0 : (1 << (l - 1)) - 1, s = 1 << l;
    v = 0;
    for (int dy = 0; dy < 2; ++dy)
      for (int dx = 0; dx < 2; ++dx) v |= m0[(s * x + o + dx) + (s * y + o + dy) * W];
  }
  out[p] = v ? 1 : 0;
}

// Mask of the pixels whose composite label belongs to a moving object
// (the dynamic-object mask of Kfusion::tracking, kfusion.cpp:358-393).
__global__ void label_mask_kernel(const int* __restrict__ label, uint32_t moving,
                                  uint8_t* __restrict__ out, int n) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int l = label[p];
  out[p] = (l >= 0 && l < 32 && ((moving >> l) & 1u)) ? 255 : 0;
}

int track_set_mask(Context* ctx, const uint8_t* d_mask0) {
  TrackState& T = *ctx->track;
  PyrPtrs& P = T.pyr;
  MaskLevels ml{};
  for (int l = 0; l < T.levels; ++l) {
    ml.out[l] = P.MASK[l];
    ml.w[l] = P.w[l];
    ml.h[l] = P.h[l];
  }
  mask_pyramid_kernel<<<dim3(div_up((long long)P.w[0] * P.h[0], 256), T.levels), 256, 0,
                        ctx->stream>>>(d_mask0, ml, ctx->W);
  MF_CUDA(cudaGetLastError());
  return MF_OK;
}

static int render_reference(Context* ctx, const IdList& slots) {
  TrackState& T = *ctx->track;
  PyrPtrs& P = T.pyr;
  const int WH = ctx->W * ctx->H;
  SlotPtrs sp{};
  for (int i = 0; i < slots.n; ++i) sp.D[i] = T.rD[slots.v[i]][0];
  render_depth_kernel<<<dim3(div_up(WH, 256), slots.n), 256, 0, ctx->stream>>>(
      ctx->d_vertex, ctx->d_label, T.d_state, slots, sp, ctx->W, WH);
  MF_CUDA(cudaGetLastError());
  SlotLevels sl{};
  for (int l = 0; l < T.levels; ++l) {
    for (int i = 0; i < slots.n; ++i) {
      sl.D[l][i] = T.rD[slots.v[i]][l];
      sl.V[l][i] = T.rV[slots.v[i]][l];
    }
    sl.w[l] = P.w[l];
    sl.h[l] = P.h[l];
    sl.invK[l] = inverse_camera_matrix(kdiv(ctx->cfg, l));
  }
  sl.levels = T.levels;
  reference_levels_kernel<<<dim3(div_up(P.w[0], 2 * HALF_T), div_up(P.h[0], 2 * HALF_T), slots.n),
                            HALF_T * HALF_T, 0, ctx->stream>>>(sl, 0.1f * 3);
  MF_CUDA(cudaGetLastError());
  return MF_OK;
}

static const void* sums_ptr(const TrackState& T, int slot, int L) {
  return (const char*)(T.d_state + slot) + offsetof(GNState, sums) + sizeof(double) * 32 * L;
}

static GNArgs make_args(Context* ctx) {
  TrackState& T = *ctx->track;
  GNArgs a;
  std::memset(&a, 0, sizeof(a));
  a.pyr = T.pyr;
  a.cur = T.cur;
  a.W = ctx->W; a.H = ctx->H;
  a.mvertex = ctx->d_vertex; a.mnormal = ctx->d_normal; a.mlabel = ctx->d_label;
  for (int l = 0; l < T.levels; ++l) {
    for (int s = 0; s < ctx->cfg.max_instances; ++s) a.rV[l][s] = T.rV[s][l];
    a.kL[l] = kdiv(ctx->cfg, l);
  }
  a.st = T.d_state;
  a.partials = T.d_partials;
  a.max_tiles = T.max_tiles;
  a.zr = T.d_zr;
  a.zs = T.d_zs;
  a.max_segs = T.max_segs;
  a.k0 = kdiv(ctx->cfg, 0);
  // obtainErrorParameters (TUM branch, tracking.cpp:766-772) keeps sigma_bright
  // in a float member; trackRGB uses 1.0 / sigma_bright (double) as a float.
  const float sigma_bright = (float)(sqrtf(100.0f) / 255.0);
  a.inv_cov_rgb = (float)(1.0 / (double)sigma_bright);
  a.robust = ctx->cfg.robust_kernel;
  a.use_icp = ctx->cfg.use_icp;
  a.use_rgb = ctx->cfg.use_rgb;
  return a;
}

// Live depth range of every GN tile at every level (object problems read it to
// skip tiles that cannot hold a valid row).  Recomputed before each object
// evaluation, so it always matches the live vertex and normal maps.
static int tile_depth_range(Context* ctx) {
  TrackState& T = *ctx->track;
  const int tiles = div_up((long long)T.pyr.w[0] * T.pyr.h[0], GN_THREADS * gn_pix(0));
  tile_depth_range_kernel<<<dim3(tiles, T.levels), GN_THREADS, 0, ctx->stream>>>(
      T.pyr, T.cur, T.d_zr, T.max_tiles, T.d_zs, T.max_segs);
  MF_CUDA(cudaGetLastError());
  return MF_OK;
}

int track_waited(Context* ctx) {
  if (!*(volatile int*)ctx->gn_timeout) return MF_OK;
  ctx->last_error = "a Gauss-Newton launch gave up waiting for its CTAs (mf_status clears this)";
  return MF_E_TIMEOUT;
}

// The camera's GN launch: the whole loop, or with `only` >= 0 one evaluation
// of that level whose sums land in the problem's state (plain mode).
static int launch_gn_camera(Context* ctx, const GNArgs& a, int only) {
  TrackState& T = *ctx->track;
  GNLoop g{};
  g.levels = T.levels;
  g.only = only;
  g.rows = T.d_gnrows;
  g.bar = T.d_gnbar;
  g.polls = ctx->gn_polls;
  g.status = ctx->d_status;
  g.timeout = ctx->gn_timeout;
  g.poses = ctx->d_Twc;
  int rows = 1;
  for (int L = 0; L < T.levels; ++L) {
    g.iters[L] = ctx->cfg.gn_iterations[L];
    rows = std::max(rows, std::min(div_up((long long)T.pyr.w[L] * T.pyr.h[L],
                                          GN_THREADS * gn_pix(L)), GN_CAM_ROWS));
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(std::min(rows, T.coop_blocks));
  cfg.blockDim = dim3(GN_BLOCK);
  cfg.dynamicSmemBytes = sizeof(GNShared);
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, gn_camera_kernel, a, g);
  if (e != cudaSuccess) {
    ctx->last_error = std::string("camera GN launch: ") + cudaGetErrorString(e);
    return MF_E_CUDA;
  }
  return MF_OK;
}

// The objects' GN launch, as launch_gn_camera: GO_CTAS CTAs per object while
// the device has them, so that in a frame with few objects the background's
// allocation and integration find SMs beside it.  Frame with three objects at
// 640x480: 8 per object 1119 us, 16 1017, 24 980, 32 975, every SM 980; with
// six at 1280x720: 3097, 2651, 2518, 2522, 2527.
constexpr int GO_CTAS = 32;
static int launch_gn_objects(Context* ctx, const GNArgs& a, const IdList& slots, int only) {
  TrackState& T = *ctx->track;
  GNLoop g{};
  g.levels = T.levels;
  g.only = only;
  g.rows = T.d_objrows;
  g.lives = T.d_objlive;
  g.slots = ctx->cfg.max_instances;
  g.bar = T.d_gnbar;
  g.polls = ctx->gn_polls;
  g.status = ctx->d_status;
  g.timeout = ctx->gn_timeout;
  g.poses = ctx->d_Two;
  for (int L = 0; L < T.levels; ++L) g.iters[L] = ctx->cfg.gn_iterations[L];
  const int ctas = std::min(T.obj_blocks, GO_CTAS * slots.n);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(GO_BLOCK);
  cfg.dynamicSmemBytes = sizeof(GOShared);
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e =
      cudaLaunchKernelEx(&cfg, gn_objects_kernel, a, g, slots, (const float*)ctx->d_Twc);
  if (e != cudaSuccess) {
    ctx->last_error = std::string("object GN launch: ") + cudaGetErrorString(e);
    return MF_E_CUDA;
  }
  return MF_OK;
}

// Host-driven GN of one problem: the sums come back to the host every
// iteration and the step runs there (the reference's structure on a GPU).
static int gn_host(Context* ctx, int slot) {
  TrackState& T = *ctx->track;
  IdList one;
  one.n = 1;
  one.v[0] = slot;
  GNState S;
  MF_CUDA(cudaMemcpyAsync(&S, T.d_state + slot, sizeof(GNState), cudaMemcpyDeviceToHost,
                          ctx->stream));
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  for (int L = T.levels - 1; L >= 0; --L) {
    S.prev_err = INFINITY;
    S.done = 0;
    S.ticket = 0;
    const GNArgs a = make_args(ctx);
    for (int it = 0; it < ctx->cfg.gn_iterations[L] && !S.done; ++it) {
      MF_CUDA(cudaMemcpyAsync(T.d_state + slot, &S, sizeof(GNState), cudaMemcpyHostToDevice,
                              ctx->stream));
      MF_CUDA(cudaMemsetAsync(T.d_gnbar + slot, 0, sizeof(unsigned), ctx->stream));
      if (S.kind == 0) {
        if (int rc = launch_gn_camera(ctx, a, L)) return rc;
      } else {
        if (int rc = launch_gn_objects(ctx, a, one, L)) return rc;
      }
      MF_CUDA(cudaMemcpyAsync(S.sums[L], sums_ptr(T, slot, L), sizeof(double) * 32,
                              cudaMemcpyDeviceToHost, ctx->stream));
      MF_CUDA(cudaStreamSynchronize(ctx->stream));
      if (int rc = track_waited(ctx)) return rc;
      gn_step(S, S.sums[L], L);
    }
  }
  MF_CUDA(cudaMemcpyAsync(T.d_state + slot, &S, sizeof(GNState), cudaMemcpyHostToDevice,
                          ctx->stream));
  return MF_OK;
}

// Tracking::trackLiveFrame with the current model maps; the camera pose is read
// from and written back to the device.  `moving` (bit per label) selects the
// pixels excluded from ICP (trackLiveFrame(..., mask)); 0 = no mask.
// The parts of trackLiveFrame before its GN that read neither the live
// pyramid nor the ICP outlier mask: the problem's setup from the current
// (pre-tracking) camera pose and the rendered reference of the model maps.
int track_camera_pre(Context* ctx, int retrack) {
  if (int rc = track_init(ctx)) return rc;
  TrackState& T = *ctx->track;
  const mf_config& c = ctx->cfg;
  if (retrack && !T.tracked) {
    ctx->last_error = "mf_retrack_camera: no mf_track_camera on this frame";
    return MF_E_STATE;
  }
  T.tracked = true;
  T.slot_kind[0] = 0;
  setup_camera_kernel<<<1, 32, 0, ctx->stream>>>(T.d_state, ctx->d_Twc, T.d_Twc_prev,
                                                 F4{c.k[0], c.k[1], c.k[2], c.k[3]}, retrack,
                                                 T.d_gnbar);
  MF_CUDA(cudaGetLastError());
  IdList cam;
  cam.n = 1;
  cam.v[0] = 0;
  return render_reference(ctx, cam);
}

// The ICP outlier mask of the moving objects' pixels (after the pyramid,
// whose normals kernel clears the mask planes).
int track_camera_mask(Context* ctx, uint32_t moving) {
  if (!moving) return MF_OK;
  TrackState& T = *ctx->track;
  label_mask_kernel<<<div_up((long long)ctx->W * ctx->H, 256), 256, 0, ctx->stream>>>(
      ctx->d_label, moving, T.d_mask0, ctx->W * ctx->H);
  return track_set_mask(ctx, T.d_mask0);
}

int track_camera_gn(Context* ctx) {
  TrackState& T = *ctx->track;
  if (ctx->cfg.batched) return launch_gn_camera(ctx, make_args(ctx), -1);
  if (int rc = gn_host(ctx, 0)) return rc;
  finalize_camera_kernel<<<1, 1, 0, ctx->stream>>>(T.d_state, ctx->d_Twc);
  MF_CUDA(cudaGetLastError());
  return MF_OK;
}

int track_camera(Context* ctx, uint32_t moving, int retrack) {
  if (int rc = track_camera_pre(ctx, retrack)) return rc;
  if (int rc = track_camera_mask(ctx, moving)) return rc;
  return track_camera_gn(ctx);
}

// Tracking::trackEachObject for every id (instance ids >= 1), against the
// model maps of the last raycast, from the previous camera pose (saved by
// track_camera) to the current one.

// The parts of trackEachObject before its GN that need neither the freshly
// tracked camera pose nor the live pyramid: the problems' setup from the
// previous camera pose (saved by track_camera_pre) and the objects' last
// poses, and their rendered references.
int track_objects_pre(Context* ctx, const IdList& ids) {
  if (int rc = track_init(ctx)) return rc;
  if (ids.n == 0) return MF_OK;
  TrackState& T = *ctx->track;
  for (int i = 0; i < ids.n; ++i) T.slot_kind[ids.v[i]] = 1;
  setup_objects_pre_kernel<<<div_up(ids.n, 4), 128, 0, ctx->stream>>>(
      T.d_state, T.d_gnbar, ids, T.d_Twc_prev, ctx->d_Two, ctx->d_inst_label);
  MF_CUDA(cudaGetLastError());
  return render_reference(ctx, ids);
}

// After track_objects_pre: the rest of the setup with the tracked camera pose,
// the GN and its results (all three in the batched mode's one launch).
int track_objects_gn(Context* ctx, const IdList& ids) {
  if (ids.n == 0) return MF_OK;
  if (int rc = tile_depth_range(ctx)) return rc;
  if (ctx->cfg.batched) return launch_gn_objects(ctx, make_args(ctx), ids, -1);
  TrackState& T = *ctx->track;
  setup_objects_post_kernel<<<1, 32, 0, ctx->stream>>>(T.d_state, ids, ctx->d_Twc);
  MF_CUDA(cudaGetLastError());
  for (int i = 0; i < ids.n; ++i)
    if (int rc = gn_host(ctx, ids.v[i])) return rc;
  finalize_objects_kernel<<<1, 32, 0, ctx->stream>>>(T.d_state, ids, ctx->d_Two);
  MF_CUDA(cudaGetLastError());
  return MF_OK;
}

int track_objects(Context* ctx, const IdList& ids) {
  if (int rc = track_objects_pre(ctx, ids)) return rc;
  return track_objects_gn(ctx, ids);
}

bool track_has_ref(Context* ctx) { return ctx->track && ctx->track->have_ref; }
int track_parity(Context* ctx) { return ctx->track->cur; }
void track_set_parity(Context* ctx, int parity) { ctx->track->cur = parity; }

void track_save_prev_camera(Context* ctx) {
  cudaMemcpyAsync(ctx->track->d_Twc_prev, ctx->d_Twc, 64, cudaMemcpyDeviceToDevice, ctx->stream);
}

int track_info(Context* ctx, int slot, int* iters, double* sums, double* T64) {
  if (!ctx->track) return MF_E_STATE;
  GNState S;
  MF_CUDA(cudaMemcpyAsync(&S, ctx->track->d_state + slot, sizeof(GNState),
                          cudaMemcpyDeviceToHost, ctx->stream));
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  if (int rc = track_waited(ctx)) return rc;
  for (int l = 0; l < MAX_PYR; ++l) {
    if (iters) iters[l] = S.iters[l];
    if (sums) for (int i = 0; i < 32; ++i) sums[32 * l + i] = S.sums[l][i];
  }
  if (T64) for (int i = 0; i < 16; ++i) T64[i] = S.T[i];
  return S.fallback ? 1 : 0;
}

// One evaluation of the normal equations at a given level for one problem at
// its current pose, without a step (parity checks of residuals + reduction).
int track_eval(Context* ctx, int slot, int L, const float* pose16, double* sums) {
  if (!ctx->track) return MF_E_STATE;
  TrackState& T = *ctx->track;
  if (T.slot_kind[slot] < 0) {
    ctx->last_error = "mf_track_eval: slot " + std::to_string(slot) + " has no tracking problem";
    return MF_E_STATE;
  }
  GNState S;
  MF_CUDA(cudaMemcpyAsync(&S, T.d_state + slot, sizeof(GNState), cudaMemcpyDeviceToHost,
                          ctx->stream));
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  if (pose16) {
    std::memcpy(&S.Tf, pose16, 64);
    S.invTf = inverse(S.Tf);
    for (int i = 0; i < 16; ++i) S.T[i] = pose16[i];
  }
  S.done = 0;
  S.ticket = 0;
  MF_CUDA(cudaMemcpyAsync(T.d_state + slot, &S, sizeof(GNState), cudaMemcpyHostToDevice,
                          ctx->stream));
  const GNArgs a = make_args(ctx);
  const int tiles = div_up((long long)T.pyr.w[L] * T.pyr.h[L], GN_THREADS * gn_pix(L));
  if (S.kind == 1)
    if (int rc = tile_depth_range(ctx)) return rc;
  if (S.kind == 0) gn_eval_kernel<0><<<tiles, GN_THREADS, 0, ctx->stream>>>(a, slot, L);
  else gn_eval_kernel<1><<<tiles, GN_THREADS, 0, ctx->stream>>>(a, slot, L);
  MF_CUDA(cudaGetLastError());
  MF_CUDA(cudaMemcpyAsync(sums, sums_ptr(T, slot, L), sizeof(double) * 32,
                          cudaMemcpyDeviceToHost, ctx->stream));
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  return MF_OK;
}

// Timing and algorithmic bytes of one camera GN evaluation at level 0 on the
// current frame (used after the timed region).  Bytes per pixel: ICP live
// vertex, normal, covariance and the model vertex and normal (5 x 12 B), RGB
// rendered and live reference vertex (2 x 12 B), reference intensity (4 B), the
// 4-tap intensity and gradient gathers (16 + 32 B) and the outlier mask (2 B).
int profile_gn(Context* ctx, int reps, double* us, double* bytes) {
  if (!ctx->track) return MF_E_STATE;
  TrackState& T = *ctx->track;
  GNState S;
  MF_CUDA(cudaMemcpyAsync(&S, T.d_state, sizeof(GNState), cudaMemcpyDeviceToHost, ctx->stream));
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  S.done = 0;
  S.ticket = 0;
  MF_CUDA(cudaMemcpyAsync(T.d_state, &S, sizeof(GNState), cudaMemcpyHostToDevice, ctx->stream));
  const GNArgs a = make_args(ctx);
  auto launch = [&]() -> int {
    MF_CUDA(cudaMemsetAsync(T.d_gnbar, 0, sizeof(unsigned), ctx->stream));
    return launch_gn_camera(ctx, a, 0);
  };
  if (int rc = launch()) return rc;  // warm
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, ctx->stream);
  for (int r = 0; r < reps; ++r)
    if (int rc = launch()) return rc;
  cudaEventRecord(e1, ctx->stream);
  MF_CUDA(cudaEventSynchronize(e1));
  float ms = 0;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  MF_CUDA(cudaGetLastError());
  *us = 1e3 * ms / reps;
  *bytes = 138.0 * T.pyr.w[0] * T.pyr.h[0];
  return MF_OK;
}

int track_download_level(Context* ctx, int L, int which, float* out) {
  if (!ctx->track) return MF_E_STATE;
  TrackState& T = *ctx->track;
  const PyrPtrs& P = T.pyr;
  const size_t n = (size_t)P.w[L] * P.h[L];
  const void* src = nullptr;
  size_t bytes = 4 * n;
  switch (which) {
    case 0: src = P.D[L]; break;
    case 1: src = P.I[T.cur][L]; break;
    case 2: src = P.V[T.cur][L]; bytes = 12 * n; break;
    case 3: src = P.N[L]; bytes = 12 * n; break;
    case 4: src = P.GX[L]; break;
    case 5: src = P.GY[L]; break;
    case 6: src = P.COV[L]; bytes = 12 * n; break;
    case 7: src = T.rV[0][L]; bytes = 12 * n; break;
    default: return MF_E_ARG;
  }
  MF_CUDA(cudaMemcpyAsync(out, src, bytes, cudaMemcpyDeviceToHost, ctx->stream));
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  return MF_OK;
}

// ------------------------------------------------------------------------
// Normal-equation evaluation that allocates nothing (mf_track_eval_static).
//
// Same sums as track_eval (the per-pixel rows and the FP64 reduction of
// gn_eval_kernel, in the same order, so the two agree bit for bit), but the
// scratch -- the per-CTA FP64 partials, the 32 result sums and the CTA ticket
// -- is the file-scope array below, not a cudaMalloc'd buffer, and the pose is
// a kernel argument, so the context's GN state is not touched either.
// Layout of the array (bytes):
//   [0, EVAL_PARTIALS_BYTES)        double partials[EVAL_MAX_TILES][32]
//   [EVAL_SUMS_OFF, +256)           double sums[32]
//   [EVAL_TICKET_OFF, +4)           unsigned ticket (zeroed before each launch)
// EVAL_MAX_TILES bounds the level's pixel count: 4096 CTAs x 768 pixels at
// level 0 (3 145 728 px, e.g. 2048x1536) and 4096 x 256 above it.
constexpr int EVAL_MAX_TILES = 4096;
constexpr size_t EVAL_PARTIALS_BYTES = (size_t)EVAL_MAX_TILES * 32 * sizeof(double);
constexpr size_t EVAL_SUMS_OFF = EVAL_PARTIALS_BYTES;
constexpr size_t EVAL_TICKET_OFF = EVAL_SUMS_OFF + 32 * sizeof(double);
constexpr size_t EVAL_SCRATCH_BYTES = EVAL_TICKET_OFF + 256;
static __device__ __align__(256) unsigned char g_eval_scratch[EVAL_SCRATCH_BYTES];

template <int KIND>
__global__ void __launch_bounds__(GN_THREADS, 2)
gn_eval_static_kernel(GNArgs a, int s, int L, int set_pose, M4 Tf, M4 invTf,
                      unsigned char* scratch) {
  // the problem's constants, with the pose to evaluate at, in shared memory
  __shared__ GNState S;
  {
    static_assert(sizeof(GNState) % 4 == 0, "GNState is copied as words");
    const int* src = reinterpret_cast<const int*>(&a.st[s]);
    int* dst = reinterpret_cast<int*>(&S);
    for (int i = threadIdx.x; i < (int)(sizeof(GNState) / 4); i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  if (threadIdx.x == 0 && set_pose) {
    S.Tf = Tf;
    S.invTf = invTf;
  }
  __syncthreads();
  double* partials = reinterpret_cast<double*>(scratch);
  double* out = reinterpret_cast<double*>(scratch + EVAL_SUMS_OFF);
  unsigned* ticket = reinterpret_cast<unsigned*>(scratch + EVAL_TICKET_OFF);

  const GNView lv = gn_view(a, L);
  const int w = lv.w, n = w * lv.h;
  // object problems: a tile that cannot hold a valid row skips its pixels
  bool live = true;
  if (KIND == 1) {
    __shared__ int s_live;
    if (threadIdx.x < 32) {
      const bool tl = object_tile_live(a, lv.kL, S, L, blockIdx.x, w, n);
      if (threadIdx.x == 0) s_live = tl ? 1 : 0;
    }
    __syncthreads();
    live = s_live != 0;
  }
  // FP64 from the warp level up
  __shared__ double sh[GN_THREADS / 32][32];
  __shared__ float red[GN_THREADS / 32][32][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (live) {
    float acc[29];
#pragma unroll
    for (int i = 0; i < 29; ++i) acc[i] = 0.f;
    int cnt[3] = {0, 0, 0};
    const F3* rV = gn_ref_vertex(a, L, s);
    const int ppt = gn_pix(L);
#pragma unroll 1
    for (int k = 0; k < ppt; ++k) {
      const int p = blockIdx.x * (GN_THREADS * ppt) + k * GN_THREADS + threadIdx.x;
      if (p >= n) break;
      Row ri, rr;
      gn_rows<KIND>(a, lv, S, rV, L, p, ri, rr);
      if (a.use_icp) accumulate(acc, cnt, ri, a.robust);
      if (a.use_rgb) accumulate(acc, cnt, rr, a.robust);
    }
    sh[warp][lane] = warp_sum_fp64(acc, cnt, red[warp], lane);
  } else {
    sh[warp][lane] = 0.0;
  }
  __syncthreads();
  __shared__ bool last;
  if (threadIdx.x < 32) {
    double v = 0;
#pragma unroll
    for (int wi = 0; wi < GN_THREADS / 32; ++wi) v += sh[wi][threadIdx.x];
    partials[(size_t)blockIdx.x * 32 + threadIdx.x] = v;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
  __syncthreads();
  if (!last) return;
  __threadfence();
  {
    const int i = threadIdx.x & 31, g = threadIdx.x >> 5;
    double v = 0;
    for (int b = g; b < (int)gridDim.x; b += GN_THREADS / 32)
      v += __ldcg(&partials[(size_t)b * 32 + i]);
    sh[g][i] = v;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = 0;
#pragma unroll
    for (int g = 0; g < GN_THREADS / 32; ++g) v += sh[g][threadIdx.x];
    out[threadIdx.x] = v;
  }
  if (threadIdx.x == 0) *ticket = 0u;
}

// Device address of g_eval_scratch for each device, looked up once per device
// with that device current, on the first call (host code cannot use the
// address of a __device__ variable directly).
static std::mutex g_eval_mutex;
static unsigned char* g_eval_ptr[64] = {};

static int eval_scratch_setup(Context* ctx, unsigned char** out) {
  int dev = -1;
  MF_CUDA(cudaGetDevice(&dev));
  if (dev != ctx->device) {
    ctx->last_error = "mf_track_eval_static: the context's device is not the current device";
    return MF_E_STATE;
  }
  if (dev < 0 || dev >= 64) {
    ctx->last_error = "mf_track_eval_static: device ordinal above 63";
    return MF_E_ARG;
  }
  std::lock_guard<std::mutex> lock(g_eval_mutex);
  if (!g_eval_ptr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_eval_scratch);
    if (e != cudaSuccess || !p) {
      ctx->last_error = std::string("cudaGetSymbolAddress(g_eval_scratch): ") +
                        cudaGetErrorString(e);
      return MF_E_CUDA;
    }
    g_eval_ptr[dev] = static_cast<unsigned char*>(p);
  }
  *out = g_eval_ptr[dev];
  return MF_OK;
}

int track_eval_static(Context* ctx, int slot, int L, const float* pose16, double* sums) {
  const int tiles = div_up((long long)(ctx->W >> L) * (ctx->H >> L), GN_THREADS * gn_pix(L));
  if (tiles > EVAL_MAX_TILES) {
    ctx->last_error = "mf_track_eval_static: level has more than 4096 x " +
                      std::to_string(GN_THREADS * gn_pix(L)) +
                      " pixels (the static scratch holds 4096 CTA partials)";
    return MF_E_ARG;
  }
  if (!ctx->track) return MF_E_STATE;
  const int kind = ctx->track->slot_kind[slot];
  if (kind < 0) {
    ctx->last_error = "mf_track_eval_static: slot " + std::to_string(slot) +
                      " has no tracking problem";
    return MF_E_STATE;
  }
  unsigned char* scratch = nullptr;
  if (int rc = eval_scratch_setup(ctx, &scratch)) return rc;
  M4 Tf{}, invTf{};
  const int set_pose = pose16 ? 1 : 0;
  if (pose16) {
    std::memcpy(&Tf, pose16, 64);
    invTf = inverse(Tf);
  }
  const GNArgs a = make_args(ctx);
  if (kind == 1)
    if (int rc = tile_depth_range(ctx)) return rc;
  // the ticket must be zero when the launch starts (the last CTA also resets it)
  MF_CUDA(cudaMemsetAsync(scratch + EVAL_TICKET_OFF, 0, sizeof(unsigned), ctx->stream));
  if (kind == 0)
    gn_eval_static_kernel<0><<<tiles, GN_THREADS, 0, ctx->stream>>>(a, slot, L, set_pose, Tf,
                                                                     invTf, scratch);
  else
    gn_eval_static_kernel<1><<<tiles, GN_THREADS, 0, ctx->stream>>>(a, slot, L, set_pose, Tf,
                                                                     invTf, scratch);
  MF_CUDA(cudaGetLastError());
  MF_CUDA(cudaMemcpyAsync(sums, scratch + EVAL_SUMS_OFF, 32 * sizeof(double),
                          cudaMemcpyDeviceToHost, ctx->stream));
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  return MF_OK;
}

// ------------------------------------------------------------------------
// The GN step on given inputs, on the device (gn_step_warp, one warp per
// problem) and on the host (gn_step), for checking that the two agree.
// state: n x 36 doubles: T[16], prevT[16], prev_err, kind, first, level;
// sums: n x 32.  out_dev / out_host: n x 68 doubles: T[16], prevT[16],
// prev_err, done, fallback, iterations at the level, Tf[16], invTf[16].
__global__ void gn_step_check_kernel(GNState* st, const double* __restrict__ sums,
                                     const int* __restrict__ first, const int* __restrict__ level) {
  const int i = blockIdx.x;
  gn_step_warp(st + i, sums + 32 * i, level[i], first[i]);
}

static void gn_step_out(const GNState& S, int level, double* o) {
  for (int k = 0; k < 16; ++k) { o[k] = S.T[k]; o[16 + k] = S.prevT[k]; }
  o[32] = S.prev_err;
  o[33] = S.done;
  o[34] = S.fallback;
  o[35] = S.iters[level];
  for (int k = 0; k < 16; ++k) {
    o[36 + k] = m_at(S.Tf, k / 4, k % 4);
    o[52 + k] = m_at(S.invTf, k / 4, k % 4);
  }
}

int gn_step_check(Context* ctx, int n, const double* state, const double* sums, double* out_dev,
                  double* out_host) {
  std::vector<GNState> hs(n);
  std::vector<int> first(n), level(n);
  for (int i = 0; i < n; ++i) {
    GNState& S = hs[i];
    std::memset(&S, 0, sizeof(GNState));
    const double* q = state + 36 * i;
    for (int k = 0; k < 16; ++k) { S.T[k] = q[k]; S.prevT[k] = q[16 + k]; }
    S.prev_err = q[32];
    S.kind = (int)q[33];
    first[i] = (int)q[34];
    level[i] = (int)q[35];
    if (level[i] < 0 || level[i] >= MAX_PYR || (S.kind != 0 && S.kind != 1)) {
      ctx->last_error = "mf_debug_gn_step: level or kind out of range";
      return MF_E_ARG;
    }
    S.Tf = to_m4f(S.T);
    S.invTf = inverse(S.Tf);
  }
  GNState* d_st = nullptr;
  double* d_sums = nullptr;
  int* d_int = nullptr;
  int rc = MF_OK;
  if (cudaMalloc(&d_st, sizeof(GNState) * n) != cudaSuccess ||
      cudaMalloc(&d_sums, sizeof(double) * 32 * n) != cudaSuccess ||
      cudaMalloc(&d_int, sizeof(int) * 2 * n) != cudaSuccess) {
    ctx->last_error = "mf_debug_gn_step: allocation failed";
    rc = MF_E_CUDA;
  }
  std::vector<GNState> ds(n);
  if (rc == MF_OK) {
    cudaMemcpyAsync(d_st, hs.data(), sizeof(GNState) * n, cudaMemcpyHostToDevice, ctx->stream);
    cudaMemcpyAsync(d_sums, sums, sizeof(double) * 32 * n, cudaMemcpyHostToDevice, ctx->stream);
    cudaMemcpyAsync(d_int, first.data(), sizeof(int) * n, cudaMemcpyHostToDevice, ctx->stream);
    cudaMemcpyAsync(d_int + n, level.data(), sizeof(int) * n, cudaMemcpyHostToDevice,
                    ctx->stream);
    gn_step_check_kernel<<<n, 32, 0, ctx->stream>>>(d_st, d_sums, d_int, d_int + n);
    cudaMemcpyAsync(ds.data(), d_st, sizeof(GNState) * n, cudaMemcpyDeviceToHost, ctx->stream);
    const cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) {
      ctx->last_error = std::string("mf_debug_gn_step: ") + cudaGetErrorString(e);
      rc = MF_E_CUDA;
    }
  }
  if (d_st) cudaFree(d_st);
  if (d_sums) cudaFree(d_sums);
  if (d_int) cudaFree(d_int);
  if (rc) return rc;
  for (int i = 0; i < n; ++i) {
    GNState& S = hs[i];
    if (first[i]) S.prev_err = INFINITY;
    gn_step(S, sums + 32 * i, level[i]);
    gn_step_out(S, level[i], out_host + 68 * i);
    gn_step_out(ds[i], level[i], out_dev + 68 * i);
  }
  return MF_OK;
}

// ------------------------------------------------------------------------
// Camera cost at level 0 and its adjoint (no reference counterpart).
//
//   E(T_live, tsdf) = sum_p rho(e_icp(p)) + rho(e_rgb(p))
//
// with the camera rows of the GN (the same validity tests, residuals,
// whitening and robust kernel) at level 0.  Per valid row the kernel adds
// rho'(e) de/d(twist) -- the exact derivative for a left perturbation
// T <- exp(twist) T_live, with the bilinear image gradient of the photometric
// lookup -- and, when asked, rho'(e) de/d(model vertex, normal) into per
// model-pixel FP64 buffers, which the raycast adjoint then carries back to the
// TSDF voxels.  ICP: e = ic n.(v_m - T v) with ic = (n^T P n)^(-1/2).
// Photometric: e = ic_rgb (I_ref(p) - I_live(pi(K T^-1 T_w_r rv(p)))), where
// the reference vertex rv(p) = d(p) K^-1 (x, y, 1) and d(p) is the depth of the
// model vertex at p in the reference camera.
struct CostOut {
  double* partials;  // 8 per CTA: loss, dE/d twist (6), rows
  double* gV;        // 3 per model pixel (may be null)
  double* gN;
  int want_grad;
};

__device__ __forceinline__ void atomic_add3(double* p, F3 v) {
  atomicAdd(p, (double)v.x);
  atomicAdd(p + 1, (double)v.y);
  atomicAdd(p + 2, (double)v.z);
}

__global__ void __launch_bounds__(256)
camera_cost_kernel(GNArgs a, CostOut c) {
  const GNState& S = a.st[0];
  const int w = a.pyr.w[0], h = a.pyr.h[0];
  const int p = blockIdx.x * 256 + threadIdx.x;
  float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // loss, grad[6], rows
  if (p < w * h) {
    // ---- ICP (icp_camera)
    if (a.use_icp && !a.pyr.MASK[0][p]) {
      const F3 nl = a.pyr.N[0][p];
      if (nl.x != INVALIDF) {
        const F3 pv = xform(S.Tf, a.pyr.V[a.cur][0][p]);
        const F3 pp = xform(S.view, pv);
        const float px = pp.x / pp.z, py = pp.y / pp.z;
        if (!(px < 1 || px > (float)(unsigned)(a.W - 2) || py < 1 ||
              py > (float)(unsigned)(a.H - 2) || isnan(px) || isnan(py))) {
          const int q = (int)((unsigned)px + (unsigned)py * a.W);
          const F3 rn = a.mnormal[q];
          if (rn.x != INVALIDF) {
            const F3 diff = a.mvertex[q] - pv;
            const F3 pn = rotate(S.Tf, nl);
            if (!(length(diff) > 0.1f) && !(dot(pn, rn) < 0.8f)) {
              const F3 P = a.pyr.COV[0][p];
              const float sig = rn.x * rn.x * P.x + rn.y * rn.y * P.y + rn.z * rn.z * P.z;
              const float ic = sqrtf((float)(1.0 / (double)sig));
              const float e = ic * dot(rn, diff);
              float wt, loss;
              robust(e, a.robust, wt, loss);
              const float de = wt * e;  // rho'(e)
              v[0] += loss;
              v[7] += 1.f;
              // de/d(v, w) = -ic (n, pv x n)
              const F3 j1 = cross(pv, rn);
              v[1] -= de * ic * rn.x; v[2] -= de * ic * rn.y; v[3] -= de * ic * rn.z;
              v[4] -= de * ic * j1.x; v[5] -= de * ic * j1.y; v[6] -= de * ic * j1.z;
              if (c.want_grad) {
                atomic_add3(c.gV + 3 * (size_t)q, (de * ic) * rn);
                // d ic / d n = -ic^3 (n * P)
                const float ic3 = ic * ic * ic;
                const F3 dic = mk3(-ic3 * rn.x * P.x, -ic3 * rn.y * P.y, -ic3 * rn.z * P.z);
                atomic_add3(c.gN + 3 * (size_t)q, de * (ic * diff + dot(rn, diff) * dic));
              }
            }
          }
        }
      }
    }
    // ---- photometric (rgb_row, camera, level 0)
    if (a.use_rgb) {
      const F3 rv = a.rV[0][0][p];
      const F3 rl = a.pyr.V[1 - a.cur][0][p];
      if (!(rv.z <= 0.f || rv.z == INVALIDF) && !(length(rv - rl) > 0.1f && rl.z > 0.f)) {
        const M4 KL = camera_matrix(a.kL[0]);
        const F3 wv = xform(S.T_w_r, rv);
        const F3 lv = xform(S.invTf, wv);
        const F3 pr = rotate(KL, lv);
        const float px = pr.x / pr.z, py = pr.y / pr.z;
        if (!(px < 1 || px > (float)(unsigned)(w - 2) || py < 1 || py > (float)(unsigned)(h - 2) ||
              isnan(px) || isnan(py))) {
          const float* IL = a.pyr.I[a.cur][0];
          const float fx0 = floorf(px), fy0 = floorf(py);
          const int bx = (int)fx0, by = (int)fy0;
          const float ax = px - fx0, ay = py - fy0;
          const float i00 = IL[bx + by * w], i10 = IL[bx + 1 + by * w];
          const float i01 = IL[bx + (by + 1) * w], i11 = IL[bx + 1 + (by + 1) * w];
          const float residual = a.pyr.I[1 - a.cur][0][p] - bil(IL, w, px, py);
          const float ic = a.inv_cov_rgb;
          const float e = ic * residual;
          float wt, loss;
          robust(e, a.robust, wt, loss);
          const float de = wt * e;
          v[0] += loss;
          v[7] += 1.f;
          // d bil / d(px, py) of the bilinear interpolation itself
          const float gx = (i10 - i00) * (1.f - ay) + (i11 - i01) * ay;
          const float gy = (i01 - i00) * (1.f - ax) + (i11 - i10) * ax;
          const float fxk = KL.r[0].x, fyk = KL.r[1].y, iz = 1.f / lv.z;
          // de/d lv = -ic (gx dpx/dlv + gy dpy/dlv)
          const F3 g_lv = -ic * mk3(gx * fxk * iz, gy * fyk * iz,
                                     -(gx * fxk * lv.x + gy * fyk * lv.y) * iz * iz);
          const F3 g3 = rotate_t(g_lv, S.invTf);  // in world coordinates
          const F3 j1 = cross(wv, g3);
          // lv = T^-1 exp(-twist) wv: de/d(v, w) = -(g3, wv x g3)
          v[1] -= de * g3.x; v[2] -= de * g3.y; v[3] -= de * g3.z;
          v[4] -= de * j1.x; v[5] -= de * j1.y; v[6] -= de * j1.z;
          if (c.want_grad) {
            // rv = d K^-1 (x, y, 1), d = (T_w_r^-1 v_m).z
            const int x = p % w, y = p / w;
            const F3 ray = rotate(inverse_camera_matrix(a.kL[0]), mk3((float)x, (float)y, 1.f));
            const float g_d = dot(rotate_t(g3, S.T_w_r), ray);
            atomic_add3(c.gV + 3 * (size_t)p, (de * g_d) * xyz(S.inv_T_w_r.r[2]));
          }
        }
      }
    }
  }
  // FP64 block sums, fixed order
  __shared__ double sh[8][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    double d = v[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d += __shfl_down_sync(0xffffffffu, d, o);
    if (lane == 0) sh[warp][i] = d;
  }
  __syncthreads();
  if (threadIdx.x < 8) {
    double d = 0;
    for (int i = 0; i < 8; ++i) d += sh[i][threadIdx.x];
    c.partials[(size_t)blockIdx.x * 8 + threadIdx.x] = d;
  }
}

// The eight sums over the CTAs' partials: thread t adds value t & 7 of CTAs
// g, g + 32, ... (g = t / 8) and eight threads add the 32 groups, both in a
// fixed order.  One chain of loads per value over all 1200 CTAs of a 640x480
// frame took 73 us, a chain of 38 takes under 4.
constexpr int COST_GROUPS = 32;
__global__ void __launch_bounds__(8 * COST_GROUPS)
cost_sum_kernel(const double* __restrict__ partials, int n, double* out) {
  __shared__ double sh[COST_GROUPS][8];
  const int i = threadIdx.x & 7, g = threadIdx.x >> 3;
  double d = 0;
#pragma unroll 8
  for (int b = g; b < n; b += COST_GROUPS) d += partials[(size_t)b * 8 + i];
  sh[g][i] = d;
  __syncthreads();
  if (threadIdx.x >= 8) return;
  d = 0;
#pragma unroll
  for (int k = 0; k < COST_GROUPS; ++k) d += sh[k][threadIdx.x];
  out[threadIdx.x] = d;
}

// Camera problem (slot 0) for a cost evaluation: reference pose = the current
// camera pose, live pose = T_live.
__global__ void cost_setup_kernel(GNState* st, const float* __restrict__ Twc, F4 k, M4 Tl,
                                  M4 iTl) {
  GNState& S = st[0];
  const M4 T = load_m4(Twc);
  S.kind = 0; S.label = 0; S.inst = 0; S.done = 0; S.ticket = 0;
  S.T_w_r = T;
  S.inv_T_w_r = inverse(T);
  S.view = mul(camera_matrix(k), S.inv_T_w_r);
  S.Tf = Tl;
  S.invTf = iTl;
}

int camera_cost(Context* ctx, const float* T_live16, int want_grad, double* out8,
                float* d_grad) {
  if (!ctx->track || !ctx->track->have_ref) {
    ctx->last_error = "mf_camera_cost: needs a reference frame (mf_set_ref_from_current) "
                      "and a preprocessed live frame";
    return MF_E_STATE;
  }
  TrackState& T = *ctx->track;
  const size_t WH = (size_t)ctx->W * ctx->H;
  const int nb = (int)((WH + 255) / 256);
  if (!T.d_cost) {
    MF_CUDA(cudaMalloc(&T.d_gmodel, sizeof(double) * 6 * WH));
    MF_CUDA(cudaMalloc(&T.d_cost_part, sizeof(double) * 8 * nb));
    MF_CUDA(cudaMalloc(&T.d_cost, sizeof(double) * 8));
    T.allocs.push_back(T.d_gmodel);
    T.allocs.push_back(T.d_cost_part);
    T.allocs.push_back(T.d_cost);
    T.cost_blocks = nb;
  }
  // the model maps of the current TSDF at the current (reference) camera pose,
  // and with a TSDF gradient each pixel's winner
  const bool grad = want_grad && d_grad;
  if (grad && !T.d_win_hit) {
    MF_CUDA(cudaMalloc(&T.d_win_hit, (sizeof(F4) + 1) * WH));
    T.allocs.push_back(T.d_win_hit);
    T.d_win = (uint8_t*)(T.d_win_hit + WH);
  }
  IdList all;
  all.n = (int)ctx->inst.size();
  for (int i = 0; i < all.n; ++i) all.v[i] = i;
  if (int rc = stage_prepare(ctx, all)) return rc;
  if (int rc = stage_raycast_to(ctx, all, ctx->ray_epsilon, ctx->d_vertex, ctx->d_normal,
                                ctx->d_label, grad ? T.d_win : nullptr,
                                grad ? T.d_win_hit : nullptr))
    return rc;
  M4 Tl;
  std::memcpy(&Tl, T_live16, 64);
  const mf_config& c = ctx->cfg;
  T.slot_kind[0] = 0;
  cost_setup_kernel<<<1, 1, 0, ctx->stream>>>(T.d_state, ctx->d_Twc,
                                              F4{c.k[0], c.k[1], c.k[2], c.k[3]}, Tl,
                                              inverse(Tl));
  MF_CUDA(cudaGetLastError());
  IdList cam;
  cam.n = 1;
  cam.v[0] = 0;
  if (int rc = render_reference(ctx, cam)) return rc;
  double* gV = want_grad ? T.d_gmodel : nullptr;
  double* gN = want_grad ? T.d_gmodel + 3 * WH : nullptr;
  if (want_grad) MF_CUDA(cudaMemsetAsync(T.d_gmodel, 0, sizeof(double) * 6 * WH, ctx->stream));
  const GNArgs a = make_args(ctx);
  camera_cost_kernel<<<nb, 256, 0, ctx->stream>>>(a, CostOut{T.d_cost_part, gV, gN, want_grad});
  cost_sum_kernel<<<1, 8 * COST_GROUPS, 0, ctx->stream>>>(T.d_cost_part, nb, T.d_cost);
  MF_CUDA(cudaGetLastError());
  if (grad)
    if (int rc = stage_raycast_adjoint(ctx, all, T.d_win, T.d_win_hit, gV, gN, d_grad)) return rc;
  MF_CUDA(cudaMemcpyAsync(out8, T.d_cost, sizeof(double) * 8, cudaMemcpyDeviceToHost,
                          ctx->stream));
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  return MF_OK;
}


// ------------------------------------------------------------------------
// Motion residuals (Tracking::compute_residuals, tracking.cpp:1535-1553,
// compute_residual_kernel :1555-1612, compute_icp_residual_kernel :1615-1677,
// compute_rgb_residual_kernel :1680-1747) and the moving-object test
// (check_static_state, rendering/rendering.cpp:907-947, and the inlier ratio
// of kfusion.cpp:312-341).  T_w_l is the freshly tracked camera pose, T_w_r
// the reference pose of the model maps; the photometric reference vertices
// come from the model raycast at T_w_l with the objects at their last poses,
// turned into depth relative to T_w_r (vertex2depth with T_w_r, as the
// reference passes it, preprocessing.cpp:292-309) and back into vertices.
struct MotionArgs {
  PyrPtrs pyr;
  int cur, W, H;
  const F3* mvertex; const F3* mnormal;   // model maps at T_w_r
  const int* mlabel;
  const F3* lvert;                          // model vertices raycast at T_w_l
  const int* llabel;
  int obj_label;    // >= 0: one object's maps (its pixels of the composite maps,
                    // m_vertex / m_normal, and of the live raycast,
                    // m_vertex_bef_integ, rendering.cpp:152-176), no counts
  M4 T_w_l, T_w_r, inv_T_w_r, K, invK;
  float sigma_bright, threshold;
  int use_icp, use_rgb;
  int8_t* res; float* err;
  int* count;                               // [label]: object pixels, [32 + label]: inliers
};

__global__ void motion_residual_kernel(MotionArgs a) {
  const int n = a.W * a.H;
  // the last CTA's idle threads repeat the last pixel (its rows are written
  // with the same values) and count nothing
  const int p0 = blockIdx.x * blockDim.x + threadIdx.x;
  const int p = min(p0, n - 1);
  const int x = p % a.W, y = p / a.W;
  int8_t ri = 0, rr = 0;
  float ei = 0.f, er = 0.f;
  // the outlier-mask test of :1586-1590 never fires: the reference's
  // outlier_mask_ stays the all-zero mask of set_params_frame (:170), since
  // the mask variant of trackLiveFrame keeps its pyramid local (:1781-1787)
  {
    if (a.use_icp) {
      const F3 ln = a.pyr.N[0][p];
      if (ln.x == INVALIDF) {
        ri = -1;
      } else {
        const F3 w_vertex = xform(a.T_w_l, a.pyr.V[a.cur][0][p]);
        const F3 r_vertex = xform(a.inv_T_w_r, w_vertex);
        const F3 proj = rotate(a.K, r_vertex);
        const float px = proj.x / proj.z, py = proj.y / proj.z;
        if (px < 1 || px > (float)(unsigned)(a.W - 2) || py < 1 || py > (float)(unsigned)(a.H - 2) ||
            isnan(px) || isnan(py)) {
          ri = -2;
        } else {
          const int q = (int)((unsigned)px + (unsigned)py * a.W);
          const bool own = a.obj_label < 0 || a.mlabel[q] == a.obj_label;
          const F3 rn = own ? a.mnormal[q] : mk3(INVALIDF, 0.f, 0.f);
          const F3 rv = own ? a.mvertex[q] : mk3(0.f);
          if (rn.x == INVALIDF) {
            ri = -3;
          } else {
            const F3 diff = rv - w_vertex;
            const F3 wn = rotate(a.T_w_l, ln);
            if (length(diff) > 0.1f) ri = -4;
            else if (dot(wn, rn) < 0.8f) ri = -5;
            else {
              const F3 P = a.pyr.COV[0][p];
              const double sig = rn.x * rn.x * P.x + rn.y * rn.y * P.y + rn.z * rn.z * P.z;
              const double e = sqrt(1.0 / sig) * dot(rn, diff);
              if (fabs(e) > a.threshold) ri = -4;
              else { ri = 1; ei = (float)e; }
            }
          }
        }
      }
    }
    if (a.use_rgb) {
      // rendered live vertex -> depth relative to T_w_r -> vertex
      const F3 vl = (a.obj_label < 0 || a.llabel[p] == a.obj_label) ? a.lvert[p] : mk3(0.f);
      const float d = vl.z > 0.0 ? xform(a.inv_T_w_r, vl).z : 0.f;
      const F3 ref = d > 0 ? d * rotate(a.invK, mk3((float)x, (float)y, 1.f)) : mk3(0.f);
      const F3 live = a.pyr.V[a.cur][0][p];
      if (ref.z <= 0.f || ref.z == INVALIDF) {
        rr = -1;
      } else if (length(ref - live) > 0.1f && live.z > 0.f) {
        rr = -5;
      } else {
        const F3 w_vertex = xform(a.T_w_l, ref);
        const F3 r_vertex = xform(a.inv_T_w_r, w_vertex);
        const F3 proj = rotate(a.K, r_vertex);
        const float px = proj.x / proj.z, py = proj.y / proj.z;
        if (px < 1 || px > (float)(unsigned)(a.W - 2) || py < 1 || py > (float)(unsigned)(a.H - 2) ||
            isnan(px) || isnan(py)) {
          rr = -2;
        } else {
          const float residual = a.pyr.I[a.cur][0][p] - bil(a.pyr.I[1 - a.cur][0], a.W, px, py);
          const double e = (1.0 / a.sigma_bright) * residual;
          if (fabs(e) > a.threshold) rr = -4;
          else { rr = 1; er = (float)e; }
        }
      }
    }
  }
  a.res[p] = ri; a.res[n + p] = rr;
  if (a.err) { a.err[p] = ei; a.err[n + p] = er; }
  if (a.obj_label >= 0) return;
  // check_static_state: an object pixel of the live render is an inlier when
  // its rows' results are > -3
  const int l = a.llabel[p];
  bool inl;
  if (a.use_icp && a.use_rgb) inl = ri > -3 && rr > -3;
  else if (a.use_icp) inl = ri > -3;
  else inl = a.use_rgb && rr > -3;
  // one atomic per warp and label: 31 -> 12 us at 640x480 (one per pixel, all
  // of an object's on the same two words, was a serial chain in L2)
  const int mine = p0 < n && l >= 1 && l < 32 ? l : 0;
  for (unsigned left = __ballot_sync(0xffffffffu, mine); left;) {
    const int lab = __shfl_sync(0xffffffffu, mine, __ffs(left) - 1);
    const unsigned m = __ballot_sync(0xffffffffu, mine == lab);
    const unsigned in = __ballot_sync(0xffffffffu, mine == lab && inl);
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(a.count + lab, __popc(m));
      if (in) atomicAdd(a.count + 32 + lab, __popc(in));
    }
    left &= ~m;
  }
}

// Object::refine_mask_use_motion (object/object.cpp:255-315, outliers not
// absorbed into the background): inside the band, pixels whose ICP row is -4
// or -6, or whose photometric row is below -3, leave the object's mask.
__global__ void refine_mask_kernel(float* __restrict__ mask, const int8_t* __restrict__ res,
                                   int n, int use_icp, int use_rgb) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n || !(mask[p] >= 0)) return;
  if (use_icp && (res[p] == -4 || res[p] == -6)) { mask[p] = -1; return; }
  if (use_rgb && res[n + p] < -3) mask[p] = -1;
}

// Object::static_object, object.cpp:326: classes that never move (tv 63,
// and 69, 70)
static bool never_moving_class(int c) { return c == 63 || c == 69 || c == 70; }

int motion_residuals(Context* ctx, float threshold, float moved, float* ratio,
                     uint32_t* moving) {
  if (!ctx->track || !ctx->track->have_ref) {
    ctx->last_error = "mf_motion_residuals: needs a reference frame and a tracked live frame";
    return MF_E_STATE;
  }
  TrackState& T = *ctx->track;
  const size_t WH = (size_t)ctx->W * ctx->H;
  if (!T.d_mres) {
    MF_CUDA(cudaMalloc(&T.d_mres, 2 * WH));
    T.allocs.push_back(T.d_mres);
    MF_CUDA(cudaMalloc(&T.d_merr, sizeof(float) * 2 * WH));
    T.allocs.push_back(T.d_merr);
    MF_CUDA(cudaMalloc(&T.d_lvert, sizeof(F3) * WH));
    T.allocs.push_back(T.d_lvert);
    MF_CUDA(cudaMalloc(&T.d_lnorm, sizeof(F3) * WH));
    T.allocs.push_back(T.d_lnorm);
    MF_CUDA(cudaMalloc(&T.d_llabel, sizeof(int) * WH));
    T.allocs.push_back(T.d_llabel);
    MF_CUDA(cudaMalloc(&T.d_mcount, sizeof(int) * 64));
    T.allocs.push_back(T.d_mcount);
    // like the reference's persistent render buffers, the maps start zeroed
    // and keep what a later raycast does not overwrite
    MF_CUDA(cudaMemsetAsync(T.d_lvert, 0, sizeof(F3) * WH, ctx->stream));
    MF_CUDA(cudaMemsetAsync(T.d_lnorm, 0, sizeof(F3) * WH, ctx->stream));
    MF_CUDA(cudaMemsetAsync(T.d_llabel, 0, sizeof(int) * WH, ctx->stream));
  }
  // the model raycast at the live pose, objects at their last poses
  // (kfusion.cpp:291-296)
  IdList all;
  all.n = (int)ctx->inst.size();
  for (int i = 0; i < all.n; ++i) all.v[i] = i;
  if (int rc = stage_prepare(ctx, all)) return rc;
  if (int rc = stage_raycast_to(ctx, all, ctx->ray_epsilon, T.d_lvert, T.d_lnorm, T.d_llabel))
    return rc;
  float Tl[16], Tr[16];
  MF_CUDA(cudaMemcpyAsync(Tl, ctx->d_Twc, 64, cudaMemcpyDeviceToHost, ctx->stream));
  MF_CUDA(cudaMemcpyAsync(Tr, T.d_Twc_prev, 64, cudaMemcpyDeviceToHost, ctx->stream));
  MF_CUDA(cudaMemsetAsync(T.d_mcount, 0, sizeof(int) * 64, ctx->stream));
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  if (int rc = track_waited(ctx)) return rc;
  const mf_config& c = ctx->cfg;
  const F4 k{c.k[0], c.k[1], c.k[2], c.k[3]};
  MotionArgs a;
  a.pyr = T.pyr;
  a.cur = T.cur;
  a.W = ctx->W;
  a.H = ctx->H;
  a.mvertex = ctx->d_vertex;
  a.mnormal = ctx->d_normal;
  a.mlabel = ctx->d_label;
  a.lvert = T.d_lvert;
  a.llabel = T.d_llabel;
  a.obj_label = -1;
  a.T_w_l = load_m4(Tl);
  a.T_w_r = load_m4(Tr);
  a.inv_T_w_r = inverse(a.T_w_r);
  a.K = camera_matrix(k);
  a.invK = inverse_camera_matrix(k);
  a.sigma_bright = (float)(sqrtf(100.0f) / 255.0);  // tracking.cpp:766-772
  a.threshold = threshold;
  a.use_icp = c.use_icp;
  a.use_rgb = c.use_rgb;
  a.res = T.d_mres;
  a.err = T.d_merr;
  a.count = T.d_mcount;
  motion_residual_kernel<<<div_up((long long)WH, 256), 256, 0, ctx->stream>>>(a);
  MF_CUDA(cudaGetLastError());
  int cnt[64];
  MF_CUDA(cudaMemcpyAsync(cnt, T.d_mcount, sizeof(cnt), cudaMemcpyDeviceToHost, ctx->stream));
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  // kfusion.cpp:312-338: an object in view (with pixels in the live render)
  // moves when move-out threshold 0.05 < inliers / pixels < `moved` and its
  // class is not one of the never-moving classes (Object::static_object)
  uint32_t mv = 0;
  for (int i = 0; i < (int)ctx->inst.size(); ++i) {
    const int l = ctx->inst[i].label;
    float r = -1.f;
    if (i >= 1 && l >= 1 && l < 32 && cnt[l] > 0) {
      r = static_cast<float>(cnt[32 + l]) / (cnt[l]);
      if (r < moved && r > 0.05f && !never_moving_class(ctx->inst[i].class_id)) mv |= 1u << l;
    }
    if (ratio) ratio[i] = r;
  }
  if (moving) *moving = mv;
  return MF_OK;
}

// kfusion.cpp:446-466: a moving object's result rows recomputed after its
// tracking, Tracking::compute_residuals at the object's virtual camera pose
// (tracking.cpp:696) against its own model maps (m_vertex / m_normal: its
// pixels of the last frame's composite maps) and its pixels of the live
// raycast (m_vertex_bef_integ, the raycast at the current camera pose and the
// objects' new poses, i.e. the last mf_motion_residuals).  Rows (2 x W*H
// int8) to d_rows; the virtual pose (16 floats) to T_virtual when given.
int object_residuals(Context* ctx, int i, float threshold, int8_t* d_rows, float* T_virtual) {
  TrackState* T = ctx->track;
  if (!T || !T->have_ref || !T->d_mres || T->slot_kind[i] != 1) {
    ctx->last_error = "mf_object_residuals: needs the object tracked (mf_track_objects) and "
                      "the live raycast of mf_motion_residuals";
    return MF_E_STATE;
  }
  GNState S;
  MF_CUDA(cudaMemcpyAsync(&S, T->d_state + i, sizeof(GNState), cudaMemcpyDeviceToHost,
                          ctx->stream));
  float Tr[16];
  MF_CUDA(cudaMemcpyAsync(Tr, T->d_Twc_prev, 64, cudaMemcpyDeviceToHost, ctx->stream));
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  if (int rc = track_waited(ctx)) return rc;
  const mf_config& c = ctx->cfg;
  const F4 k{c.k[0], c.k[1], c.k[2], c.k[3]};
  MotionArgs a;
  a.pyr = T->pyr;
  a.cur = T->cur;
  a.W = ctx->W;
  a.H = ctx->H;
  a.mvertex = ctx->d_vertex;
  a.mnormal = ctx->d_normal;
  a.mlabel = ctx->d_label;
  a.lvert = T->d_lvert;
  a.llabel = T->d_llabel;
  a.obj_label = ctx->inst[i].label;
  a.T_w_l = S.T_virtual;
  a.T_w_r = load_m4(Tr);
  a.inv_T_w_r = inverse(a.T_w_r);
  a.K = camera_matrix(k);
  a.invK = inverse_camera_matrix(k);
  a.sigma_bright = (float)(sqrtf(100.0f) / 255.0);  // tracking.cpp:766-772
  a.threshold = threshold;
  a.use_icp = c.use_icp;
  a.use_rgb = c.use_rgb;
  a.res = d_rows;
  a.err = nullptr;
  a.count = nullptr;
  const size_t WH = (size_t)ctx->W * ctx->H;
  motion_residual_kernel<<<div_up((long long)WH, 256), 256, 0, ctx->stream>>>(a);
  MF_CUDA(cudaGetLastError());
  if (T_virtual) store_m4(T_virtual, S.T_virtual);
  return MF_OK;
}

int motion_download(Context* ctx, int8_t* res, float* err, float* lvert, int32_t* llabel) {
  TrackState* T = ctx->track;
  if (!T || !T->d_mres) {
    ctx->last_error = "mf_motion_download: no motion residuals yet";
    return MF_E_STATE;
  }
  const size_t WH = (size_t)ctx->W * ctx->H;
  if (res) MF_CUDA(cudaMemcpyAsync(res, T->d_mres, 2 * WH, cudaMemcpyDeviceToHost, ctx->stream));
  if (err)
    MF_CUDA(cudaMemcpyAsync(err, T->d_merr, sizeof(float) * 2 * WH, cudaMemcpyDeviceToHost,
                            ctx->stream));
  if (lvert)
    MF_CUDA(cudaMemcpyAsync(lvert, T->d_lvert, sizeof(F3) * WH, cudaMemcpyDeviceToHost,
                            ctx->stream));
  if (llabel)
    MF_CUDA(cudaMemcpyAsync(llabel, T->d_llabel, sizeof(int) * WH, cudaMemcpyDeviceToHost,
                            ctx->stream));
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  return MF_OK;
}

// The result codes of problem `slot`'s rows at level 0, evaluated at the pose
// of its last level-0 GN iteration: Tracking::trackingResult_[0] after
// trackLiveFrame / trackEachObject, which kfusion.cpp:282-283 and :397-405
// copy into Object::trackresult_.  ICP rows first, then photometric rows; a
// term that is switched off leaves 0.
__global__ void row_codes_kernel(GNArgs a, int slot, int8_t* __restrict__ out,
                                 float* __restrict__ out_err) {
  // The problem's constants (all but the sums) in shared memory, copied by the
  // whole CTA, and the inverse of the evaluated pose by one warp: with one
  // thread copying and inverting, that prologue was 50 of the kernel's 57 us at
  // 637x479.  The rows themselves are two gathers per pixel, latency-bound.
  __shared__ GNState S;
  {
    const int* src = reinterpret_cast<const int*>(&a.st[slot]);
    int* dst = reinterpret_cast<int*>(&S);
    for (int i = threadIdx.x; i < (int)(offsetof(GNState, sums) / 4); i += blockDim.x)
      dst[i] = src[i];
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    const float* eval = reinterpret_cast<const float*>(&S.evalTf);
    const float ie = inverse_warp(eval, lane);
    if (lane < 16) {
      reinterpret_cast<float*>(&S.Tf)[lane] = eval[lane];
      reinterpret_cast<float*>(&S.invTf)[lane] = ie;
    }
  }
  __syncthreads();
  const GNView lv = gn_view(a, 0);
  const int n = lv.w * lv.h;
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  Row ri, rr;
  if (S.kind == 0) gn_rows<0>(a, lv, S, a.rV[0][slot], 0, p, ri, rr);
  else gn_rows<1>(a, lv, S, a.rV[0][slot], 0, p, ri, rr);
  const int8_t ci = a.use_icp ? (int8_t)ri.result : 0, cr = a.use_rgb ? (int8_t)rr.result : 0;
  const float ei = ci == 1 ? ri.e : 0.f, er = cr == 1 ? rr.e : 0.f;  // TrackData::error
  out[p] = ci;
  out[n + p] = cr;
  if (out_err) {
    out_err[p] = ei;
    out_err[n + p] = er;
  }
}

int track_results(Context* ctx, int slot, int8_t* d_out, float* d_err, float* pose_eval) {
  if (!ctx->track || !ctx->track->have_ref) {
    ctx->last_error = "mf_track_results: no tracking has run";
    return MF_E_STATE;
  }
  const int n = ctx->W * ctx->H;
  GNArgs a = make_args(ctx);
  row_codes_kernel<<<div_up(n, 256), 256, 0, ctx->stream>>>(a, slot, d_out, d_err);
  MF_CUDA(cudaGetLastError());
  if (pose_eval) {
    static_assert(sizeof(M4) == 64, "M4 is 16 row-major floats");
    MF_CUDA(cudaMemcpyAsync(pose_eval, &ctx->track->d_state[slot].evalTf, sizeof(M4),
                            cudaMemcpyDeviceToHost, ctx->stream));
    MF_CUDA(cudaStreamSynchronize(ctx->stream));
    return track_waited(ctx);
  }
  return MF_OK;
}

int refine_mask_use_motion(Context* ctx, int id, const int8_t* d_res, int use_icp, int use_rgb) {
  TrackState* T = ctx->track;
  if (!d_res) {
    if (!T || !T->d_mres) {
      ctx->last_error = "mf_refine_mask_use_motion: no motion residuals yet";
      return MF_E_STATE;
    }
    d_res = T->d_mres;
  }
  const int n = ctx->W * ctx->H;
  refine_mask_kernel<<<div_up(n, 256), 256, 0, ctx->stream>>>(ctx->d_masks + (size_t)id * n,
                                                              d_res, n, use_icp, use_rgb);
  MF_CUDA(cudaGetLastError());
  return MF_OK;
}


// The planes of the last mf_motion_residuals (for renders), or MF_E_STATE.
int motion_planes(Context* ctx, const int8_t** res, const float** err) {
  if (!ctx->track || !ctx->track->d_mres) {
    ctx->last_error = "no motion residuals yet";
    return MF_E_STATE;
  }
  *res = ctx->track->d_mres;
  *err = ctx->track->d_merr;
  return MF_OK;
}

}  // namespace mf
