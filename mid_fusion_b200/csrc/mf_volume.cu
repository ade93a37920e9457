// Voxel-block allocation and projective TSDF integration on the device.
//
// Allocation is sort-free: each octree level is a dense table indexed by the
// Morton code of its octants, so the reference's sort + unique_multiscale +
// level-by-level updateLevel (lib/octree.hpp:761-863) becomes (1) every ray
// sample of an unallocated block adds to that table entry's request count and
// (2) one pass over the block table creates the requested blocks and flags their
// ancestors.  The resulting key sets and topology equal the reference's; the
// request counts also reproduce the reference's allocation-list quirks (see
// alloc_commit_kernel).
#include <algorithm>
#include <climits>
#include <cstdio>
#include <cstring>
#include "mf_internal.h"
#include "mf_sample.cuh"
#include "mf_warp.cuh"

namespace mf {

// ------------------------------------------------------------------ prepare
// Per-instance matrices every stage needs, computed from the device-resident
// camera and volume poses with the reference's float operation order.
// One block per instance, one warp per inverse: the three 4x4 eliminations and
// the products run on lanes, side by side (one thread per instance took 10 us
// for them, on the frame's critical path; now 3).  `reset`: the allocation and
// the visit list that follow start from zeroed counters (each memset node of a
// frame's graph cost 4 us, two per instance).
__global__ void __launch_bounds__(96)
prepare_kernel(const float* __restrict__ Twc_p, const float* __restrict__ Two_p,
               const Volume* __restrict__ vols, InstFrame* __restrict__ out, F4 k, float mu,
               IdList ids, const unsigned long long* __restrict__ reserved,
               const int* __restrict__ labels, int reset, int* __restrict__ visit_count) {
  __shared__ InstFrame f;
  __shared__ M4 A[3], I[3], iK;   // T_w_o, K, T_w_c; their inverses; K's closed-form inverse
  const int i = ids.v[blockIdx.x];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Volume& V = vols[i];
  const float vs = V.dim / V.size;
  auto at = [](M4& m) { return reinterpret_cast<float*>(&m); };
  if (warp == 0 && lane < 16) at(A[0])[lane] = Two_p[16 * i + lane];
  if (warp == 2 && lane < 16) at(A[2])[lane] = Twc_p[lane];
  if (warp == 1 && lane == 0) {
    A[1] = camera_matrix(k);
    iK = inverse_camera_matrix(k);
    f.inv_voxel = 1 / vs;
    f.band = 2 * mu;
    f.num_steps = (int)ceilf(f.band * f.inv_voxel);
    f.reserved = reserved[i];
    f.label = labels[i];
    if (reset) {
      *V.last_emit = 0;
      *V.emit_total = 0;
      if (blockIdx.x == 0) *visit_count = 0;
    }
  }
  __syncthreads();
  {
    const float e = inverse_warp(at(A[warp]), lane);
    if (lane < 16) at(I[warp])[lane] = e;
  }
  __syncthreads();
  if (warp == 0) {
    const float kp = mul_warp(at(A[2]), at(I[1]), lane);
    if (lane < 16) {
      at(f.T_w_o)[lane] = at(A[0])[lane];
      at(f.inv_T_w_o)[lane] = at(I[0])[lane];
      at(f.kPose)[lane] = kp;
    }
    if (lane == 0) f.o_cam = xform(I[0], get_translation(A[2]));
  } else if (warp == 1) {
    const float c = mul_warp(at(I[2]), at(A[0]), lane);
    if (lane < 16) at(f.Tcw)[lane] = c;
    __syncwarp();
    const float kc = mul_warp(at(A[1]), at(f.Tcw), lane);
    if (lane < 16) at(f.KTcw)[lane] = kc;
    if (lane == 0) {
      f.delta = rotate(f.Tcw, mk3(vs, 0, 0));
      f.cam_delta = rotate(A[1], f.delta);
    }
  } else {
    const float w = mul_warp(at(A[2]), at(iK), lane);
    if (lane < 16) at(f.view)[lane] = w;
    __syncwarp();
    if (lane == 0) f.o_origin = xform(I[0], get_translation(f.view));
  }
  __syncthreads();
  for (int w = threadIdx.x; w < (int)(sizeof(InstFrame) / 4); w += 96)
    reinterpret_cast<int*>(out + i)[w] = reinterpret_cast<const int*>(&f)[w];
}

// ------------------------------------------------------------------ allocation
// buildVolumeAllocationList, apps/kfusion/src/cpp/kfusion/alloc_impl.hpp:121-191.
// One thread per ray-casting (pixel, instance).  A sample in an allocated
// block marks it active; a sample in an unallocated block adds to that block's
// request count (runs of equal blocks along a ray are added at once).  The
// emission order of the single-threaded reference (row, column, step) of the
// thread's last emitted sample is folded into last_emit with atomicMax.
// Bound by instruction issue.  Background 512^3 and three objects 256^3 at
// 640x480, all four in one launch: 116 us with 64-bit indices and the slot
// waited for on entry, 71 us with 32-bit ones and the slot looked at when the
// block is left, now 46 (the objects' long rays launched first).
constexpr int RUN_SHIFT = 27;                          // table indices are below 2^27
constexpr uint32_t RUN_INDEX = (1u << RUN_SHIFT) - 1;
// A step is half a voxel to a voxel long, so a run through a block (8 sqrt 3
// voxels) has at most 29 samples, and 24 samples leave at most 3 * (24 / 8 + 1)
// blocks, one more at the ray's end.
constexpr int MARK_STEPS = 24, RUN_LIST = 14;
__global__ void __launch_bounds__(256)
alloc_mark_kernel(const float* __restrict__ depth, const float* __restrict__ masks, int W,
                  int H, const Volume* __restrict__ vols, const InstFrame* __restrict__ frames,
                  IdList ids, Pool pool) {
  // the objects' long rays first: the background's short ones fill the tail
  const int inst = ids.v[gridDim.y - 1 - blockIdx.y];
  const Volume& V = vols[inst];
  const InstFrame& F = frames[inst];
  unsigned count = 0, last_order = 0, last_idx = 0;
  // The CTA's pixels that cast a ray (depth != 0, mask >= 0) are packed, in
  // pixel order, onto its first threads: an object's pixels are sparse, and a
  // ray of 100 samples on one lane of a warp idled the other 31.  Every result
  // below is a sum, a maximum or an idempotent flag, so which thread handles
  // which pixel does not change it.
  __shared__ int s_pix[256];
  __shared__ float s_d[256];
  __shared__ int s_wn[8];
  __shared__ uint32_t s_spread[512];   // spread3_10 of a block coordinate
  __shared__ uint32_t s_list[RUN_LIST][256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < (V.size >> 3); i += 256) s_spread[i] = spread3_10(i);
  {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const float dq = q < W * H ? depth[q] : 0.f;
    const bool ray = dq != 0 && !(masks[(size_t)inst * W * H + (q < W * H ? q : 0)] < 0);
    const unsigned b = __ballot_sync(0xffffffffu, ray);
    if (lane == 0) s_wn[warp] = __popc(b);
    __syncthreads();
    int base = 0;
    for (int w = 0; w < warp; ++w) base += s_wn[w];
    if (ray) {
      const int slot = base + __popc(b & ((1u << lane) - 1u));
      s_pix[slot] = q;
      s_d[slot] = dq;
    }
    __syncthreads();
  }
  int n_rays = 0;
  for (int w = 0; w < 8; ++w) n_rays += s_wn[w];
  const bool has_ray = (int)threadIdx.x < n_rays;
  const int p = has_ray ? s_pix[threadIdx.x] : 0;
  const float d = has_ray ? s_d[threadIdx.x] : 0.f;
  // no early return: every lane reaches the warp-wide steps below
  const int32_t* __restrict__ tab = V.block_tab;   // not written by this kernel
  uint32_t* __restrict__ req = V.req;
  uint8_t* __restrict__ active = pool.active;
  const float inv_voxel = F.inv_voxel, size_f = (float)(unsigned)V.size;
  const int num_steps = F.num_steps;
  F3 pos = mk3(0.f), step = mk3(0.f);
  bool all_in = false;
  if (has_ray) {
    const unsigned x = p % W, y = p / W;
    const F3 w_vertex = xform(F.kPose, mk3((x + 0.5f) * d, (y + 0.5f) * d, d));
    const F3 o_vertex = xform(F.inv_T_w_o, w_vertex);
    const F3 direction = normalize(F.o_cam - o_vertex);
    pos = o_vertex - (F.band * 0.5f) * direction;
    step = (direction * F.band) / (float)num_steps;
    // both ends at least two voxels inside: so is every sample (the sums'
    // rounding stays far below a voxel over 4096 steps)
    const F3 end = pos + (float)num_steps * step;
    const float lo = 2.f, hi = size_f - 2.f;
    auto inside = [&](F3 q) {
      const float fx = q.x * inv_voxel, fy = q.y * inv_voxel, fz = q.z * inv_voxel;
      return fx > lo && fx < hi && fy > lo && fy < hi && fz > lo && fz < hi;
    };
    all_in = num_steps <= 4096 && inside(pos) && inside(end);
  }
  // The march lists the blocks it leaves (samples << 27 | table index, in shared
  // memory), MARK_STEPS samples at a time; the warp then looks the listed blocks
  // up together.  A lookup inside the march made the warp wait for it at nearly
  // every step, because some lane enters a block there.
  uint32_t key = 0, bidx = 0;   // keys start at BIG_BITS
  int run = 0, n_list = 0, order = 0;   // order: step of the next listed sample
  // floor(f / 8) of 0 <= f < 4096 in the low bits: with rounding towards minus
  // infinity the sum's last place is 8 (a truncating conversion runs at a
  // quarter of the rate)
  constexpr float BIG = 100663296.f;   // 2^26 + 2^25
  constexpr uint32_t BIG_BITS = 0x4cc00000u;
  auto sample = [&](int i, float fx, float fy, float fz) {
    const uint32_t kx = __float_as_uint(__fadd_rd(fx, BIG)), ky = __float_as_uint(__fadd_rd(fy, BIG)),
                   kz = __float_as_uint(__fadd_rd(fz, BIG));
    const uint32_t k = kx + (ky << 10) + (kz << 20);
    if (k != key) {
      if (run) s_list[n_list++][threadIdx.x] = ((uint32_t)run << RUN_SHIFT) | bidx;
      else order = i;
      key = k;
      bidx = s_spread[kx - BIG_BITS] | (s_spread[ky - BIG_BITS] << 1) |
             (s_spread[kz - BIG_BITS] << 2);
      run = 0;
    }
    ++run;
  };
  const int steps = __any_sync(0xffffffffu, has_ray) ? num_steps : 0;
  for (int i0 = 0; i0 < steps; i0 += MARK_STEPS) {
    const int i1 = min(i0 + MARK_STEPS, steps);
    if (has_ray) {
      if (all_in) {
        for (int i = i0; i < i1; i++) {
          sample(i, pos.x * inv_voxel, pos.y * inv_voxel, pos.z * inv_voxel);
          pos = pos + step;
        }
      } else {
        for (int i = i0; i < i1; i++) {
          // the reference floors pos / voxel and tests 0 <= floor < size; with an
          // integer size that holds exactly when 0 <= pos / voxel < size (NaN
          // fails the test either way).  The samples inside are consecutive:
          // the positions are monotone along every axis.
          const float fx = pos.x * inv_voxel, fy = pos.y * inv_voxel, fz = pos.z * inv_voxel;
          if (fx < size_f && fy < size_f && fz < size_f && fx >= 0 && fy >= 0 && fz >= 0)
            sample(i, fx, fy, fz);
          pos = pos + step;
        }
      }
      if (i1 == steps && run)
        s_list[n_list++][threadIdx.x] = ((uint32_t)run << RUN_SHIFT) | bidx;
    }
    const int n_max = __reduce_max_sync(0xffffffffu, n_list);
    for (int e = 0; e < n_max; e += 4) {
      uint32_t ent[4];
      int slot[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        ent[u] = e + u < n_list ? s_list[e + u][threadIdx.x] : 0;   // 0: no samples
        slot[u] = ent[u] ? __ldg(tab + (ent[u] & RUN_INDEX)) : 0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t n = ent[u] >> RUN_SHIFT;
        order += n;
        if (ent[u] && slot[u] >= 0) active[slot[u]] = 1;
        if (slot[u] < 0) {
          last_idx = ent[u] & RUN_INDEX;
          last_order = (unsigned)p * (unsigned)num_steps + (unsigned)(order - 1);
          atomicAdd(&req[last_idx], n);
          count += n;
        }
      }
    }
    n_list = 0;
  }
  // one emission-count and one last-emission atomic per warp
  unsigned long long last = count ? (((unsigned long long)last_order << 32) | last_idx) : 0ULL;
  unsigned long long tot = count;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    tot += __shfl_xor_sync(0xffffffffu, tot, o);
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, last, o);
    last = other > last ? other : last;
  }
  if ((threadIdx.x & 31) == 0 && tot) {
    atomicAdd(V.emit_total, tot);
    atomicMax(V.last_emit, last);
  }
}

// Grows the instance's box of allocated blocks (read by the raycast to skip
// rays that cannot meet a block); block 0 is left out, the raycast tests it on
// its own.
__device__ __forceinline__ void note_block(const Volume& V, long long bidx, int cx, int cy,
                                           int cz) {
  if (bidx == 0) return;
  atomicMin(&V.bbox[0], cx); atomicMin(&V.bbox[1], cy); atomicMin(&V.bbox[2], cz);
  atomicMax(&V.bbox[3], cx); atomicMax(&V.bbox[4], cy); atomicMax(&V.bbox[5], cz);
}

// Octree::alloc_update + updateLevel, lib/octree.hpp:761-786, :826-863.
// One thread per (block-table entry, instance).  Reference semantics kept:
//  - the list's slot 0 is never written (alloc_impl.hpp:175, pre-increment) and
//    stays 0, and unique_multiscale keeps keys[0] unconditionally
//    (lib/algorithms/unique.hpp:76-79), so the path to block (0,0,0) is
//    allocated by every call;
//  - [0, count) is passed on while the keys sit in slots 1..count, so the last
//    emitted key is not allocated unless another sample requested its block.
__global__ void __launch_bounds__(256)
alloc_commit_kernel(const Volume* __restrict__ vols, const InstFrame* __restrict__ frames,
                    IdList ids, Pool pool, int* __restrict__ status) {
  const int inst = ids.v[blockIdx.y];
  const Volume& V = vols[inst];
  const long long n_tab = 1LL << (3 * V.block_level);
  const long long bidx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (bidx >= n_tab) return;
  const uint32_t r = V.req[bidx];
  if (r == 0 && bidx != 0) return;
  const unsigned long long total = *V.emit_total;
  const unsigned long long last = *V.last_emit;
  bool need = (r > 0) || (bidx == 0);
  if (total >= frames[inst].reserved) {
    if (bidx == 0) atomicOr(status, ST_ALLOC_OVERFLOW);
  } else if (r == 1 && bidx != 0 && (long long)(last & 0xffffffffULL) == bidx) {
    need = false;  // the dropped last slot was this block's only request
  }
  if (need && V.block_tab[bidx] < 0) {
    const int slot = atomicAdd(pool.count, 1);
    if (slot >= pool.cap) {
      atomicOr(status, ST_POOL_FULL);
    } else {
      const int cx = (int)gather3((uint64_t)bidx) << 3;
      const int cy = (int)gather3((uint64_t)bidx >> 1) << 3;
      const int cz = (int)gather3((uint64_t)bidx >> 2) << 3;
      pool.meta[slot] = make_int4(cx, cy, cz, inst);
      pool.active[slot] = 1;
      V.block_tab[bidx] = slot;
      note_block(V, bidx, cx, cy, cz);
      for (int l = V.block_level - 1; l >= 1; --l)
        V.node_tab[V.node_off[l] + (bidx >> (3 * (V.block_level - l)))] = 1;
    }
  }
  if (r) V.req[bidx] = 0;
}

// Octree::alloc_update on caller-supplied keys: (code, level) pairs already
// reduced on the host to "create the octant at this level and its ancestors".
__global__ void alloc_keys_kernel(const Volume* __restrict__ vols, int inst,
                                  const unsigned long long* __restrict__ codes,
                                  const int* __restrict__ levels, int n, Pool pool,
                                  int* __restrict__ status) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const Volume& V = vols[inst];
  const int L = levels[t];
  const unsigned long long code = codes[t];
  for (int l = 1; l <= L && l < V.block_level; ++l)
    V.node_tab[V.node_off[l] + (long long)(code >> (3 * (V.max_level - l)))] = 1;
  if (L == V.block_level) {
    const long long bidx = (long long)(code >> (3 * (V.max_level - V.block_level)));
    if (atomicCAS(&V.block_tab[bidx], -1, -2) == -1) {
      const int slot = atomicAdd(pool.count, 1);
      if (slot >= pool.cap) {
        atomicOr(status, ST_POOL_FULL);
        V.block_tab[bidx] = -1;
        return;
      }
      const int cx = (int)gather3(bidx) << 3, cy = (int)gather3(bidx >> 1) << 3,
                cz = (int)gather3(bidx >> 2) << 3;
      pool.meta[slot] = make_int4(cx, cy, cz, inst);
      pool.active[slot] = 1;
      V.block_tab[bidx] = slot;
      note_block(V, bidx, cx, cy, cz);
    }
  }
}

// ------------------------------------------------------------------ integration
// projective_functor::build_active_list, lib/functors/projective_functor.hpp:54-71
// with algorithms::filter (lib/algorithms/filter.hpp:42-61, predicates ORed):
// a block is visited when it is active or its corner projects into the frame.
// clear: the integration that follows sets VoxelBlock::active_ anew; it is
// cleared here, so that each of its warps can set it without a barrier.
__global__ void __launch_bounds__(256)
visit_list_kernel(Pool pool, const Volume* __restrict__ vols,
                  const InstFrame* __restrict__ frames, uint32_t inst_mask, int W, int H,
                  int* __restrict__ visit, int* __restrict__ visit_count, int clear) {
  const int slot = blockIdx.x * blockDim.x + threadIdx.x;
  bool take = false;
  if (slot < min(*pool.count, pool.cap)) {   // the count runs on when the pool is full
    const int4 m = pool.meta[slot];
    // a slot that the other stream's allocation has counted but not written
    // yet (w < 0) belongs to that stream's instances
    if (m.w >= 0 && ((inst_mask >> m.w) & 1u)) {
      if (pool.active[slot]) {
        take = true;
      } else {
        const Volume& V = vols[m.w];
        const float vs = V.dim / V.size;
        const F3 bc = mk3((float)m.x, (float)m.y, (float)m.z) * vs;
        const F3 vc = xform(frames[m.w].KTcw, bc);
        const int px = (int)(vc.x / vc.z), py = (int)(vc.y / vc.z);
        take = px >= 0 && px < W && py >= 0 && py < H;
      }
    }
  }
  // warp-aggregated append
  const unsigned ballot = __ballot_sync(0xffffffffu, take);
  if (!ballot) return;
  const int lane = threadIdx.x & 31;
  int base = 0;
  if (lane == __ffs(ballot) - 1) base = atomicAdd(visit_count, __popc(ballot));
  base = __shfl_sync(0xffffffffu, base, __ffs(ballot) - 1);
  if (take) {
    visit[base + __popc(ballot & ((1u << lane) - 1))] = slot;
    if (clear) pool.active[slot] = 0;
  }
}

struct SdfArgs {
  const float* depth; const F3* rgb; const float* masks;
  int W, H; float mu; float maxweight;
};

// sdf_update::operator(), apps/kfusion/src/cpp/kfusion/mapping_impl.hpp:17-49,
// on one voxel held as separate field references.
template <typename FT, typename FW, typename FC, typename FG, typename FWI>
__device__ __forceinline__ void sdf_update(const SdfArgs& a, const float* mask, F3 pos,
                                           float px_f, float py_f, FT& tsdf, FW& wt,
                                           float* r, float* g, float* b, FC& c, FG& fg,
                                           FWI& w) {
  const unsigned px = (unsigned)px_f, py = (unsigned)py_f;
  const float depthSample = a.depth[px + a.W * py];
  const float m = mask[px + a.W * py];
  if (depthSample <= 0 || m < 0) return;
  const float diff =
      (depthSample - pos.z) * sqrtf(1 + sq(pos.x / pos.z) + sq(pos.y / pos.z));
  if (diff > -a.mu) {
    const float sdf = fmn(1.f, diff / a.mu);
    float x = tsdf, y = wt;
    x = clampf((y * x + sdf) / (y + 1), -1.f, 1.f);
    y = fmn(y + 1, a.maxweight);
    tsdf = x; wt = y;
    const F3 rgb = a.rgb[px + a.W * py];
    const int cc = c;
    *r = (rgb.x + *r * cc) / (cc + 1);
    *g = (rgb.y + *g * cc) / (cc + 1);
    *b = (rgb.z + *b * cc) / (cc + 1);
    c = cc + 1;
    const int ww = w;
    fg = ((double)m + fg * ww) / (ww + 1);
    w = ww + 1;
  }
}

// Hint: bring the 36 128-byte lines holding the eight fields of this warp's
// 128 voxels (from v0 on) of pool slot `slot` into L2.
__device__ __forceinline__ void prefetch_fields(const Pool& pool, int slot, int v0, int lane) {
  const size_t o = (size_t)slot * 512 + v0;
  const int f = lane >> 2;
  const void* base = f == 0   ? (const void*)(pool.tsdf + o)
                     : f == 1 ? (const void*)(pool.wt + o)
                     : f == 2 ? (const void*)(pool.r + o)
                     : f == 3 ? (const void*)(pool.g + o)
                     : f == 4 ? (const void*)(pool.b + o)
                     : f == 5 ? (const void*)(pool.c + o)
                     : f == 6 ? (const void*)(pool.w + o)
                              : (const void*)(pool.fg + o);
  const char* p = (const char*)base + (lane & 3) * 128;
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
  if (f == 7) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + 512));
}

// projective_functor::update_block, lib/functors/projective_functor.hpp:73-111.
// A warp takes a quarter of a visited block (two z layers), four neighbouring
// voxels of a row per thread: the row's transforms are computed once for the
// four, their depth and mask fetches are in flight together, and every field
// plane is read and written 16 bytes at a time, only where one of the four
// passes the update test.  Warps never wait for each other
// (VoxelBlock::active_ is cleared by the visit list and set by any warp that
// sees a voxel).  The next block's slot and corner are loaded during the
// current one; the instances' constants come from shared memory.
// Bound by instruction issue (seven divisions and a square root per updated
// voxel; the double one of the foreground mean is left out where the mean is
// 0 or 1 exactly, as for every voxel that one kind of mask has seen) and by
// the fields' traffic.  Background 512^3 and three objects 256^3 at 640x480:
// 98 us, 4.0 TB/s, issue slots 55 % busy (one voxel per thread and a barrier
// per block: 130 us, 65 %, half again as many instructions; without the barrier
// alone 131).  Registers bound the warps in flight: 4 CTAs per SM (64
// registers) beat 5 (48, spills) by 4 to 14 % and 3 (80) by 12 to 20 % from one
// object at 160x120 to six at 1280x720.
// Persistent: INT_CTAS CTAs per SM; with PF the warp prefetches its quarter of
// the next block's fields into L2 while it works on the current one (mostly no
// gain, since the loads wait for the pixels, not for DRAM).  Both forms update
// each voxel alike (int_variants).
constexpr int INT_THREADS = 256;  // two blocks per CTA
constexpr int INT_CTAS = 4;
template <bool PF>
__global__ void __launch_bounds__(INT_THREADS, INT_CTAS)
integrate_blocks_kernel(Pool pool, const Volume* __restrict__ vols,
                        const InstFrame* __restrict__ frames, SdfArgs args, F4 k,
                        const int* __restrict__ visit, const int* __restrict__ visit_count) {
  const int n = *visit_count;
  const M4 K = camera_matrix(k);
  const float wlim = args.W - 1.5f, hlim = args.H - 1.5f;
  const int W = args.W;
  const float mu = args.mu, maxweight = args.maxweight;
  // the instances' constants, staged once per CTA (the tables hold
  // MAX_INSTANCES entries)
  __shared__ M4 s_Tcw[MAX_INSTANCES];
  __shared__ F3 s_delta[MAX_INSTANCES], s_cdelta[MAX_INSTANCES];
  __shared__ float s_vs[MAX_INSTANCES];
  for (int i = threadIdx.x; i < MAX_INSTANCES; i += blockDim.x) {
    s_Tcw[i] = frames[i].Tcw;
    s_delta[i] = frames[i].delta;
    s_cdelta[i] = frames[i].cam_delta;
    s_vs[i] = vols[i].dim / vols[i].size;
  }
  __syncthreads();
  // four warps per block; the next block's corner is
  // fetched one block ahead and (PF) the slot after it two blocks ahead
  const int lane = threadIdx.x & 31;
  const int v = (threadIdx.x & 127) * 4;
  const int x0 = v & 7, y = (v >> 3) & 7, z = v >> 6;
  const int stride = INT_THREADS / 128 * gridDim.x;
  int item = (threadIdx.x >> 7) * gridDim.x + blockIdx.x;
  int next_slot = item < n ? visit[item] : 0;
  int4 next_m = item < n ? pool.meta[next_slot] : make_int4(0, 0, 0, 0);
  int after_slot = 0;
  if (PF && item + stride < n) after_slot = visit[item + stride];
  for (; item < n; item += stride) {
    const int slot = next_slot;
    const int4 m = next_m;
    if (item + stride < n) {
      if (PF) {
        prefetch_fields(pool, after_slot, v & ~127, lane);
        next_slot = after_slot;
        if (item + 2 * stride < n) after_slot = visit[item + 2 * stride];
      } else {
        next_slot = visit[item + stride];
      }
      next_m = pool.meta[next_slot];
    }
    const float vs = s_vs[m.w];
    const float* mask = args.masks + (size_t)m.w * args.W * args.H;
    // voxel -> pixel
    const F3 start = xform(s_Tcw[m.w], mk3(m.x * vs, (m.y + y) * vs, (m.z + z) * vs));
    const F3 camerastart = xform(K, start);
    const F3 delta = s_delta[m.w], cdelta = s_cdelta[m.w];
    int pix[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const F3 cv = camerastart + ((float)(x0 + i) * cdelta);
      pix[i] = -1;
      if (start.z + (float)(x0 + i) * delta.z >= 0.0001f) {
        const float inv = 1.f / cv.z;
        const float pxf = cv.x * inv + 0.5f, pyf = cv.y * inv + 0.5f;
        if (!(pxf < 0.5f || pxf > wlim || pyf < 0.5f || pyf > hlim))
          pix[i] = (int)((unsigned)pxf + W * (unsigned)pyf);
      }
    }
    const bool vis = (pix[0] & pix[1] & pix[2] & pix[3]) >= 0;
    if (__any_sync(0xffffffffu, vis) && lane == 0) pool.active[slot] = 1;
    // depth / mask at the pixel, the update test of sdf_update
    float depthS[4], mval[4], sdf[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      depthS[i] = pix[i] >= 0 ? __ldg(args.depth + pix[i]) : 0.f;
      mval[i] = pix[i] >= 0 ? __ldg(mask + pix[i]) : -1.f;
    }
    bool any = false;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      bool upd = false;
      if (depthS[i] > 0 && mval[i] >= 0) {
        const F3 pos = start + ((float)(x0 + i) * delta);
        const float diff =
            (depthS[i] - pos.z) * sqrtf(1 + sq(pos.x / pos.z) + sq(pos.y / pos.z));
        if (diff > -mu) {
          upd = true;
          sdf[i] = fmn(1.f, diff / mu);
        }
      }
      if (!upd) pix[i] = -1;
      any |= upd;
    }
    // read-modify-write of the voxels: sdf_update,
    // apps/kfusion/src/cpp/kfusion/mapping_impl.hpp:26-46
    if (any) {
      const size_t o = ((size_t)slot * 512 + v) / 4;
      float4 t4 = ((const float4*)pool.tsdf)[o], wt4 = ((const float4*)pool.wt)[o];
      float4 r4 = ((const float4*)pool.r)[o], g4 = ((const float4*)pool.g)[o],
             b4 = ((const float4*)pool.b)[o];
      int4 c4 = ((const int4*)pool.c)[o];
      int4 w4 = ((const int4*)pool.w)[o];
      float *t = &t4.x, *wt = &wt4.x, *r = &r4.x, *g = &g4.x, *b = &b4.x;
      int *c = &c4.x, *w = &w4.x;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (pix[i] >= 0) {
          const F3 rgb = args.rgb[pix[i]];
          t[i] = clampf((wt[i] * t[i] + sdf[i]) / (wt[i] + 1), -1.f, 1.f);
          wt[i] = fmn(wt[i] + 1, maxweight);
          const float cf = c[i], c1 = c[i] + 1;
          r[i] = (rgb.x + r[i] * cf) / c1;
          g[i] = (rgb.y + g[i] * cf) / c1;
          b[i] = (rgb.z + b[i] * cf) / c1;
          c[i] = c[i] + 1;
        }
      ((float4*)pool.tsdf)[o] = t4;
      ((float4*)pool.wt)[o] = wt4;
      ((float4*)pool.r)[o] = r4;
      ((float4*)pool.g)[o] = g4;
      ((float4*)pool.b)[o] = b4;
      ((int4*)pool.c)[o] = c4;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        double2 f2 = ((const double2*)pool.fg)[2 * o + h];
        double* f = &f2.x;
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (pix[2 * h + i] >= 0) {
            const int wi = w[2 * h + i];
            const double num = (double)mval[2 * h + i] + f[i] * wi, den = (double)(wi + 1);
            // den / den and +-0 / den of a positive den
            f[i] = wi >= 0 && num == den ? 1.0 : wi >= 0 && num == 0.0 ? num : num / den;
            w[2 * h + i] = wi + 1;
          }
        ((double2*)pool.fg)[2 * o + h] = f2;
      }
      ((int4*)pool.w)[o] = w4;
    }
    __syncwarp();
  }
}

// Work counts of update_block for the roofline: voxels whose pixel is read
// (visible: depth and mask fetched) and voxels updated (fields read + written).
__global__ void __launch_bounds__(256)
integrate_count_kernel(Pool pool, const Volume* __restrict__ vols,
                       const InstFrame* __restrict__ frames, SdfArgs args, F4 k,
                       const int* __restrict__ visit, const int* __restrict__ visit_count,
                       unsigned long long* __restrict__ counts) {
  const int n = *visit_count;
  const M4 K = camera_matrix(k);
  const float wlim = args.W - 1.5f, hlim = args.H - 1.5f;
  unsigned long long nvis = 0, nupd = 0;
  for (int item = blockIdx.x; item < n; item += gridDim.x) {
    const int slot = visit[item];
    const int4 m = pool.meta[slot];
    const Volume& V = vols[m.w];
    const InstFrame& F = frames[m.w];
    const float vs = V.dim / V.size;
    const float* mask = args.masks + (size_t)m.w * args.W * args.H;
    for (int h = 0; h < 2; ++h) {
      const int v = threadIdx.x + h * 256;
      const int x = v & 7, y = (v >> 3) & 7, z = v >> 6;
      const F3 start = xform(F.Tcw, mk3(m.x * vs, (m.y + y) * vs, (m.z + z) * vs));
      const F3 cv = xform(K, start) + ((float)x * F.cam_delta);
      const F3 p = start + ((float)x * F.delta);
      if (p.z < 0.0001f) continue;
      const float inv = 1.f / cv.z;
      const float pxf = cv.x * inv + 0.5f, pyf = cv.y * inv + 0.5f;
      if (pxf < 0.5f || pxf > wlim || pyf < 0.5f || pyf > hlim) continue;
      ++nvis;
      const int pix = (int)((unsigned)pxf + args.W * (unsigned)pyf);
      const float d = args.depth[pix];
      if (d <= 0 || mask[pix] < 0) continue;
      const float diff = (d - p.z) * sqrtf(1 + sq(p.x / p.z) + sq(p.y / p.z));
      if (diff > -args.mu) ++nupd;
    }
  }
  atomicAdd(&counts[0], nvis);
  atomicAdd(&counts[1], nupd);
}

// projective_functor::update_node, lib/functors/projective_functor.hpp:113-137,
// over every internal node of the selected instances.  The reference takes the
// node's voxel from unpack_morton(code) with the level bits still in the code,
// and offsets child i by dir * rotate(Tcw, (h, h, h)) element-wise; both kept.
// One thread per (node, child): the eight children update disjoint values, so
// the reference's loop over them runs as eight threads.
__global__ void __launch_bounds__(128)
integrate_nodes_kernel(const Volume* __restrict__ vols, const InstFrame* __restrict__ frames,
                       SdfArgs args, F4 k, IdList ids) {
  const int inst = ids.v[blockIdx.y];
  const Volume& V = vols[inst];
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long e = t >> 3;
  const int i = (int)(t & 7);
  if (e >= V.n_nodes || !V.node_tab[e]) return;
  int l = 1;
  while (l + 1 < V.block_level && e >= V.node_off[l + 1]) ++l;
  const unsigned long long mcode = (unsigned long long)(e - V.node_off[l]);
  const unsigned long long code = (mcode << (3 * (V.max_level - l))) | (unsigned long long)l;
  const InstFrame& F = frames[inst];
  const M4 K = camera_matrix(k);
  const float vs = V.dim / V.size;
  const unsigned side = (unsigned)V.size >> l;
  const F3 voxel = mk3((float)(int)gather3(code), (float)(int)gather3(code >> 1),
                       (float)(int)gather3(code >> 2));
  const F3 delta = rotate(F.Tcw, mk3(0.5f * vs * side));
  const F3 delta_c = rotate(K, delta);
  const F3 base_cam = xform(F.Tcw, voxel * vs);
  const F3 basepix = xform(K, base_cam);
  const float* mask = args.masks + (size_t)inst * args.W * args.H;
  const float wlim = args.W - 1.5f, hlim = args.H - 1.5f;
  const F3 dir = mk3((float)((i & 1) > 0), (float)((i & 2) > 0), (float)((i & 4) > 0));
  const F3 vox_cam = base_cam + dir * delta;
  const F3 pix_hom = basepix + dir * delta_c;
  if (vox_cam.z < 0.0001f) return;
  const float inv = 1.f / pix_hom.z;
  const float pxf = pix_hom.x * inv + 0.5f, pyf = pix_hom.y * inv + 0.5f;
  if (pxf < 0.5f || pxf > wlim || pyf < 0.5f || pyf > hlim) return;
  const size_t o = (size_t)e * 8 + i;
  sdf_update(args, mask, vox_cam, pxf, pyf, V.n_tsdf[o], V.n_wt[o], &V.n_r[o], &V.n_g[o],
             &V.n_b[o], V.n_c[o], V.n_fg[o], V.n_w[o]);
}

__global__ void interp_points_kernel(Pool pool, const Volume* __restrict__ vols, int inst,
                                     const float* __restrict__ pos, int n, int field,
                                     float* __restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  out[t] = volume_interp(pool, vols[inst], mk3(pos[3 * t], pos[3 * t + 1], pos[3 * t + 2]),
                         field);
}

// Gather selected blocks into the reference's 40-byte AoS voxel layout.
__global__ void export_blocks_kernel(Pool pool, const int* __restrict__ slots, int n,
                                     unsigned char* __restrict__ out) {
  const int b = blockIdx.x;
  if (b >= n) return;
  const int slot = slots[b];
  for (int v = threadIdx.x; v < 512; v += blockDim.x) {
    const size_t o = (size_t)slot * 512 + v;
    unsigned char* d = out + ((size_t)b * 512 + v) * 40;
    *(float*)(d + 0) = pool.tsdf[o];
    *(float*)(d + 4) = pool.wt[o];
    *(float*)(d + 8) = pool.r[o];
    *(float*)(d + 12) = pool.g[o];
    *(float*)(d + 16) = pool.b[o];
    *(int*)(d + 20) = pool.c[o];
    *(double*)(d + 24) = pool.fg[o];
    *(int*)(d + 32) = pool.w[o];
    *(int*)(d + 36) = 0;
  }
}

// ------------------------------------------------------------------ host side
static int div_up(long long a, int b) { return (int)((a + b - 1) / b); }

template <typename T>
static cudaError_t dalloc(T** p, size_t count) {
  return cudaMalloc((void**)p, sizeof(T) * (count ? count : 1));
}

__global__ void fill_node_values_kernel(Volume V) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V.n_nodes * 8) return;
  V.n_tsdf[i] = 1.f; V.n_wt[i] = 0.f; V.n_r[i] = 0.f; V.n_g[i] = 0.f; V.n_b[i] = 0.f;
  V.n_c[i] = 0; V.n_fg[i] = 0.0; V.n_w[i] = 0;
}

int volume_create(Context* ctx, Instance& in) {
  Volume& V = in.vol;
  std::memset(&V, 0, sizeof(V));
  V.size = in.size;
  V.dim = in.dim;
  int ml = 0;
  while ((1 << ml) < in.size) ++ml;
  V.max_level = ml;
  V.block_level = ml - 3;
  long long off = 0;
  for (int l = 1; l < V.block_level; ++l) { V.node_off[l] = off; off += 1LL << (3 * l); }
  V.node_off[V.block_level] = off;
  V.n_nodes = off;
  const long long n_tab = 1LL << (3 * V.block_level);
  MF_CUDA(dalloc(&V.block_tab, n_tab));
  MF_CUDA(cudaMemsetAsync(V.block_tab, 0xff, sizeof(int32_t) * n_tab, ctx->stream));
  MF_CUDA(dalloc(&V.req, n_tab));
  MF_CUDA(cudaMemsetAsync(V.req, 0, sizeof(uint32_t) * n_tab, ctx->stream));
  MF_CUDA(dalloc(&V.node_tab, V.n_nodes));
  MF_CUDA(cudaMemsetAsync(V.node_tab, 0, V.n_nodes ? V.n_nodes : 1, ctx->stream));
  const size_t nv = (size_t)V.n_nodes * 8;
  MF_CUDA(dalloc(&V.n_tsdf, nv)); MF_CUDA(dalloc(&V.n_wt, nv));
  MF_CUDA(dalloc(&V.n_r, nv)); MF_CUDA(dalloc(&V.n_g, nv)); MF_CUDA(dalloc(&V.n_b, nv));
  MF_CUDA(dalloc(&V.n_c, nv)); MF_CUDA(dalloc(&V.n_fg, nv)); MF_CUDA(dalloc(&V.n_w, nv));
  MF_CUDA(dalloc(&V.last_emit, 1)); MF_CUDA(dalloc(&V.emit_total, 1));
  MF_CUDA(dalloc(&V.bbox, 6));
  const int empty_box[6] = {INT_MAX, INT_MAX, INT_MAX, INT_MIN, INT_MIN, INT_MIN};
  MF_CUDA(cudaMemcpyAsync(V.bbox, empty_box, sizeof(empty_box), cudaMemcpyHostToDevice,
                          ctx->stream));
  if (nv) fill_node_values_kernel<<<div_up(nv, 256), 256, 0, ctx->stream>>>(V);
  MF_CUDA(cudaGetLastError());
  return MF_OK;
}

void volume_free(Instance& in) {
  Volume& V = in.vol;
  void* ps[] = {V.block_tab, V.req, V.node_tab, V.n_tsdf, V.n_wt, V.n_r, V.n_g, V.n_b,
                V.n_c, V.n_fg, V.n_w, V.last_emit, V.emit_total, V.bbox};
  for (void* p : ps) if (p) cudaFree(p);
  std::memset(&V, 0, sizeof(V));
}


int stage_prepare(Context* ctx, const IdList& ids, bool reset) {
  if (ids.n == 0) return MF_OK;
  const mf_config& c = ctx->cfg;
  prepare_kernel<<<ids.n, 96, 0, ctx->stream>>>(ctx->d_Twc, ctx->d_Two, ctx->d_vols, ctx->d_frames,
                                                F4{c.k[0], c.k[1], c.k[2], c.k[3]}, c.mu, ids,
                                                ctx->d_reserved, ctx->d_inst_label, reset,
                                                ctx->d_visit_count);
  MF_CUDA(cudaGetLastError());
  return MF_OK;
}

// After stage_prepare(ids, reset = true).
int stage_alloc(Context* ctx, const IdList& ids) {
  if (ids.n == 0) return MF_OK;
  const int WH = ctx->W * ctx->H;
  int max_tab = 0;
  for (int i = 0; i < ids.n; ++i) {
    const Volume& V = ctx->inst[ids.v[i]].vol;
    max_tab = std::max(max_tab, 1 << (3 * V.block_level));
  }
  alloc_mark_kernel<<<dim3(div_up(WH, 256), ids.n), 256, 0, ctx->stream>>>(
      ctx->d_depth, ctx->d_masks, ctx->W, ctx->H, ctx->d_vols, ctx->d_frames, ids, ctx->pool);
  MF_CUDA(cudaGetLastError());
  alloc_commit_kernel<<<dim3(div_up(max_tab, 256), ids.n), 256, 0, ctx->stream>>>(
      ctx->d_vols, ctx->d_frames, ids, ctx->pool, ctx->d_status);
  MF_CUDA(cudaGetLastError());
  return MF_OK;
}

// Timing and algorithmic bytes of integrate_blocks_kernel on the current
// frame (re-integrates the frame `reps` times; used after the timed region).
int profile_integrate(Context* ctx, int reps, double* us, double* bytes) {
  const int n = (int)ctx->inst.size();
  IdList all;
  all.n = n;
  for (int i = 0; i < n; ++i) all.v[i] = i;
  const mf_config& c = ctx->cfg;
  if (int rc = stage_prepare(ctx, all)) return rc;
  uint32_t mask = 0;
  for (int i = 0; i < n; ++i) mask |= 1u << i;
  MF_CUDA(cudaMemsetAsync(ctx->d_visit_count, 0, sizeof(int), ctx->stream));
  visit_list_kernel<<<div_up(ctx->pool.cap, 256), 256, 0, ctx->stream>>>(
      ctx->pool, ctx->d_vols, ctx->d_frames, mask, ctx->W, ctx->H, ctx->d_visit,
      ctx->d_visit_count, 1);
  SdfArgs a{ctx->d_depth, ctx->d_rgb, ctx->d_masks, ctx->W, ctx->H, c.mu, (float)c.max_weight};
  const F4 k{c.k[0], c.k[1], c.k[2], c.k[3]};
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  unsigned long long* d_cnt = nullptr;
  MF_CUDA(cudaMalloc(&d_cnt, 2 * sizeof(unsigned long long)));
  MF_CUDA(cudaMemsetAsync(d_cnt, 0, 2 * sizeof(unsigned long long), ctx->stream));
  integrate_count_kernel<<<sms * 8, 256, 0, ctx->stream>>>(ctx->pool, ctx->d_vols, ctx->d_frames,
                                                          a, k, ctx->d_visit, ctx->d_visit_count,
                                                          d_cnt);
  unsigned long long cnt[2] = {0, 0};
  int nv = 0;
  MF_CUDA(cudaMemcpyAsync(cnt, d_cnt, sizeof(cnt), cudaMemcpyDeviceToHost, ctx->stream));
  MF_CUDA(cudaMemcpyAsync(&nv, ctx->d_visit_count, sizeof(int), cudaMemcpyDeviceToHost,
                          ctx->stream));
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, ctx->stream);
  for (int r = 0; r < reps; ++r)
    if (int rc = launch_integrate_blocks(ctx, ctx->pool, ctx->tune.integrate)) return rc;
  cudaEventRecord(e1, ctx->stream);
  MF_CUDA(cudaEventSynchronize(e1));
  float ms = 0;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(d_cnt);
  MF_CUDA(cudaGetLastError());
  *us = 1e3 * ms / reps;
  // per visible voxel: depth + mask (8 B); per updated voxel: the 36-byte field
  // payload read and written and the pixel's rgb (12 B); per block: slot + meta.
  *bytes = 8.0 * cnt[0] + (36.0 + 36.0 + 12.0) * cnt[1] + 20.0 * nv;
  return MF_OK;
}

// Launch-shape candidates of integrate_blocks_kernel; entry 0 is the default.
// Callers keep the numbers (mf_tune_get): 0..2 have stood for three residencies
// without the prefetch and 3..5 for the same with it.  One residency is the
// fastest everywhere now, so each three are one shape.  Integration alone, 0 and
// 3 (us): one object 160x120 53 / 55, 640x480 59 / 62; three at 640x480
// 105 / 109; twelve uneven 72 / 76; six at 1280x720 157 / 169; whole frames are
// within 1 % of each other.
struct IntVariant {
  bool prefetch;
  void (*fn)(Pool, const Volume*, const InstFrame*, SdfArgs, F4, const int*, const int*);
};
static const IntVariant int_variants[] = {
    {false, integrate_blocks_kernel<false>}, {false, integrate_blocks_kernel<false>},
    {false, integrate_blocks_kernel<false>}, {true, integrate_blocks_kernel<true>},
    {true, integrate_blocks_kernel<true>},   {true, integrate_blocks_kernel<true>},
};
constexpr int N_INT_VARIANTS = (int)(sizeof(int_variants) / sizeof(int_variants[0]));
static_assert(N_INT_VARIANTS <= MAX_TUNE_VARIANTS, "integration candidate table too long");

int int_variant_count() { return N_INT_VARIANTS; }

void int_variant_describe(int v, char* buf, int cap) {
  snprintf(buf, cap, "integrate %d x 256-thread CTAs per SM%s", INT_CTAS,
           int_variants[v].prefetch ? ", next block's fields prefetched to L2" : "");
}

// The first number of the same shape.
int int_variant_first(int v) {
  int f = 0;
  while (int_variants[f].fn != int_variants[v].fn) ++f;
  return f;
}

// ctas > 0: that many CTAs instead of the variant's residency times the SM
// count (the grid-stride loop over the visit list gives the same voxels).
int launch_integrate_blocks(Context* ctx, const Pool& pool, int variant, int ctas) {
  const mf_config& c = ctx->cfg;
  SdfArgs a{ctx->d_depth, ctx->d_rgb, ctx->d_masks, ctx->W, ctx->H, c.mu, (float)c.max_weight};
  const F4 k{c.k[0], c.k[1], c.k[2], c.k[3]};
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  const IntVariant& v = int_variants[variant];
  // `ctas` counts 512 threads (mf_set_overlap)
  const int grid = ctas > 0 ? ctas * (512 / INT_THREADS) : sms * INT_CTAS;
  v.fn<<<grid, INT_THREADS, 0, ctx->stream>>>(pool, ctx->d_vols, ctx->d_frames, a, k, ctx->d_visit,
                                      ctx->d_visit_count);
  MF_CUDA(cudaGetLastError());
  return MF_OK;
}

// projective_functor::build_active_list over the instances in `inst_mask`.
// zeroed: stage_prepare has reset the list's counter, and the integration of
// the listed blocks follows (else the pool is left as it is).
int build_visit_list(Context* ctx, uint32_t inst_mask, bool zeroed) {
  if (!zeroed) MF_CUDA(cudaMemsetAsync(ctx->d_visit_count, 0, sizeof(int), ctx->stream));
  visit_list_kernel<<<div_up(ctx->pool.cap, 256), 256, 0, ctx->stream>>>(
      ctx->pool, ctx->d_vols, ctx->d_frames, inst_mask, ctx->W, ctx->H, ctx->d_visit,
      ctx->d_visit_count, zeroed);
  MF_CUDA(cudaGetLastError());
  return MF_OK;
}

// After stage_prepare(ids, reset = true).
int stage_integrate(Context* ctx, const IdList& ids, int ctas) {
  if (ids.n == 0) return MF_OK;
  const mf_config& c = ctx->cfg;
  uint32_t mask = 0;
  long long max_nodes = 0;
  for (int i = 0; i < ids.n; ++i) {
    mask |= 1u << ids.v[i];
    max_nodes = std::max(max_nodes, ctx->inst[ids.v[i]].vol.n_nodes);
  }
  if (int rc = build_visit_list(ctx, mask, true)) return rc;
  if (int rc = launch_integrate_blocks(ctx, ctx->pool, ctx->tune.integrate, ctas)) return rc;
  SdfArgs a{ctx->d_depth, ctx->d_rgb, ctx->d_masks, ctx->W, ctx->H, c.mu, (float)c.max_weight};
  const F4 k{c.k[0], c.k[1], c.k[2], c.k[3]};
  if (max_nodes > 0) {
    integrate_nodes_kernel<<<dim3(div_up(max_nodes * 8, 128), ids.n), 128, 0, ctx->stream>>>(
        ctx->d_vols, ctx->d_frames, a, k, ids);
    MF_CUDA(cudaGetLastError());
  }
  return MF_OK;
}

// Octree::alloc_update(keys, n), lib/octree.hpp:761-786, on explicit keys.
// Set semantics of the reference: after sorting, every key of level L >= 1
// creates its prefix octant at level min(L, block level) and the ancestors;
// the smallest key is kept at every level (unique.hpp:76-79), which creates
// its whole path down to a block.
int alloc_keys(Context* ctx, int id, const uint64_t* keys, int n) {
  Instance& in = ctx->inst[id];
  const Volume& V = in.vol;
  std::vector<unsigned long long> codes;
  std::vector<int> levels;
  uint64_t kmin = ~0ULL;
  const int cnt = n < 1 ? 1 : n;  // unique_multiscale returns 1 for n < 2
  for (int i = 0; i < cnt; ++i) kmin = std::min<uint64_t>(kmin, keys[i]);
  for (int i = 0; i < cnt; ++i) {
    int L = (int)(keys[i] & SCALE_MASK);
    if (keys[i] == kmin) L = V.block_level;
    if (L < 1) continue;
    if (L > V.block_level) L = V.block_level;
    codes.push_back(keys[i] & ~SCALE_MASK);
    levels.push_back(L);
  }
  if (codes.empty()) return MF_OK;
  unsigned long long* d_codes = nullptr;
  int* d_levels = nullptr;
  MF_CUDA(cudaMalloc(&d_codes, sizeof(unsigned long long) * codes.size()));
  MF_CUDA(cudaMalloc(&d_levels, sizeof(int) * levels.size()));
  MF_CUDA(cudaMemcpyAsync(d_codes, codes.data(), sizeof(unsigned long long) * codes.size(),
                          cudaMemcpyHostToDevice, ctx->stream));
  MF_CUDA(cudaMemcpyAsync(d_levels, levels.data(), sizeof(int) * levels.size(),
                          cudaMemcpyHostToDevice, ctx->stream));
  alloc_keys_kernel<<<div_up((long long)codes.size(), 256), 256, 0, ctx->stream>>>(
      ctx->d_vols, id, d_codes, d_levels, (int)codes.size(), ctx->pool, ctx->d_status);
  MF_CUDA(cudaGetLastError());
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  cudaFree(d_codes);
  cudaFree(d_levels);
  return MF_OK;
}

int ensure_export(Context* ctx, size_t bytes) {
  if (ctx->export_bytes >= bytes) return MF_OK;
  if (ctx->d_export) cudaFree(ctx->d_export);
  ctx->d_export = nullptr;
  ctx->export_bytes = 0;
  MF_CUDA(cudaMalloc(&ctx->d_export, bytes));
  ctx->export_bytes = bytes;
  return MF_OK;
}

int export_blocks(Context* ctx, int id, uint64_t* keys, int32_t* coords, uint8_t* active,
                  void* voxels, int cap, int* n_out) {
  const Volume& V = ctx->inst[id].vol;
  const long long n_tab = 1LL << (3 * V.block_level);
  std::vector<int32_t> tab(n_tab);
  MF_CUDA(cudaMemcpyAsync(tab.data(), V.block_tab, sizeof(int32_t) * n_tab,
                          cudaMemcpyDeviceToHost, ctx->stream));
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  std::vector<int> slots;
  std::vector<long long> bidx;
  for (long long b = 0; b < n_tab; ++b)
    if (tab[b] >= 0) { slots.push_back(tab[b]); bidx.push_back(b); }
  const int n = (int)slots.size();
  if (n_out) *n_out = n;
  if (!keys && !coords && !active && !voxels) return MF_OK;
  if (n > cap) return MF_E_ARG;
  if (n == 0) return MF_OK;
  std::vector<uint8_t> act;
  if (active) {
    std::vector<uint8_t> all(ctx->pool.cap);
    MF_CUDA(cudaMemcpy(all.data(), ctx->pool.active, ctx->pool.cap, cudaMemcpyDeviceToHost));
    for (int i = 0; i < n; ++i) active[i] = all[slots[i]];
  }
  for (int i = 0; i < n; ++i) {
    const uint64_t b = (uint64_t)bidx[i];
    if (keys) keys[i] = (b << (3 * (V.max_level - V.block_level))) | (uint64_t)V.block_level;
    if (coords) {
      coords[3 * i] = (int)gather3(b) << 3;
      coords[3 * i + 1] = (int)gather3(b >> 1) << 3;
      coords[3 * i + 2] = (int)gather3(b >> 2) << 3;
    }
  }
  if (voxels) {
    const int chunk = 4096;
    if (int rc = ensure_export(ctx, (size_t)chunk * 512 * 40 + sizeof(int) * chunk)) return rc;
    int* d_slots = (int*)((char*)ctx->d_export + (size_t)chunk * 512 * 40);
    for (int s0 = 0; s0 < n; s0 += chunk) {
      const int m = std::min(chunk, n - s0);
      MF_CUDA(cudaMemcpyAsync(d_slots, slots.data() + s0, sizeof(int) * m,
                              cudaMemcpyHostToDevice, ctx->stream));
      export_blocks_kernel<<<m, 256, 0, ctx->stream>>>(ctx->pool, d_slots, m,
                                                       (unsigned char*)ctx->d_export);
      MF_CUDA(cudaGetLastError());
      MF_CUDA(cudaMemcpyAsync((char*)voxels + (size_t)s0 * 512 * 40, ctx->d_export,
                              (size_t)m * 512 * 40, cudaMemcpyDeviceToHost, ctx->stream));
      MF_CUDA(cudaStreamSynchronize(ctx->stream));
    }
  }
  return MF_OK;
}

int export_nodes(Context* ctx, int id, uint64_t* keys, uint32_t* side, uint8_t* cmask,
                 void* values, int cap, int* n_out) {
  const Volume& V = ctx->inst[id].vol;
  const long long nn = V.n_nodes;
  std::vector<uint8_t> nt(nn > 0 ? nn : 1);
  const long long n_tab = 1LL << (3 * V.block_level);
  std::vector<int32_t> tab(n_tab);
  if (nn > 0)
    MF_CUDA(cudaMemcpyAsync(nt.data(), V.node_tab, nn, cudaMemcpyDeviceToHost, ctx->stream));
  MF_CUDA(cudaMemcpyAsync(tab.data(), V.block_tab, sizeof(int32_t) * n_tab,
                          cudaMemcpyDeviceToHost, ctx->stream));
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  std::vector<long long> ent;
  for (long long e = 0; e < nn; ++e) if (nt[e]) ent.push_back(e);
  const int n = (int)ent.size();
  if (n_out) *n_out = n;
  if (!keys && !side && !cmask && !values) return MF_OK;
  if (n > cap) return MF_E_ARG;
  std::vector<float> f[5];
  std::vector<int> ci, wi;
  std::vector<double> fg;
  if (values && nn > 0) {
    float* planes[5] = {V.n_tsdf, V.n_wt, V.n_r, V.n_g, V.n_b};
    for (int q = 0; q < 5; ++q) {
      f[q].resize(nn * 8);
      MF_CUDA(cudaMemcpy(f[q].data(), planes[q], sizeof(float) * nn * 8, cudaMemcpyDeviceToHost));
    }
    ci.resize(nn * 8); wi.resize(nn * 8); fg.resize(nn * 8);
    MF_CUDA(cudaMemcpy(ci.data(), V.n_c, sizeof(int) * nn * 8, cudaMemcpyDeviceToHost));
    MF_CUDA(cudaMemcpy(wi.data(), V.n_w, sizeof(int) * nn * 8, cudaMemcpyDeviceToHost));
    MF_CUDA(cudaMemcpy(fg.data(), V.n_fg, sizeof(double) * nn * 8, cudaMemcpyDeviceToHost));
  }
  for (int i = 0; i < n; ++i) {
    const long long e = ent[i];
    int l = 1;
    while (l + 1 < V.block_level && e >= V.node_off[l + 1]) ++l;
    const uint64_t m = (uint64_t)(e - V.node_off[l]);
    if (keys) keys[i] = (m << (3 * (V.max_level - l))) | (uint64_t)l;
    if (side) side[i] = (uint32_t)(V.size >> l);
    if (cmask) {
      uint8_t cm = 0;
      for (int c = 0; c < 8; ++c) {
        const uint64_t child = m * 8 + c;
        const bool ex = (l + 1 == V.block_level) ? tab[child] >= 0 : nt[V.node_off[l + 1] + child] != 0;
        if (ex) cm |= (uint8_t)(1 << c);
      }
      cmask[i] = cm;
    }
    if (values) {
      for (int c = 0; c < 8; ++c) {
        unsigned char* d = (unsigned char*)values + ((size_t)i * 8 + c) * 40;
        const size_t o = (size_t)e * 8 + c;
        std::memcpy(d + 0, &f[0][o], 4); std::memcpy(d + 4, &f[1][o], 4);
        std::memcpy(d + 8, &f[2][o], 4); std::memcpy(d + 12, &f[3][o], 4);
        std::memcpy(d + 16, &f[4][o], 4); std::memcpy(d + 20, &ci[o], 4);
        std::memcpy(d + 24, &fg[o], 8); std::memcpy(d + 32, &wi[o], 4);
        std::memset(d + 36, 0, 4);
      }
    }
  }
  return MF_OK;
}

int root_children(Context* ctx, int id, uint8_t* mask) {
  const Volume& V = ctx->inst[id].vol;
  uint8_t cm = 0;
  if (V.block_level == 1) {
    int32_t tab[8];
    MF_CUDA(cudaMemcpy(tab, V.block_tab, sizeof(tab), cudaMemcpyDeviceToHost));
    for (int c = 0; c < 8; ++c) if (tab[c] >= 0) cm |= (uint8_t)(1 << c);
  } else {
    uint8_t nt[8];
    MF_CUDA(cudaMemcpy(nt, V.node_tab + V.node_off[1], 8, cudaMemcpyDeviceToHost));
    for (int c = 0; c < 8; ++c) if (nt[c]) cm |= (uint8_t)(1 << c);
  }
  *mask = cm;
  return MF_OK;
}

int interp_points(Context* ctx, int id, const float* pos, int n, int field, float* out) {
  if (n <= 0) return MF_OK;
  if (int rc = ensure_export(ctx, sizeof(float) * 4 * n)) return rc;
  float* d_pos = (float*)ctx->d_export;
  float* d_out = d_pos + 3 * n;
  MF_CUDA(cudaMemcpyAsync(d_pos, pos, sizeof(float) * 3 * n, cudaMemcpyHostToDevice, ctx->stream));
  interp_points_kernel<<<div_up(n, 256), 256, 0, ctx->stream>>>(ctx->pool, ctx->d_vols, id, d_pos,
                                                                n, field, d_out);
  MF_CUDA(cudaGetLastError());
  MF_CUDA(cudaMemcpyAsync(out, d_out, sizeof(float) * n, cudaMemcpyDeviceToHost, ctx->stream));
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  return MF_OK;
}

}  // namespace mf
