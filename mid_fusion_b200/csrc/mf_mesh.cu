// Mesh export: marching cubes over one instance's octree, the reference's
// algorithms::marching_cube (lib/algorithms/meshing.hpp:20-208) as
// Kfusion::dump_mesh calls it (kfusion.cpp:1560-1588, inside = tsdf < 0), and
// writeVtkMesh (apps/kfusion/include/commons.h:945-1011).
//
// One CTA per allocated block at a time, one thread per cell, two passes: the
// first counts each block's kept triangles, the second writes them at the
// block's offset in cell order (x-major, then y, then z, as the reference
// loops).  The block list and the offsets are made on the device; the host
// waits once, for the triangle count.
// Blocks are taken in Morton order.  The triangulation table is this
// project's (gen_mc_tables.py) unless the caller supplies one
// (mf_mesh_set_triangle_table: the reference's triTable gives its triangles
// one for one); the cell test, the edge intersections and the vertex bounds
// are the reference's.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>
#include "mf_internal.h"
#include "mf_mc_tables.h"

namespace mf {

// corner offsets and edges (meshing.hpp:31-74); each edge is interpolated from
// its first corner to its second
__constant__ int8_t c_corner[8][3] = {{0, 0, 0}, {1, 0, 0}, {1, 0, 1}, {0, 0, 1},
                                      {0, 1, 0}, {1, 1, 0}, {1, 1, 1}, {0, 1, 1}};
#define MF_EDGE_CORNERS                                           \
  {{0, 1}, {1, 2}, {2, 3}, {0, 3}, {4, 5}, {5, 6}, {6, 7}, {4, 7}, \
   {0, 4}, {1, 5}, {2, 6}, {3, 7}}
__constant__ int8_t c_edge[12][2] = MF_EDGE_CORNERS;
static const int8_t edge_corners[12][2] = MF_EDGE_CORNERS;   // the host's

// A row that lists an edge whose two corners are on the same side (a caller's
// table may): its vertices lie anywhere on the edge's line, or nowhere.
constexpr int ROW_ANY_EDGE = 0x80;

struct MeshArgs {
  Pool pool;
  Volume V;
  const int8_t* tris;      // triangulation table, 256 x 3 * MF_MC_MAX_TRIS edge indices
  const uint8_t* rows;     // triangles of each table row, with ROW_ANY_EDGE
  const int* slots;        // the instance's blocks, Morton order
  const int* n_blocks;
  const long long* offset; // first triangle of each block (pass 2)
  int* count;              // kept triangles of each block (pass 1)
  float* out;              // 9 floats per triangle
  float bound;             // vertex bound: (int)dim as the reference, or dim
};

// The voxels of a block and of its neighbours' first layer, 9 x 9 x 9.
constexpr int MESH_N = 9, MESH_VOX = MESH_N * MESH_N * MESH_N;
struct MeshTile {
  float tsdf[MESH_VOX];
  uint8_t ok[MESH_VOX];    // weight, foreground and count pass compute_index's tests
  int slot[8];             // the block and its upper neighbours
  int8_t corner[8];        // a cell corner's offset, as bits x | y << 1 | z << 2
  int8_t edge[12][2];
  uint8_t rows[256];       // MeshArgs::rows
  int warp[16];
};
__device__ __forceinline__ int mesh_at(int x, int y, int z) {
  return x + MESH_N * (y + MESH_N * z);
}

// Loads the tile of the block at `m`.  get_fine (lib/octree.hpp:360-379): the
// voxel, or the initial value (tsdf 1, weight 0, fg 0, count 0) where the block
// is not allocated.  Each voxel is read and tested once; eight times, by every
// cell that it is a corner of and through a table lookup each, the two passes
// took 190 us each over the 4700 blocks of a 512^3 room (165 with 32-bit block
// indices), now 76 and 95, with the divisions that give +-0 left out.
__device__ __forceinline__ void mesh_load(const MeshArgs& a, MeshTile& s, int4 m) {
  if (threadIdx.x < 8)
    s.slot[threadIdx.x] = block_slot(a.V, m.x + 8 * (threadIdx.x & 1),
                                     m.y + 8 * ((threadIdx.x >> 1) & 1), m.z + 8 * (threadIdx.x >> 2));
  __syncthreads();
  for (int v = threadIdx.x; v < MESH_VOX; v += 512) {
    const int x = v % MESH_N, y = v / MESH_N % MESH_N, z = v / (MESH_N * MESH_N);
    const int slot = s.slot[(x >> 3) | ((y >> 3) << 1) | ((z >> 3) << 2)];
    float tsdf = 1.f;
    bool ok = false;   // weight 0
    if (slot >= 0) {
      const size_t o = (size_t)slot * 512 + voxel_index(x, y, z);
      tsdf = a.pool.tsdf[o];
      const double fg_threshold = 0.5f;
      ok = !(a.pool.wt[o] == 0.f) && !(a.pool.fg[o] <= fg_threshold || a.pool.w[o] <= 3);
    }
    s.tsdf[v] = tsdf;
    s.ok[v] = ok;
  }
  __syncthreads();
}

// meshing::compute_intersection (meshing.hpp:20-29) on edge e of the cell at
// voxel (x, y, z), element `cell` of the tile; any_edge: the edge's corners may
// be on the same side
__device__ __forceinline__ F3 edge_vertex(const MeshArgs& a, const MeshTile& t, int cell, int x,
                                          int y, int z, int e, bool any_edge) {
  const float voxelSize = a.V.dim / a.V.size;
  const int c0 = t.corner[t.edge[e][0]], c1 = t.corner[t.edge[e][1]];
  const unsigned sx = x + (c0 & 1), sy = y + ((c0 >> 1) & 1), sz = z + (c0 >> 2);
  const unsigned dx = x + (c1 & 1), dy = y + ((c1 >> 1) & 1), dz = z + (c1 >> 2);
  const F3 s = mk3(sx * voxelSize, sy * voxelSize, sz * voxelSize);
  const F3 d = mk3(dx * voxelSize, dy * voxelSize, dz * voxelSize);
  const float v1 = t.tsdf[cell + mesh_at(c0 & 1, (c0 >> 1) & 1, c0 >> 2)];
  const float v2 = t.tsdf[cell + mesh_at(c1 & 1, (c1 >> 1) & 1, c1 >> 2)];
  const float k = (float)(0.0 - v1);
  const float den = v2 - v1;
  // s + (k * (d - s)) / den: on the two axes along which the edge does not run
  // the addend is +-0, unless k or den is not finite, or den is 0 (which takes
  // corners on the same side)
  if (!any_edge && fabsf(k) < INFINITY && fabsf(den) < INFINITY) {
    const int axis = c0 ^ c1;   // one bit: the axis of the edge
    const float ss = axis == 1 ? s.x : axis == 2 ? s.y : s.z;
    const float ds = axis == 1 ? d.x : axis == 2 ? d.y : d.z;
    const float v = ss + (k * (ds - ss)) / den;
    return mk3(axis == 1 ? v : s.x, axis == 2 ? v : s.y, axis == 4 ? v : s.z);
  }
  const F3 dd = d - s;
  return mk3(s.x + (k * dd.x) / den, s.y + (k * dd.y) / den, s.z + (k * dd.z) / den);
}

// meshing::checkVertex (meshing.hpp:148-150), whose int dim is the
// volume's extent truncated (meshing.hpp:169)
__device__ __forceinline__ bool outside_dim(F3 p, float dim) {
  return p.x <= 0 || p.y <= 0 || p.z <= 0 || p.x > dim || p.y > dim || p.z > dim;
}

template <bool EMIT>
__global__ void __launch_bounds__(512) mesh_kernel(MeshArgs a) {
  __shared__ MeshTile s;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if (t < 8) s.corner[t] = c_corner[t][0] | (c_corner[t][1] << 1) | (c_corner[t][2] << 2);
  if (t < 24) s.edge[t >> 1][t & 1] = c_edge[t >> 1][t & 1];
  if (t < 256) s.rows[t] = a.rows[t];
  const float voxelSize = a.V.dim / a.V.size;
  const int nb = *a.n_blocks;
  const int bound = a.V.size - 1;  // clamp(corner + 8, 0, size - 1)
  const int lx = t >> 6, ly = (t >> 3) & 7, lz = t & 7, cell = mesh_at(lx, ly, lz);
  for (int b = blockIdx.x; b < nb; b += gridDim.x) {
    if (EMIT && a.count[b] == 0) continue;   // uniform
    const int4 m = a.pool.meta[a.slots[b]];
    const int x = m.x + lx, y = m.y + ly, z = m.z + lz;
    __syncthreads();   // the last block's tile has been read
    mesh_load(a, s, m);
    int index = 0;
    if (x < min(m.x + 8, bound) && y < min(m.y + 8, bound) && z < min(m.z + 8, bound)) {
      // meshing::compute_index (meshing.hpp:76-132)
      bool ok = true;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int c = s.corner[i];
        const int v = cell + mesh_at(c & 1, (c >> 1) & 1, c >> 2);
        ok = ok && s.ok[v];
        if (s.tsdf[v] < 0.f) index |= 1 << i;
      }
      if (!ok) index = 0;
    }
    // kept triangles of this cell, in table order
    const int8_t* tr = a.tris + index * (3 * MF_MC_MAX_TRIS);
    // the vertex of an edge whose corners are on different sides lies between
    // them, so only cells next to 0 or within two voxels of the bound can have
    // one outside
    const bool any_edge = s.rows[index] & ROW_ANY_EDGE;
    unsigned keep = (1u << (s.rows[index] & ~ROW_ANY_EDGE)) - 1u;
    if (keep && (any_edge || !(x > 0 && y > 0 && z > 0 &&
                               (max(x, max(y, z)) + 2) * voxelSize <= a.bound)))
      for (int e = 0; e < 3 * MF_MC_MAX_TRIS && tr[e] != -1; e += 3)
        if (outside_dim(edge_vertex(a, s, cell, x, y, z, tr[e], any_edge), a.bound) ||
            outside_dim(edge_vertex(a, s, cell, x, y, z, tr[e + 1], any_edge), a.bound) ||
            outside_dim(edge_vertex(a, s, cell, x, y, z, tr[e + 2], any_edge), a.bound))
          keep &= ~(1u << (e / 3));
    const int kept = __popc(keep);
    // exclusive scan of the cells' counts in thread (cell) order
    int inc = kept;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += n;
    }
    if (lane == 31) s.warp[warp] = inc;
    __syncthreads();
    if (t < 32) {
      int w = t < 16 ? s.warp[t] : 0;
#pragma unroll
      for (int d = 1; d < 16; d <<= 1) {
        const int n = __shfl_up_sync(0xffffffffu, w, d);
        if (t >= d) w += n;
      }
      if (t < 16) s.warp[t] = w;  // inclusive over warps
    }
    __syncthreads();
    if (!EMIT) {
      if (t == 0) a.count[b] = s.warp[15];
      continue;
    }
    float* o = a.out + 9 * (a.offset[b] + inc - kept + (warp > 0 ? s.warp[warp - 1] : 0));
    for (int k = 0; keep; ++k, keep >>= 1) {
      if (!(keep & 1u)) continue;
#pragma unroll
      for (int c = 0; c < 3; ++c, o += 3) {
        const F3 v = edge_vertex(a, s, cell, x, y, z, tr[3 * k + c], any_edge);
        o[0] = v.x;
        o[1] = v.y;
        o[2] = v.z;
      }
    }
  }
}

// The allocated slots of a block table in the table's (Morton) order: the
// number in each chunk of the table, then every chunk's slots behind those of
// the chunks before it.
__global__ void __launch_bounds__(1024)
mesh_count_slots_kernel(const int32_t* __restrict__ tab, long long n_tab, int chunk,
                        int* __restrict__ chunk_count) {
  const long long e0 = (long long)blockIdx.x * chunk;
  int c = 0;
  for (long long e = e0 + threadIdx.x; e < min(e0 + chunk, n_tab); e += 1024) c += tab[e] >= 0;
  c = __reduce_add_sync(0xffffffffu, c);
  __shared__ int sw[32];
  if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x < 32) {
    c = __reduce_add_sync(0xffffffffu, sw[threadIdx.x]);
    if (threadIdx.x == 0) chunk_count[blockIdx.x] = c;
  }
}

__global__ void __launch_bounds__(1024)
mesh_list_slots_kernel(const int32_t* __restrict__ tab, long long n_tab, int chunk,
                       const int* __restrict__ chunk_count, int* __restrict__ slots, int cap,
                       int* __restrict__ n_blocks) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ int sw[32], s_base;
  // the slots before this chunk
  int c = 0;
  for (int b = threadIdx.x; b < (int)blockIdx.x; b += 1024) c += chunk_count[b];
  c = __reduce_add_sync(0xffffffffu, c);
  if (lane == 0) sw[warp] = c;
  __syncthreads();
  if (warp == 0) {
    c = __reduce_add_sync(0xffffffffu, sw[lane]);
    if (lane == 0) s_base = c;
  }
  __syncthreads();
  int base = s_base;
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0)
    *n_blocks = min(base + chunk_count[blockIdx.x], cap);
  const long long e0 = (long long)blockIdx.x * chunk, e1 = min(e0 + chunk, n_tab);
  for (long long r = e0; r < e1; r += 1024) {
    const long long e = r + threadIdx.x;
    const int slot = e < e1 ? tab[e] : -1;
    const unsigned m = __ballot_sync(0xffffffffu, slot >= 0);
    __syncthreads();
    if (lane == 0) sw[warp] = __popc(m);
    __syncthreads();
    int before = 0, total = 0;
    for (int w = 0; w < 32; ++w) {
      before += w < warp ? sw[w] : 0;
      total += sw[w];
    }
    const int at = base + before + __popc(m & ((1u << lane) - 1u));
    if (slot >= 0 && at < cap) slots[at] = slot;
    base += total;
  }
}

// Exclusive offsets of the blocks' triangle counts, and their total; one CTA.
__global__ void __launch_bounds__(1024)
mesh_offsets_kernel(const int* __restrict__ count, const int* __restrict__ n_blocks,
                    long long* __restrict__ offset, long long* __restrict__ total) {
  __shared__ int sw[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = *n_blocks;
  long long base = 0;
  for (int b0 = 0; b0 < n; b0 += 1024) {
    const int b = b0 + threadIdx.x;
    const int c = b < n ? count[b] : 0;
    int inc = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += v;
    }
    __syncthreads();
    if (lane == 31) sw[warp] = inc;
    __syncthreads();
    int before = 0, sum = 0;
    for (int w = 0; w < 32; ++w) {
      before += w < warp ? sw[w] : 0;
      sum += sw[w];
    }
    if (b < n) offset[b] = base + before + inc - c;
    base += sum;
  }
  if (threadIdx.x == 0) *total = base;
}

// The context's triangulation table on the device: `table` (256 rows of 16
// ints, edge triples ended by -1, the layout of the reference's triTable,
// lib/algorithms/edge_tables.h), or the built-in one when table is NULL.
int mesh_set_table(Context* ctx, const int* table) {
  struct {
    int8_t t[256][3 * MF_MC_MAX_TRIS];
    uint8_t rows[256];   // MeshArgs::rows, behind the table on the device
  } host;
  auto& t = host.t;
  if (!table) {
    std::memcpy(t, MF_MC_TRIS, sizeof(t));
  } else {
    for (int r = 0; r < 256; ++r) {
      const int* row = table + 16 * r;
      int n = 0;
      while (n < 16 && row[n] != -1) ++n;
      if (n == 16 || n % 3 != 0 || n > 3 * MF_MC_MAX_TRIS) {
        ctx->last_error = "mf_mesh_set_triangle_table: row " + std::to_string(r) +
                          " is not at most 5 edge triples ended by -1";
        return MF_E_ARG;
      }
      for (int e = 0; e < 3 * MF_MC_MAX_TRIS; ++e) {
        if (e < n && (row[e] < 0 || row[e] > 11)) {
          ctx->last_error = "mf_mesh_set_triangle_table: edge index outside 0..11 in row " +
                            std::to_string(r);
          return MF_E_ARG;
        }
        t[r][e] = e < n ? (int8_t)row[e] : (int8_t)-1;
      }
    }
  }
  for (int r = 0; r < 256; ++r) {
    int n = 0;
    bool any_edge = false;
    for (; n < 3 * MF_MC_MAX_TRIS && t[r][n] != -1; ++n) {
      const int8_t* e = edge_corners[t[r][n]];
      any_edge = any_edge || ((r >> e[0]) & 1) == ((r >> e[1]) & 1);
    }
    host.rows[r] = (uint8_t)(n / 3 | (any_edge ? ROW_ANY_EDGE : 0));
  }
  if (!ctx->d_mc_tris) MF_CUDA(cudaMalloc(&ctx->d_mc_tris, sizeof(host)));
  MF_CUDA(cudaMemcpyAsync(ctx->d_mc_tris, &host, sizeof(host), cudaMemcpyHostToDevice,
                          ctx->stream));
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  return MF_OK;
}

// Scratch for a mesh that a context keeps between calls: 1.8 million
// triangles, six times those of a 3.2 m room at 1 cm.  A larger mesh allocates
// for its call, so that a single export does not hold that much for good.
constexpr size_t MESH_KEEP = 64 << 20;

int mesh_volume(Context* ctx, int id, int float_bounds, float* tris, long long cap,
                long long* n_tris) {
  if (!ctx->d_mc_tris)
    if (int rc = mesh_set_table(ctx, nullptr)) return rc;
  const Volume& V = ctx->inst[id].vol;
  const long long n_tab = 1LL << (3 * V.block_level);
  // scratch: triangle count and block count, slots, triangle counts, offsets
  // of every block that the instance can hold, chunk counts
  const int chunk = (int)std::max(1024LL, n_tab / 4096);
  const int n_chunks = (int)((n_tab + chunk - 1) / chunk);
  const int cap_blocks = (int)std::min<long long>(n_tab, ctx->pool.cap);
  const size_t sb = (sizeof(int) * (size_t)cap_blocks + 15) / 16 * 16;
  if (int rc = ensure_export(ctx, 16 + 2 * sb + sizeof(long long) * cap_blocks +
                                      sizeof(int) * (size_t)n_chunks))
    return rc;
  char* base = (char*)ctx->d_export;
  long long* d_total = (long long*)base;
  int* d_nblocks = (int*)(base + 8);
  int* d_slots = (int*)(base + 16);
  int* d_count = (int*)(base + 16 + sb);
  long long* d_off = (long long*)(base + 16 + 2 * sb);
  int* d_chunks = (int*)(d_off + cap_blocks);
  mesh_count_slots_kernel<<<n_chunks, 1024, 0, ctx->stream>>>(V.block_tab, n_tab, chunk, d_chunks);
  mesh_list_slots_kernel<<<n_chunks, 1024, 0, ctx->stream>>>(V.block_tab, n_tab, chunk, d_chunks,
                                                             d_slots, cap_blocks, d_nblocks);
  MeshArgs a;
  a.tris = ctx->d_mc_tris;
  a.rows = (const uint8_t*)ctx->d_mc_tris + 256 * 3 * MF_MC_MAX_TRIS;
  a.pool = ctx->pool;
  a.V = V;
  a.slots = d_slots;
  a.n_blocks = d_nblocks;
  a.offset = d_off;
  a.count = d_count;
  a.out = nullptr;
  a.bound = float_bounds ? V.dim : (float)(int)V.dim;
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  const int grid = std::min(cap_blocks, 4 * sms);
  mesh_kernel<false><<<grid, 512, 0, ctx->stream>>>(a);
  mesh_offsets_kernel<<<1, 1024, 0, ctx->stream>>>(d_count, d_nblocks, d_off, d_total);
  MF_CUDA(cudaGetLastError());
  long long total = 0;
  MF_CUDA(cudaMemcpyAsync(&total, d_total, sizeof(total), cudaMemcpyDeviceToHost, ctx->stream));
  MF_CUDA(cudaStreamSynchronize(ctx->stream));
  *n_tris = total;
  if (!tris || cap < total || total == 0) return MF_OK;
  // the triangles: straight into a device destination, else through scratch
  // that the context keeps up to MESH_KEEP (mf_destroy frees it)
  cudaPointerAttributes at{};
  const bool dev = cudaPointerGetAttributes(&at, tris) == cudaSuccess &&
                   (at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged);
  cudaGetLastError();
  const size_t bytes = sizeof(float) * 9 * (size_t)total;
  if (!dev && ctx->mesh_bytes < bytes) {
    if (ctx->d_mesh) cudaFree(ctx->d_mesh);
    ctx->d_mesh = nullptr;
    ctx->mesh_bytes = 0;
    MF_CUDA(cudaMalloc(&ctx->d_mesh, bytes));
    ctx->mesh_bytes = bytes;
  }
  float* const scratch = ctx->d_mesh;
  a.out = dev ? tris : scratch;
  mesh_kernel<true><<<grid, 512, 0, ctx->stream>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && !dev)
    e = cudaMemcpyAsync(tris, scratch, bytes, cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (ctx->mesh_bytes > MESH_KEEP) {
    cudaFree(ctx->d_mesh);
    ctx->d_mesh = nullptr;
    ctx->mesh_bytes = 0;
  }
  if (e != cudaSuccess) {
    ctx->last_error = std::string("mf_mesh: ") + cudaGetErrorString(e);
    return MF_E_CUDA;
  }
  return MF_OK;
}

// writeVtkMesh (commons.h:945-1011) without point or cell data: every
// triangle its own three points, floats as std::ostream prints them (%g).
int write_vtk_mesh(const char* path, const float* tris, long long n) {
  FILE* f = std::fopen(path, "w");
  if (!f) return MF_E_NOT_FOUND;
  std::fprintf(f, "# vtk DataFile Version 1.0\nvtk mesh generated from KFusion\nASCII\n"
                  "DATASET POLYDATA\nPOINTS %lld FLOAT\n", 3 * n);
  for (long long i = 0; i < 3 * n; ++i)
    std::fprintf(f, "%g %g %g\n", (double)tris[3 * i], (double)tris[3 * i + 1],
                 (double)tris[3 * i + 2]);
  std::fprintf(f, "POLYGONS %lld %lld\n", n, 4 * n);
  for (long long i = 0; i < n; ++i)
    std::fprintf(f, "3 %lld %lld %lld\n", 3 * i, 3 * i + 1, 3 * i + 2);
  std::fprintf(f, "\n");
  const bool ok = std::ferror(f) == 0;
  std::fclose(f);
  return ok ? MF_OK : MF_E_ARG;
}

}  // namespace mf
