// kf_mesh.cu - marching cubes on the device (MarchingCubes::extract and
// MeshBuilder, marching_cubes.cpp:311-485), dense and sparse volumes.
//
// The mesh is the one the host builder makes, element for element: the same
// cells in the same order (x fastest over the (res-1)^3 cells; sparse:
// allocated blocks in block order, x fastest within each), the same
// welded vertices numbered in order of first use, the same positions,
// normals and colours.  The triangulation table is this library's generated
// one (kf_mc_tables.h).  Passes:
//  1. per row of cells (fixed y, z; sparse: per allocated block), classify
//     the cells: a cell whose corners are all observed, finite and at least
//     min_weight has a sign case; set a bit per crossed edge (key = near
//     voxel's storage index * 3 + axis) and count the unit's triangles.  A
//     dense row reads the raycast's stencil records, eight cells at a time:
//     cells they decide (no observed corner, or all corners exactly 1) cannot
//     cross the surface and are not looked at;
//  2. exclusive scans give each row its first triangle and each crossed edge
//     a compact id;
//  3. per row again, write every triangle corner's edge id, each edge's key
//     and its first use (smallest triangle-corner position, atomicMin);
//  4. a bitmap of first-use positions, scanned, numbers the vertices in
//     order of first use; one thread per edge computes its vertex;
//  5. triangle corners are mapped to vertex numbers; a vertex without a
//     gradient normal collects its triangles and takes their face normals'
//     average, summed in triangle order as the host builder does.
//
// The working arrays stay with the pipeline between calls (up to
// kMeshKeepBytes in all), and the mesh comes back through page-locked staging
// (up to kMeshStageBytes; a larger one is copied straight to its arrays).
// 512^3 float after 8 frames: 0.7-0.9 ms a call against 5.3-6.4 ms with a pass
// over every cell, twenty allocations and the fill on the host.  A pipeline's
// first call makes the arrays and the staging: 4.1-5.4 ms against 5.5-8.2 ms;
// so does every call whose arrays are too large to keep.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "kf_internal.h"
// the triangulation tables live in constant memory
#define KF_MC_TABLE static __constant__ const
#include "kf_mc_tables.h"
#include "kf_sampler.cuh"

namespace kf {
namespace {

constexpr int kRowThreads = 256;
constexpr int kScanThreads = 256;
constexpr int kScanItems = 4;  // elements per thread of a scan block
constexpr unsigned kScanBlock = kScanThreads * kScanItems;

// Sign case of cell (x, y, z), or -1 when a corner is unobserved, not finite
// or lighter than min_weight (MeshBuilder::add_cell, marching_cubes.cpp:369-384).
template <int Kind>
__device__ __forceinline__ int cell_case(const VolumeDev& v, uint32_t x, uint32_t y, uint32_t z, float min_weight) {
  using VT = VoxelTraits<Kind>;
  const auto* voxels = reinterpret_cast<const typename VT::Raw*>(v.voxels);
  int cube = 0;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const long long i = storage_index(v, x + kMcCorner[c][0], y + kMcCorner[c][1], z + kMcCorner[c][2]);
    if (i < 0) return -1;
    const typename VT::Raw r = __ldg(voxels + i);
    if (!VT::observed(r) || !VT::finite(r) || VT::weight(r) < min_weight) return -1;
    if (VT::tsdf(r) < 0.0f) cube |= 1 << c;
  }
  return cube;
}

// Weld key of cube edge `edge` of cell (x, y, z): the near voxel's storage
// index * 3 + axis (unique per edge; the near voxel is stored whenever a
// cell using the edge is meshed).
__device__ __forceinline__ unsigned long long edge_key(const VolumeDev& v, uint32_t x, uint32_t y, uint32_t z,
                                                       int edge) {
  const int near = kMcEdge[edge][0];
  const long long i = storage_index(v, x + kMcCorner[near][0], y + kMcCorner[near][1], z + kMcCorner[near][2]);
  return static_cast<unsigned long long>(i) * 3ull + kMcEdge[edge][2];
}

__device__ __forceinline__ uint32_t triangle_count(int cube) {
  uint32_t n = 0;
  while (n < 5 && kMcTriangles[cube][3 * n] >= 0) ++n;
  return n;
}

// Exclusive scan of n values over a CTA of kRowThreads; returns the total.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t value, uint32_t& prefix, uint32_t* s_warp) {
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t incl = value;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, incl, off);
    if (lane >= static_cast<unsigned>(off)) incl += up;
  }
  if (lane == 31u) s_warp[warp] = incl;
  __syncthreads();
  uint32_t warp_base = 0, total = 0;
  for (unsigned w = 0; w < blockDim.x / 32u; ++w) {
    if (w < warp) warp_base += s_warp[w];
    total += s_warp[w];
  }
  __syncthreads();
  prefix = warp_base + incl - value;
  return total;
}

// Pass 1 (Write = false): the crossed-edge bits of an active cell.  Pass 3
// (Write = true): its triangle corners' edge ids from `first` on, and each
// edge's first use.
template <bool Write>
__device__ __forceinline__ void emit_cell(const VolumeDev& v, uint32_t x, uint32_t y, uint32_t z, int cube,
                                          uint32_t tris, uint32_t first, uint32_t* __restrict__ edge_words,
                                          const uint32_t* __restrict__ word_first, uint32_t* __restrict__ corner_edge,
                                          uint32_t* __restrict__ first_use,
                                          unsigned long long* __restrict__ edge_of) {
  if constexpr (!Write) {
    const uint32_t mask = kMcEdgeMask[cube];
    for (int e = 0; e < 12; ++e) {
      if (!((mask >> e) & 1u)) continue;
      const unsigned long long key = edge_key(v, x, y, z, e);
      atomicOr(edge_words + (key >> 5), 1u << (key & 31u));
    }
  } else {
    for (uint32_t t = 0; t < tris; ++t) {
      for (int k = 0; k < 3; ++k) {
        const unsigned long long key = edge_key(v, x, y, z, kMcTriangles[cube][3 * t + k]);
        const uint32_t w = static_cast<uint32_t>(key >> 5), b = static_cast<uint32_t>(key & 31u);
        const uint32_t id = word_first[w] + __popc(edge_words[w] & ((1u << b) - 1u));
        const uint32_t position = 3u * (first + t) + static_cast<uint32_t>(k);
        corner_edge[position] = id;
        edge_of[id] = key;
        atomicMin(first_use + id, position);
      }
    }
  }
}

// Dense volumes: one warp per row of cells (fixed y, z), x fastest (the host
// builder's GridIndices order), a lane per brick of the row: the brick layer's
// stencil record has the row's eight cells in one byte.  Pass 1 counts the
// row's triangles.  (One thread per cell of every row took 820 us a pass at
// 512^3; 143 and 196 us.)
template <int Kind, bool Write>
__global__ void __launch_bounds__(kRowThreads)
    mc_rows_kernel(VolumeDev v, const uint4* __restrict__ stencil_bits, float min_weight,
                   uint32_t* __restrict__ edge_words, uint32_t* __restrict__ row_tris,
                   const uint32_t* __restrict__ row_first, const uint32_t* __restrict__ word_first,
                   uint32_t* __restrict__ corner_edge, uint32_t* __restrict__ first_use,
                   unsigned long long* __restrict__ edge_of) {
  const uint32_t cx = v.rx - 1, cy = v.ry - 1, lane = threadIdx.x & 31u;
  const uint32_t row = blockIdx.x * (kRowThreads / 32) + (threadIdx.x >> 5);
  if (row >= cy * (v.rz - 1)) return;
  const uint32_t y = row % cy, z = row / cy;
  uint32_t base = Write ? row_first[row] : 0u;
  for (uint32_t b0 = 0; b0 < v.bx; b0 += 32u) {
    const uint32_t b = b0 + lane;
    uint32_t cells = 0u;  // bit i: cell (8 b + i, y, z) may cross the surface
    if (b < v.bx) {
      const uint4 r = __ldg(stencil_bits + ((static_cast<size_t>(z >> 3) * v.by + (y >> 3)) * v.bx + b) * 8u + (z & 7u));
      cells = (((y & 4u) != 0u ? r.y : r.x) >> ((y & 3u) * 8u)) & 0xFFu;
      if (8u * b + 8u > cx) cells &= 8u * b < cx ? (1u << (cx - 8u * b)) - 1u : 0u;
    }
    if (__ballot_sync(0xFFFFFFFFu, cells != 0u) == 0u) continue;
    unsigned long long cubes = 0ull;
    uint32_t active = 0u, tris = 0u;
    for (uint32_t m = cells; m != 0u; m &= m - 1u) {
      const uint32_t i = static_cast<uint32_t>(__ffs(static_cast<int>(m)) - 1), x = 8u * b + i;
      const int cube = cell_case<Kind>(v, x, y, z, min_weight);
      if (cube < 0 || kMcEdgeMask[cube] == 0) continue;
      tris += triangle_count(cube);
      if constexpr (Write) {
        active |= 1u << i;
        cubes |= static_cast<unsigned long long>(cube) << (8u * i);
      } else {
        emit_cell<false>(v, x, y, z, cube, 0u, 0u, edge_words, word_first, corner_edge, first_use, edge_of);
      }
    }
    uint32_t incl = tris;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, incl, off);
      if (lane >= static_cast<unsigned>(off)) incl += up;
    }
    if constexpr (Write) {
      uint32_t at = base + incl - tris;
      for (uint32_t m = active; m != 0u; m &= m - 1u) {
        const uint32_t i = static_cast<uint32_t>(__ffs(static_cast<int>(m)) - 1);
        const int cube = static_cast<int>((cubes >> (8u * i)) & 0xFFull);
        const uint32_t n = triangle_count(cube);
        emit_cell<true>(v, 8u * b + i, y, z, cube, n, at, edge_words, word_first, corner_edge, first_use, edge_of);
        at += n;
      }
    }
    base += __shfl_sync(0xFFFFFFFFu, incl, 31);
  }
  if (!Write && lane == 0) row_tris[row] = base;
}

// Sparse volumes: one CTA of 512 threads per allocated block, in block order,
// its cells x fastest, then y, then z (BlockVoxels order, clipped to the
// cells of the volume).  Pass 1 counts the block's triangles.
template <int Kind, bool Write>
__global__ void __launch_bounds__(512)
    mc_blocks_kernel(VolumeDev v, const uint32_t* __restrict__ blocks, float min_weight,
                     uint32_t* __restrict__ edge_words, uint32_t* __restrict__ unit_tris,
                     const uint32_t* __restrict__ unit_first, const uint32_t* __restrict__ word_first,
                     uint32_t* __restrict__ corner_edge, uint32_t* __restrict__ first_use,
                     unsigned long long* __restrict__ edge_of) {
  __shared__ uint32_t s_warp[512 / 32];
  const uint32_t block = blocks[blockIdx.x];
  const uint32_t x = (block % v.bx) * 8u + (threadIdx.x & 7u);
  const uint32_t y = ((block / v.bx) % v.by) * 8u + ((threadIdx.x >> 3) & 7u);
  const uint32_t z = (block / (v.bx * v.by)) * 8u + (threadIdx.x >> 6);
  int cube = -1;
  uint32_t tris = 0;
  if (x < v.rx - 1 && y < v.ry - 1 && z < v.rz - 1) {
    cube = cell_case<Kind>(v, x, y, z, min_weight);
    if (cube >= 0 && kMcEdgeMask[cube] != 0) tris = triangle_count(cube);
  }
  uint32_t prefix;
  const uint32_t total = block_exclusive_scan(tris, prefix, s_warp);
  if (tris != 0u) {
    emit_cell<Write>(v, x, y, z, cube, tris, (Write ? unit_first[blockIdx.x] : 0u) + prefix, edge_words, word_first,
                     corner_edge, first_use, edge_of);
  }
  if (!Write && threadIdx.x == 0) unit_tris[blockIdx.x] = total;
}

// Allocated blocks of a sparse grid, in block order.
// Sparse storage: flag the block of every used pool slot (the slots are
// handed out in order, min(attempts, capacity) of them).
__global__ void allocated_flags_kernel(const uint32_t* __restrict__ slot_block,
                                       const unsigned long long* __restrict__ allocated, unsigned long long capacity,
                                       uint32_t* __restrict__ flags) {
  const unsigned long long used = allocated[0] < capacity ? allocated[0] : capacity;
  for (unsigned long long s = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; s < used;
       s += static_cast<unsigned long long>(gridDim.x) * blockDim.x) {
    flags[slot_block[s]] = 1u;
  }
}

__global__ void allocated_list_kernel(const uint32_t* __restrict__ flags, const uint32_t* __restrict__ position,
                                      uint32_t blocks, uint32_t* __restrict__ list) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < blocks && flags[b] != 0u) list[position[b]] = b;
}

// Exclusive scan of n values (or of their popcounts) in blocks of
// kScanBlock; block totals to `sums`.
template <bool Popc>
__global__ void __launch_bounds__(kScanThreads)
    scan_block_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, uint32_t* __restrict__ sums,
                      uint32_t n) {
  __shared__ uint32_t s_warp[kScanThreads / 32];
  const uint32_t first = blockIdx.x * kScanBlock + threadIdx.x * kScanItems;
  uint32_t v[kScanItems], local = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    const uint32_t e = first + i;
    const uint32_t raw = e < n ? in[e] : 0u;
    v[i] = Popc ? static_cast<uint32_t>(__popc(raw)) : raw;
    local += v[i];
  }
  uint32_t prefix;
  const uint32_t total = block_exclusive_scan(local, prefix, s_warp);
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    const uint32_t e = first + i;
    if (e < n) out[e] = prefix;
    prefix += v[i];
  }
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void scan_add_kernel(uint32_t* __restrict__ out, const uint32_t* __restrict__ offsets, uint32_t n) {
  const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < n) out[e] += offsets[e / kScanBlock];
}

// Words of scratch an exclusive scan of n values takes.
size_t scan_scratch(size_t n) {
  size_t words = 0;
  do {
    n = (n + kScanBlock - 1) / kScanBlock;
    words += 2 * n;
  } while (n > 1);
  return words;
}

// Exclusive scan of `n` > 0 device values (popcounts when `popc`) into `out`;
// returns where on the device the total is.  Recursive over the block totals.
const uint32_t* exclusive_scan(const uint32_t* in, uint32_t* out, uint32_t n, bool popc, uint32_t* scratch,
                               cudaStream_t s) {
  const uint32_t blocks = ceil_div(n, kScanBlock);
  uint32_t* sums = scratch;
  uint32_t* offsets = scratch + blocks;
  if (popc) {
    scan_block_kernel<true><<<blocks, kScanThreads, 0, s>>>(in, out, sums, n);
  } else {
    scan_block_kernel<false><<<blocks, kScanThreads, 0, s>>>(in, out, sums, n);
  }
  check(cudaGetLastError(), "scan_block_kernel launch");
  if (blocks == 1) return sums;
  const uint32_t* total = exclusive_scan(sums, offsets, blocks, false, scratch + 2 * static_cast<size_t>(blocks), s);
  scan_add_kernel<<<ceil_div(n, 256), 256, 0, s>>>(out, offsets, n);
  check(cudaGetLastError(), "scan_add_kernel launch");
  return total;
}

// Bit of every edge's first use.
__global__ void mark_first_use_kernel(const uint32_t* __restrict__ first_use, uint32_t* __restrict__ use_words,
                                      uint32_t vertices) {
  const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= vertices) return;
  const uint32_t p = first_use[id];
  atomicOr(use_words + (p >> 5), 1u << (p & 31u));
}

// Triangle corners a vertex can have: its edge is shared by four cells of at
// most five triangles each.
constexpr uint32_t kMaxIncident = 20;
constexpr uint32_t kHasNormal = 0x80000000u;

// MeshBuilder::vertex_on_edge (marching_cubes.cpp:403-437), one thread per
// crossed edge; vertex number = rank of the edge's first use.  `incident`
// starts the count of a vertex's triangles: 0 for one without a gradient
// normal, kHasNormal otherwise.
template <int Kind>
__global__ void __launch_bounds__(128)
    mc_vertex_kernel(VolumeDev v, const uint32_t* __restrict__ slot_block,
                     const unsigned long long* __restrict__ edge_of, const uint32_t* __restrict__ first_use,
                     const uint32_t* __restrict__ use_words, const uint32_t* __restrict__ use_first, uint32_t vertices,
                     float* __restrict__ positions, float* __restrict__ normals, float* __restrict__ colors,
                     uint32_t* __restrict__ vertex_of, uint32_t* __restrict__ incident) {
  const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= vertices) return;
  using VT = VoxelTraits<Kind>;
  const auto* voxels = reinterpret_cast<const typename VT::Raw*>(v.voxels);
  const Sampler<Kind> s{v};
  const unsigned long long key = edge_of[id];
  const uint32_t axis = static_cast<uint32_t>(key % 3ull);
  const unsigned long long stored = key / 3ull;
  const uint32_t slot = static_cast<uint32_t>(stored >> 9), local = static_cast<uint32_t>(stored & 511ull);
  const uint32_t block = slot_block != nullptr ? slot_block[slot] : slot;
  const uint32_t nx = (block % v.bx) * 8u + (local & 7u), ny = ((block / v.bx) % v.by) * 8u + ((local >> 3) & 7u),
                 nz = (block / (v.bx * v.by)) * 8u + (local >> 6);
  const uint32_t fx = nx + (axis == 0), fy = ny + (axis == 1), fz = nz + (axis == 2);
  const float near_value = VT::tsdf(__ldg(voxels + storage_index(v, nx, ny, nz)));
  const float far_value = VT::tsdf(__ldg(voxels + storage_index(v, fx, fy, fz)));
  const f3 near_point = cell_center(v, nx, ny, nz);
  const f3 far_point = cell_center(v, fx, fy, fz);
  const float fraction = -near_value / (far_value - near_value);
  const f3 position = near_point + ((far_point - near_point) * fraction);
  f3 normal;
  const bool has_normal = s.central_normal(position, KF_CORNERS_SKIP_MISSING, normal);
  if (!has_normal) normal = make(0.0f, 0.0f, 0.0f);
  f3 color;
  if (!s.color(position, color)) color = make(255.0f, 255.0f, 255.0f);
  const uint32_t p = first_use[id];
  const uint32_t vi = use_first[p >> 5] + __popc(use_words[p >> 5] & ((1u << (p & 31u)) - 1u));
  store3(positions + static_cast<size_t>(vi) * 3, position);
  store3(normals + static_cast<size_t>(vi) * 3, normal);
  store3(colors + static_cast<size_t>(vi) * 3, color);
  vertex_of[id] = vi;
  incident[vi] = has_normal ? kHasNormal : 0u;
}

// Triangle corners as vertex numbers; each vertex without a normal collects
// its triangles.
__global__ void mc_triangle_kernel(const uint32_t* __restrict__ corner_edge, const uint32_t* __restrict__ vertex_of,
                                   uint32_t* __restrict__ triangles, uint32_t corners,
                                   uint32_t* __restrict__ incident, uint32_t* __restrict__ incident_list) {
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= corners) return;
  const uint32_t vi = vertex_of[corner_edge[q]];
  triangles[q] = vi;
  if (__ldcg(incident + vi) & kHasNormal) return;
  const uint32_t at = atomicAdd(incident + vi, 1u);
  if (at < kMaxIncident) incident_list[static_cast<size_t>(vi) * kMaxIncident + at] = q / 3u;
}

// MeshBuilder::fill_missing_normals (marching_cubes.cpp:441-456): the face
// normals of the vertex's triangles, added in triangle order.
__global__ void mc_fill_normals_kernel(const float* __restrict__ positions, const uint32_t* __restrict__ triangles,
                                       const uint32_t* __restrict__ incident,
                                       const uint32_t* __restrict__ incident_list, uint32_t vertices,
                                       float* __restrict__ normals) {
  const uint32_t vi = blockIdx.x * blockDim.x + threadIdx.x;
  if (vi >= vertices || (incident[vi] & kHasNormal)) return;
  const uint32_t n = min(incident[vi], kMaxIncident);
  const uint32_t* list = incident_list + static_cast<size_t>(vi) * kMaxIncident;
  f3 acc = make(0.0f, 0.0f, 0.0f);
  // ascending triangle numbers; a triangle with the vertex twice counts twice
  long long previous = -1;
  for (uint32_t taken = 0; taken < n;) {
    uint32_t next = 0xFFFFFFFFu, times = 0u;
    for (uint32_t i = 0; i < n; ++i) {
      const uint32_t t = list[i];
      if (static_cast<long long>(t) <= previous) continue;
      if (t < next) {
        next = t;
        times = 0u;
      }
      if (t == next) ++times;
    }
    const uint32_t* tr = triangles + static_cast<size_t>(next) * 3u;
    const f3 p0 = ldg3(positions + static_cast<size_t>(tr[0]) * 3u);
    const f3 face = cross(ldg3(positions + static_cast<size_t>(tr[1]) * 3u) - p0,
                          ldg3(positions + static_cast<size_t>(tr[2]) * 3u) - p0);
    for (uint32_t i = 0; i < times; ++i) acc = acc + face;
    taken += times;
    previous = next;
  }
  const float length = norm(acc);
  store3(normals + static_cast<size_t>(vi) * 3u, length > 0.0f ? acc / length : make(0.0f, 0.0f, 0.0f));
}

// Working arrays of one extraction, cut from a buffer of the pipeline's.
struct Scratch {
  uint8_t* next;
  template <typename T>
  T* take(size_t n) {
    T* p = reinterpret_cast<T*>(next);
    next += (n * sizeof(T) + 255) / 256 * 256;
    return p;
  }
  static size_t bytes(size_t n) { return (n * sizeof(uint32_t) + 255) / 256 * 256; }  // n words
};

// What a pipeline keeps of the working memory after a call: this much device
// memory in all and this much page-locked memory.  The rest is given back.
constexpr size_t kMeshKeepBytes = size_t{256} << 20;
constexpr size_t kMeshStageBytes = size_t{64} << 20;

void reserve(DeviceArray<uint8_t>& buffer, size_t bytes) {
  if (buffer.count < bytes) buffer.resize(bytes);
}

// Gives back what a pipeline should not keep.
struct TrimMeshBuffers {
  Pipeline& p;
  ~TrimMeshBuffers() {
    if (p.mesh_cells.count > kMeshKeepBytes) p.mesh_cells.release();
    if (p.mesh_cells.count + p.mesh_surface.count > kMeshKeepBytes) p.mesh_surface.release();
  }
};

template <int Kind>
void extract_typed(Pipeline& p, float min_weight, kf_mesh& out, cudaStream_t s) {
  const VolumeDev& v = p.view;
  const bool sparse = v.table != nullptr;
  const TrimMeshBuffers trim{p};
  // before the first integration every voxel is unobserved: no surface
  if (!sparse && p.brick_class.count == 0) return;
  const uint4* stencil = reinterpret_cast<const uint4*>(p.stencil_bits.ptr);

  // units: rows of cells (dense) or allocated blocks in block order (sparse)
  uint32_t units = (v.ry - 1) * (v.rz - 1);
  unsigned long long stored = p.voxel_count;  // voxels an edge's near corner can be
  DeviceArray<uint32_t> block_list;
  if (sparse) {
    const uint32_t blocks = v.bx * v.by * v.bz;
    DeviceArray<uint32_t> flags(blocks), position(blocks), scan(scan_scratch(blocks));
    check(cudaMemsetAsync(flags.ptr, 0, flags.bytes(), s), "allocated flags");
    allocated_flags_kernel<<<148 * 4, 256, 0, s>>>(p.slot_block.ptr, p.allocated.ptr, p.sparse_capacity, flags.ptr);
    check(cudaGetLastError(), "allocated_flags_kernel launch");
    const uint32_t* total = exclusive_scan(flags.ptr, position.ptr, blocks, false, scan.ptr, s);
    check(cudaMemcpyAsync(&units, total, sizeof(units), cudaMemcpyDeviceToHost, s), "allocated total");
    check(cudaStreamSynchronize(s), "allocated total");
    if (units == 0) return;
    block_list.resize(units);
    allocated_list_kernel<<<ceil_div(blocks, 256), 256, 0, s>>>(flags.ptr, position.ptr, blocks, block_list.ptr);
    check(cudaGetLastError(), "allocated_list_kernel launch");
    check(cudaStreamSynchronize(s), "allocated list");  // before the scratch arrays go
    stored = static_cast<unsigned long long>(units) * 512ull;  // the slots handed out
  }
  // edge keys: storage index of the near voxel * 3 + axis
  const unsigned long long words64 = (stored * 3ull + 31ull) / 32ull;
  if (words64 > 0xFFFFFFFFull) throw Unsupported("volume too large for the device mesher");
  const uint32_t words = static_cast<uint32_t>(words64);
  const size_t scan_words = std::max(scan_scratch(words), scan_scratch(units));
  reserve(p.mesh_cells, 2 * Scratch::bytes(words) + 2 * Scratch::bytes(units) + 2 * Scratch::bytes(scan_words));
  Scratch cells{p.mesh_cells.ptr};
  uint32_t* edge_words = cells.take<uint32_t>(words);
  uint32_t* word_first = cells.take<uint32_t>(words);
  uint32_t* unit_tris = cells.take<uint32_t>(units);
  uint32_t* unit_first = cells.take<uint32_t>(units);
  uint32_t* scan_units = cells.take<uint32_t>(scan_words);
  uint32_t* scan_edges = cells.take<uint32_t>(scan_words);
  check(cudaMemsetAsync(edge_words, 0, static_cast<size_t>(words) * sizeof(uint32_t), s), "mesh edge bits");
  const unsigned row_ctas = ceil_div(units, kRowThreads / 32);
  if (sparse) {
    mc_blocks_kernel<Kind, false><<<units, 512, 0, s>>>(v, block_list.ptr, min_weight, edge_words, unit_tris, nullptr,
                                                         nullptr, nullptr, nullptr, nullptr);
  } else {
    mc_rows_kernel<Kind, false><<<row_ctas, kRowThreads, 0, s>>>(v, stencil, min_weight, edge_words, unit_tris,
                                                                 nullptr, nullptr, nullptr, nullptr, nullptr);
  }
  check(cudaGetLastError(), "mesh cell pass launch");
  const uint32_t* d_triangles = exclusive_scan(unit_tris, unit_first, units, false, scan_units, s);
  const uint32_t* d_vertices = exclusive_scan(edge_words, word_first, words, true, scan_edges, s);
  uint32_t triangles = 0, vertices = 0;
  check(cudaMemcpyAsync(&triangles, d_triangles, sizeof(uint32_t), cudaMemcpyDeviceToHost, s), "mesh totals");
  check(cudaMemcpyAsync(&vertices, d_vertices, sizeof(uint32_t), cudaMemcpyDeviceToHost, s), "mesh totals");
  check(cudaStreamSynchronize(s), "mesh totals");
  if (triangles == 0 || vertices == 0) return;
  if (static_cast<unsigned long long>(triangles) * 3ull > 0xFFFFFFFFull) throw Unsupported("mesh too large");
  const uint32_t corners = triangles * 3u;
  const uint32_t use_words_n = ceil_div(corners, 32u);
  const size_t three = static_cast<size_t>(vertices) * 3;
  const size_t incident_words = static_cast<size_t>(vertices) * kMaxIncident;
  reserve(p.mesh_surface, 2 * Scratch::bytes(corners) + 3 * Scratch::bytes(vertices) + Scratch::bytes(2 * vertices) +
                              2 * Scratch::bytes(use_words_n) + Scratch::bytes(scan_scratch(use_words_n)) +
                              3 * Scratch::bytes(three) + Scratch::bytes(incident_words));
  Scratch surface{p.mesh_surface.ptr};
  uint32_t* corner_edge = surface.take<uint32_t>(corners);
  uint32_t* first_use = surface.take<uint32_t>(vertices);
  uint32_t* vertex_of = surface.take<uint32_t>(vertices);
  uint32_t* incident = surface.take<uint32_t>(vertices);
  auto* edge_of = surface.take<unsigned long long>(vertices);
  uint32_t* use_words = surface.take<uint32_t>(use_words_n);
  uint32_t* use_first = surface.take<uint32_t>(use_words_n);
  uint32_t* scan_use = surface.take<uint32_t>(scan_scratch(use_words_n));
  float* positions = surface.take<float>(three);
  float* normals = surface.take<float>(three);
  float* colors = surface.take<float>(three);
  uint32_t* tris = surface.take<uint32_t>(corners);
  uint32_t* incident_list = surface.take<uint32_t>(incident_words);
  check(cudaMemsetAsync(first_use, 0xFF, static_cast<size_t>(vertices) * sizeof(uint32_t), s), "mesh first use");
  if (sparse) {
    mc_blocks_kernel<Kind, true><<<units, 512, 0, s>>>(v, block_list.ptr, min_weight, edge_words, nullptr, unit_first,
                                                        word_first, corner_edge, first_use, edge_of);
  } else {
    mc_rows_kernel<Kind, true><<<row_ctas, kRowThreads, 0, s>>>(v, stencil, min_weight, edge_words, nullptr,
                                                                unit_first, word_first, corner_edge, first_use,
                                                                edge_of);
  }
  check(cudaGetLastError(), "mesh corner pass launch");
  check(cudaMemsetAsync(use_words, 0, static_cast<size_t>(use_words_n) * sizeof(uint32_t), s), "mesh use bits");
  mark_first_use_kernel<<<ceil_div(vertices, 256), 256, 0, s>>>(first_use, use_words, vertices);
  check(cudaGetLastError(), "mark_first_use_kernel launch");
  exclusive_scan(use_words, use_first, use_words_n, true, scan_use, s);
  mc_vertex_kernel<Kind><<<ceil_div(vertices, 128), 128, 0, s>>>(
      v, sparse ? p.slot_block.ptr : nullptr, edge_of, first_use, use_words, use_first, vertices, positions, normals,
      colors, vertex_of, incident);
  check(cudaGetLastError(), "mc_vertex_kernel launch");
  mc_triangle_kernel<<<ceil_div(corners, 256), 256, 0, s>>>(corner_edge, vertex_of, tris, corners, incident,
                                                            incident_list);
  check(cudaGetLastError(), "mc_triangle_kernel launch");
  mc_fill_normals_kernel<<<ceil_div(vertices, 128), 128, 0, s>>>(positions, tris, incident, incident_list, vertices,
                                                                 normals);
  check(cudaGetLastError(), "mc_fill_normals_kernel launch");
  // to the host, through page-locked staging unless the mesh is larger than it
  const size_t vertex_bytes = three * sizeof(float), triangle_bytes = static_cast<size_t>(corners) * sizeof(uint32_t);
  const bool stage = 3 * vertex_bytes + triangle_bytes <= kMeshStageBytes;
  if (stage) p.mesh_staging.resize(3 * vertex_bytes + triangle_bytes);
  uint8_t* staged = p.mesh_staging.ptr;
  out.vertex_count = vertices;
  out.triangle_count = triangles;
  struct Part {
    const void* device;
    void** host;
    size_t bytes;
  };
  const Part parts[4] = {{positions, reinterpret_cast<void**>(&out.positions), vertex_bytes},
                         {normals, reinterpret_cast<void**>(&out.normals), vertex_bytes},
                         {colors, reinterpret_cast<void**>(&out.colors), vertex_bytes},
                         {tris, reinterpret_cast<void**>(&out.triangles), triangle_bytes}};
  if (stage) {
    for (const Part& part : parts) {
      check(cudaMemcpyAsync(staged, part.device, part.bytes, cudaMemcpyDeviceToHost, s), "mesh copy");
      staged += part.bytes;
    }
  }
  bool allocated = true;
  for (const Part& part : parts) {
    *part.host = std::malloc(part.bytes);
    allocated = allocated && *part.host != nullptr;
  }
  if (!allocated) {
    cudaStreamSynchronize(s);
    throw CudaError("host allocation failed");
  }
  if (!stage) {
    for (const Part& part : parts) {
      check(cudaMemcpyAsync(*part.host, part.device, part.bytes, cudaMemcpyDeviceToHost, s), "mesh copy");
    }
  }
  check(cudaStreamSynchronize(s), "mesh copy");
  if (!stage) return;
  staged = p.mesh_staging.ptr;
  for (const Part& part : parts) {
    std::memcpy(*part.host, staged, part.bytes);
    staged += part.bytes;
  }
}

}  // namespace

void extract_mesh(Pipeline& p, float min_weight, kf_mesh& out) {
  std::memset(&out, 0, sizeof(out));
  if (p.view.rx < 2 || p.view.ry < 2 || p.view.rz < 2) return;
  const std::lock_guard<std::mutex> lock(p.reading);  // the working arrays are the pipeline's
  const cudaStream_t s = p.stream;
  try {
    switch (p.config.voxel) {
      case KF_VOXEL_QUANTIZED:
        extract_typed<KF_VOXEL_QUANTIZED>(p, min_weight, out, s);
        break;
      case KF_VOXEL_BF16:
        extract_typed<KF_VOXEL_BF16>(p, min_weight, out, s);
        break;
      default:
        extract_typed<KF_VOXEL_FLOAT>(p, min_weight, out, s);
        break;
    }
  } catch (...) {
    std::free(out.positions);
    std::free(out.normals);
    std::free(out.colors);
    std::free(out.triangles);
    std::memset(&out, 0, sizeof(out));
    throw;
  }
}

}  // namespace kf
