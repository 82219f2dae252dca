// Dense occupancy: the reference's candidate-cell loop (src/convert/sdf_baker.cpp:89-118), one item
// per (triangle, candidate cell) of the triangle's clamped candidate box (expand.cuh), each running the
// exact-rounding SAT test (common.cuh) and storing 1 for a hit. Several triangles may store 1 into
// the same byte; the stores carry the same value, so no atomics are needed and the result does
// not depend on their order.
#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "expand.cuh"
#include "kernels.h"

namespace sdfb {
namespace {

constexpr int kThreads = 256;

struct TriCells {
  f3 a, b, c;
  int lo[3], hi[3];
  int mesh;
  uint32_t local;  // index within the mesh
};

__device__ __forceinline__ f3 vload(const float *v, uint32_t i) {
  return {__ldg(v + 3ull * i), __ldg(v + 3ull * i + 1), __ldg(v + 3ull * i + 2)};
}

// Triangle t (global) with its mesh's clamped candidate box. Out-of-range indices read vertex 0
// (the bake reports the mesh as bad; reads stay in bounds). A mesh without an occupancy output
// gets an empty box. err (optional): bad indices and non-finite vertices are flagged there.
__device__ __forceinline__ TriCells tri_cells(const BatchDev &B, uint64_t t, uint32_t *err = nullptr) {
  TriCells r;
  r.mesh = find_mesh(B.tri_starts, B.num_meshes, t);
  const MeshRec &M = B.recs[r.mesh];
  const uint64_t lt = t - B.tri_starts[r.mesh];
  r.local = static_cast<uint32_t>(lt);
  const uint32_t V = M.num_verts;
  const uint32_t i0 = __ldg(M.idx + 3 * lt), i1 = __ldg(M.idx + 3 * lt + 1), i2 = __ldg(M.idx + 3 * lt + 2);
  r.a = vload(M.verts, i0 < V ? i0 : 0);
  r.b = vload(M.verts, i1 < V ? i1 : 0);
  r.c = vload(M.verts, i2 < V ? i2 : 0);
  if (err) {
    if (i0 >= V || i1 >= V || i2 >= V) atomic_or_err(err, kErrBadIndex);
    if (!isfinite(r.a.x) || !isfinite(r.a.y) || !isfinite(r.a.z) || !isfinite(r.b.x) || !isfinite(r.b.y) ||
        !isfinite(r.b.z) || !isfinite(r.c.x) || !isfinite(r.c.y) || !isfinite(r.c.z))
      atomic_or_err(err, kErrNonFinite);
  }
  const GridDev &g = M.g;
  const float mn[3] = {min_ref(min_ref(r.a.x, r.b.x), r.c.x), min_ref(min_ref(r.a.y, r.b.y), r.c.y),
                       min_ref(min_ref(r.a.z, r.b.z), r.c.z)};
  const float mx[3] = {max_ref(max_ref(r.a.x, r.b.x), r.c.x), max_ref(max_ref(r.a.y, r.b.y), r.c.y),
                       max_ref(max_ref(r.a.z, r.b.z), r.c.z)};
  const float o[3] = {g.ox, g.oy, g.oz};
  const int nmax[3] = {g.nx - 1, g.ny - 1, g.nz - 1};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    r.lo[k] = cell_index_clamped(mn[k], o[k], g.voxel, nmax[k]);
    r.hi[k] = cell_index_clamped(mx[k], o[k], g.voxel, nmax[k]);
  }
  if (!M.occ) {
    r.lo[0] = 0;
    r.hi[0] = -1;
  }
  return r;
}

// Clears the occupancy grids of the batch (one pass over the global cells). A thread clears 16
// consecutive cells, with one 16-byte store where they lie in one mesh's grid at an aligned
// address (so a warp writes 512 contiguous bytes), else byte by byte. Clears the list's counts too.
__global__ __launch_bounds__(kThreads) void k_occ_clear(BatchDev B, BigList big) {
  if (blockIdx.x == 0 && threadIdx.x < 3) big.counts[threadIdx.x] = 0;
  const uint64_t stride = uint64_t(gridDim.x) * kThreads * 16;
  for (uint64_t c0 = (uint64_t(blockIdx.x) * kThreads + threadIdx.x) * 16; c0 < B.total_cells; c0 += stride) {
    int m = find_mesh(B.cell_starts, B.num_meshes, c0);
    if (c0 + 16 <= B.cell_starts[m + 1]) {
      uint8_t *occ = B.recs[m].occ;
      if (!occ) continue;
      uint8_t *p = occ + (c0 - B.cell_starts[m]);
      if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
        *reinterpret_cast<uint4 *>(p) = make_uint4(0u, 0u, 0u, 0u);
        continue;
      }
    }
    for (uint64_t c = c0; c < c0 + 16 && c < B.total_cells; ++c) {
      while (c >= B.cell_starts[m + 1]) ++m;
      uint8_t *occ = B.recs[m].occ;
      if (occ) occ[c - B.cell_starts[m]] = 0;
    }
  }
}

// Appends of (cell, triangle) hits: a warp-aggregated atomic reserves the slots of the lanes that
// hit together; keys past the capacity are counted but not written.
struct HitSink {
  uint64_t *keys = nullptr;
  uint64_t capacity = 0;
  unsigned long long *count = nullptr;
  int tri_bits = 0;
};

__device__ __forceinline__ void append_hit(const HitSink &h, bool hit, uint64_t key) {
  const unsigned mask = __activemask();
  const unsigned ballot = __ballot_sync(mask, hit);
  if (!ballot) return;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(ballot) - 1;
  unsigned long long base = 0;
  if (lane == leader) base = atomicAdd(h.count, static_cast<unsigned long long>(__popc(ballot)));
  base = __shfl_sync(mask, base, leader);
  if (hit) {
    const unsigned long long pos = base + __popc(ballot & ((1u << lane) - 1u));
    if (pos < h.capacity) h.keys[pos] = key;
  }
}

template <bool FIRST, bool HITS> struct OccOp {
  using Tri = TriCells;
  uint32_t *first_tri;
  unsigned long long *sat_tests;
  uint32_t *err;
  HitSink sink;

  // Candidate cells, as a 64-bit count: a triangle across a large grid can have more than 2^32.
  __device__ __forceinline__ uint64_t setup(const BatchDev &B, uint64_t t, Tri &tri) const {
    tri = tri_cells(B, t, err);
    if (tri.hi[0] < tri.lo[0]) return 0;
    return uint64_t(tri.hi[0] - tri.lo[0] + 1) * uint64_t(tri.hi[1] - tri.lo[1] + 1) *
           uint64_t(tri.hi[2] - tri.lo[2] + 1);
  }
  __device__ __forceinline__ void item(const BatchDev &B, const Tri &tri, uint64_t k) const {
    const MeshRec &M = B.recs[tri.mesh];
    const GridDev &g = M.g;
    const uint32_t sx = tri.hi[0] - tri.lo[0] + 1, sy = tri.hi[1] - tri.lo[1] + 1;
    int dx, dy, dz;
    if ((k >> 32) == 0) {  // 32-bit divisions where they do
      const uint32_t k32 = static_cast<uint32_t>(k), row = k32 / sx;
      dx = static_cast<int>(k32 - row * sx);
      dz = static_cast<int>(row / sy);
      dy = static_cast<int>(row - dz * sy);
    } else {
      dx = static_cast<int>(k % sx);
      dy = static_cast<int>((k / sx) % sy);
      dz = static_cast<int>(k / (uint64_t(sx) * sy));
    }
    const int x = tri.lo[0] + dx, y = tri.lo[1] + dy, z = tri.lo[2] + dz;
    const f3 c = {cell_center(g.ox, x, g.voxel), cell_center(g.oy, y, g.voxel), cell_center(g.oz, z, g.voxel)};
    const bool hit = sat_overlap(c, __fmul_rn(g.voxel, 0.5f), tri.a, tri.b, tri.c);
    const uint64_t cell = (uint64_t(z) * g.ny + y) * g.nx + x;
    if (hit) {
      M.occ[cell] = 1;
      if (FIRST) atomicMin(first_tri + cell, tri.local);
    }
    if (HITS) append_hit(sink, hit, (cell << sink.tri_bits) | tri.local);
  }
  __device__ __forceinline__ void finish(const BatchDev &, unsigned long long items) const {
    if (sat_tests && items) atomicAdd(sat_tests, items);
  }
};

cudaError_t clear(const BatchDev &B, const BigList &big, int num_sms, cudaStream_t st) {
  const uint64_t blocks = std::max<uint64_t>(
      1, std::min<uint64_t>((B.total_cells + kThreads * 16 - 1) / (kThreads * 16), uint64_t(num_sms) * 16));
  k_occ_clear<<<static_cast<unsigned>(blocks), kThreads, 0, st>>>(B, big);
  note_launch();
  return cudaGetLastError();
}

}  // namespace

size_t occupancy_temp_bytes(uint64_t total_tris) { return big_list_bytes(total_tris); }

cudaError_t occupancy_batch(const BatchDev &B, uint32_t *first_tri, void *temp, size_t temp_bytes,
                            unsigned long long *sat_tests, uint32_t *err, int num_sms, cudaStream_t st) {
  const uint64_t T = B.total_tris;
  if (big_list_bytes(T) > temp_bytes) return cudaErrorMemoryAllocation;
  const BigList big = big_list(temp, T);
  cudaError_t e = clear(B, big, num_sms, st);
  if (e != cudaSuccess) return e;
  if (first_tri) {
    if (B.num_meshes != 1) return cudaErrorInvalidValue;
    if ((e = cudaMemsetAsync(first_tri, 0xff, B.total_cells * 4, st)) != cudaSuccess) return e;
  }
  if (T == 0) return cudaSuccess;
  if (first_tri) return expand(B, T, big, OccOp<true, false>{first_tri, sat_tests, err, HitSink()}, num_sms, st);
  return expand(B, T, big, OccOp<false, false>{nullptr, sat_tests, err, HitSink()}, num_sms, st);
}

cudaError_t occupancy_hits(const BatchDev &B, void *temp, size_t temp_bytes, uint64_t *keys, uint64_t capacity,
                           unsigned long long *hit_count, int tri_bits, int num_sms, cudaStream_t st) {
  if (B.num_meshes != 1) return cudaErrorInvalidValue;
  const uint64_t T = B.total_tris;
  if (big_list_bytes(T) > temp_bytes) return cudaErrorMemoryAllocation;
  const BigList big = big_list(temp, T);
  cudaError_t e = cudaMemsetAsync(hit_count, 0, sizeof(unsigned long long), st);
  if (e != cudaSuccess || (e = clear(B, big, num_sms, st)) != cudaSuccess) return e;
  if (T == 0) return cudaSuccess;
  HitSink sink;
  sink.keys = keys;
  sink.capacity = capacity;
  sink.count = hit_count;
  sink.tri_bits = tri_bits;
  return expand(B, T, big, OccOp<false, true>{nullptr, nullptr, nullptr, sink}, num_sms, st);
}

}  // namespace sdfb
