// Soup -> indexed weld and the watertight gate on the device (weldPositions,
// src/io/mesh_weld.cpp:26-48; isWatertight, src/io/mesh_validate.cpp:21-59), so that large soups
// are welded where they already are.
//
// Weld: every position gets the lattice key lround(p / cell) per axis (FP32 division, round half
// away from zero, as std::lround) and goes into an open-addressing table of position indices; a
// position that meets an equal key lowers the slot to the smaller index, so in the end a slot holds
// its key's first occurrence whatever the order of the atomics. An exclusive scan of the
// first-occurrence flags in position order numbers the unique keys as the reference does (a hash
// map filled in position order). The gate needs no numbers: the first occurrence itself stands for
// the welded vertex.
//
// Watertight: every undirected edge of a non-degenerate triangle goes into a table of 64-bit keys
// with a use count beside each; the running numbers of edges used once (boundary) and more than
// twice (non-manifold) follow from the count each use finds.
//
// The gate of a batch is three launches and one read back. As three radix sorts over the
// lattice keys and one over the edges it was 40-80 launches and four read backs a mesh: a bake of
// 1,280 triangles at 32^3 531 -> 322 us, occupancy of 81,920 triangles at 256^3 790 -> 375 us, a
// 64-mesh batch 146 -> 119 ms. A table has at least twice (positions) or 4/3 (edges) as many slots
// as keys; what bounds the kernels is the rate of scattered L2 accesses.
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstring>
#include <vector>

#include "api_internal.h"
#include "common.cuh"
#include "host_mesh.h"
#include "kernels.h"

using namespace sdfb;

namespace {

constexpr int kThreads = 256;
constexpr uint32_t kVertsPerBlock = 1024, kTrisPerBlock = 512;
constexpr uint32_t kNone = ~0u;

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

inline unsigned grid_for(uint64_t n, int num_sms) {
  return static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>((n + kThreads - 1) / kThreads,
                                                                         uint64_t(num_sms) * 16)));
}

inline uint64_t pow2_at_least(uint64_t n) {
  uint64_t p = 64;
  while (p < n) p <<= 1;
  return p;
}

// The 64-bit finalizer of MurmurHash3 (Appleby).
__device__ __forceinline__ uint64_t mix64(uint64_t x) {
  x ^= x >> 33;
  x *= 0xff51afd7ed558ccdull;
  x ^= x >> 33;
  x *= 0xc4ceb9fe1a85ec53ull;
  return x ^ (x >> 33);
}

struct LatticeKey {
  long long x, y, z;
};
__device__ __forceinline__ LatticeKey lattice_key(const float *__restrict__ pos, uint64_t i, float cell) {
  return {llroundf(__fdiv_rn(pos[3 * i], cell)), llroundf(__fdiv_rn(pos[3 * i + 1], cell)),
          llroundf(__fdiv_rn(pos[3 * i + 2], cell))};
}

// Puts position i into the table; returns its slot. A slot, once taken, keeps its key.
__device__ __forceinline__ uint32_t weld_insert(const float *__restrict__ pos, uint32_t i, float cell, uint32_t *tab,
                                                uint32_t mask) {
  const LatticeKey k = lattice_key(pos, i, cell);
  uint32_t h = static_cast<uint32_t>(
                   mix64(mix64(mix64(uint64_t(k.x)) ^ uint64_t(k.y)) ^ uint64_t(k.z))) & mask;
  for (;;) {  // there are more slots than positions: a free or an equal one comes
    uint32_t j = *const_cast<volatile uint32_t *>(tab + h);
    if (j == kNone) j = atomicCAS(tab + h, kNone, i);
    if (j == kNone || j == i) return h;
    const LatticeKey o = lattice_key(pos, j, cell);
    if (o.x == k.x && o.y == k.y && o.z == k.z) {
      if (i < j) atomicMin(tab + h, i);
      return h;
    }
    h = (h + 1) & mask;
  }
}

// Counts one use of edge (a, b); bnd and nm follow the edges used once and more than twice. The
// counts start at ~0.
__device__ __forceinline__ void edge_insert(uint32_t a, uint32_t b, unsigned long long *keys, uint32_t *count,
                                            uint64_t mask, int &bnd, int &nm) {
  const unsigned long long key = (static_cast<unsigned long long>(min(a, b)) << 32) | max(a, b);
  uint64_t h = mix64(key) & mask;
  for (;;) {  // at most three quarters of the slots are taken
    unsigned long long k = *const_cast<volatile unsigned long long *>(keys + h);
    if (k == ~0ull) {
      k = atomicCAS(keys + h, ~0ull, key);
      if (k == ~0ull) k = key;
    }
    if (k == key) break;
    h = (h + 1) & mask;
  }
  const uint32_t before = atomicAdd(count + h, 1u) + 1u;
  bnd += before == 0 ? 1 : (before == 1 ? -1 : 0);
  nm += before == 2;
}

// Adds the block's sums to two counters that start at ~0.
__device__ __forceinline__ void add_counts(int bnd, int nm, unsigned long long *counts) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    bnd += __shfl_xor_sync(kFull, bnd, o);
    nm += __shfl_xor_sync(kFull, nm, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (bnd) atomicAdd(counts, static_cast<unsigned long long>(static_cast<long long>(bnd)));
    if (nm) atomicAdd(counts + 1, static_cast<unsigned long long>(nm));
  }
}

// ---- the gate of a batch of indexed meshes ------------------------------------------------------

struct GateRec {
  const float *verts;
  const uint32_t *idx;
  uint32_t V, T;
  uint32_t vblock, tblock;    // first thread block over the mesh's vertices / triangles
  uint32_t vmask;
  uint64_t emask;
  uint32_t *bounds;           // 6: ordered minima, complements of the ordered maxima
  uint32_t *vtab, *slot;
  unsigned long long *ekeys;
  uint32_t *ecount;
  unsigned long long *result;  // boundary and non-manifold edges, 0 in the third when an index is bad (all + 1)
};

// The mesh of a thread block: the last whose first block is not after it.
template <uint32_t GateRec::*FIRST> __device__ __forceinline__ const GateRec &gate_rec(const GateRec *r, int n) {
  int lo = 0, hi = n;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (r[mid].*FIRST <= blockIdx.x) lo = mid;
    else hi = mid;
  }
  return r[lo];
}

__global__ __launch_bounds__(kThreads) void k_gate_bounds(const GateRec *__restrict__ recs, int n) {
  __shared__ uint32_t s_min[kThreads / kWarp][6];
  const GateRec &R = gate_rec<&GateRec::vblock>(recs, n);
  const uint64_t base = uint64_t(blockIdx.x - R.vblock) * kVertsPerBlock;
  uint32_t v[6] = {~0u, ~0u, ~0u, ~0u, ~0u, ~0u};
#pragma unroll
  for (uint32_t k = 0; k < kVertsPerBlock / kThreads; ++k) {
    const uint64_t i = base + k * kThreads + threadIdx.x;
    if (i >= R.V) break;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const uint32_t u = float_to_ordered(__ldg(R.verts + 3 * i + a));
      v[a] = min(v[a], u);
      v[3 + a] = min(v[3 + a], ~u);
    }
  }
#pragma unroll
  for (int a = 0; a < 6; ++a) {
    v[a] = __reduce_min_sync(kFull, v[a]);
    if ((threadIdx.x & 31) == 0) s_min[threadIdx.x >> 5][a] = v[a];
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    uint32_t m = ~0u;
    for (int w = 0; w < kThreads / kWarp; ++w) m = min(m, s_min[w][threadIdx.x]);
    atomicMin(R.bounds + threadIdx.x, m);
  }
}

// weld_cell (host_mesh.cpp) of the vertices' bounds, with its roundings.
__device__ __forceinline__ float gate_cell(const uint32_t *__restrict__ b) {
  float e[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) e[a] = __fsub_rn(ordered_to_float(~b[3 + a]), ordered_to_float(b[a]));
  const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(e[0], e[0]), __fmul_rn(e[1], e[1])), __fmul_rn(e[2], e[2]));
  const float cell = __fmul_rn(__fsqrt_rn(d2), 1e-5f);
  return cell < 1e-6f ? 1e-6f : cell;
}

__global__ __launch_bounds__(kThreads) void k_gate_weld(const GateRec *__restrict__ recs, int n) {
  const GateRec &R = gate_rec<&GateRec::vblock>(recs, n);
  const uint64_t base = uint64_t(blockIdx.x - R.vblock) * kVertsPerBlock;
  const float cell = gate_cell(R.bounds);
#pragma unroll
  for (uint32_t k = 0; k < kVertsPerBlock / kThreads; ++k) {
    const uint64_t i = base + k * kThreads + threadIdx.x;
    if (i < R.V) R.slot[i] = weld_insert(R.verts, static_cast<uint32_t>(i), cell, R.vtab, R.vmask);
  }
}

__global__ __launch_bounds__(kThreads) void k_gate_edges(const GateRec *__restrict__ recs, int n) {
  const GateRec &R = gate_rec<&GateRec::tblock>(recs, n);
  const uint64_t base = uint64_t(blockIdx.x - R.tblock) * kTrisPerBlock;
  int bnd = 0, nm = 0;
#pragma unroll
  for (uint32_t k = 0; k < kTrisPerBlock / kThreads; ++k) {
    const uint64_t t = base + k * kThreads + threadIdx.x;
    if (t >= R.T) continue;
    const uint32_t i[3] = {__ldg(R.idx + 3 * t), __ldg(R.idx + 3 * t + 1), __ldg(R.idx + 3 * t + 2)};
    if (i[0] >= R.V || i[1] >= R.V || i[2] >= R.V) {
      R.result[2] = 0;
      continue;
    }
    const uint32_t a = R.vtab[R.slot[i[0]]], b = R.vtab[R.slot[i[1]]], c = R.vtab[R.slot[i[2]]];
    if (a == b || b == c || c == a) continue;
    edge_insert(a, b, R.ekeys, R.ecount, R.emask, bnd, nm);
    edge_insert(b, c, R.ekeys, R.ecount, R.emask, bnd, nm);
    edge_insert(c, a, R.ekeys, R.ecount, R.emask, bnd, nm);
  }
  add_counts(bnd, nm, R.result);
}

// ---- soups ---------------------------------------------------------------------------------------

__global__ __launch_bounds__(kThreads) void k_weld(const float *__restrict__ pos, uint64_t n, float cell,
                                                   uint32_t *tab, uint32_t mask, uint32_t *__restrict__ slot) {
  for (uint64_t i = uint64_t(blockIdx.x) * kThreads + threadIdx.x; i < n; i += uint64_t(gridDim.x) * kThreads)
    slot[i] = weld_insert(pos, static_cast<uint32_t>(i), cell, tab, mask);
}

__global__ __launch_bounds__(kThreads) void k_first(const uint32_t *__restrict__ tab, uint64_t n,
                                                    const uint32_t *__restrict__ slot, uint32_t *__restrict__ flag) {
  for (uint64_t i = uint64_t(blockIdx.x) * kThreads + threadIdx.x; i < n; i += uint64_t(gridDim.x) * kThreads)
    flag[i] = tab[slot[i]] == i ? 1u : 0u;
}

// welded[i]: the number of the first position with i's key; unique (optional): the first positions.
__global__ __launch_bounds__(kThreads) void k_assign(const float *__restrict__ pos, uint64_t n,
                                                     const uint32_t *__restrict__ tab,
                                                     const uint32_t *__restrict__ slot,
                                                     const uint64_t *__restrict__ number,
                                                     uint32_t *__restrict__ welded, float *__restrict__ unique) {
  for (uint64_t i = uint64_t(blockIdx.x) * kThreads + threadIdx.x; i < n; i += uint64_t(gridDim.x) * kThreads) {
    const uint32_t first = tab[slot[i]];
    const uint64_t id = number[first];
    welded[i] = static_cast<uint32_t>(id);
    if (unique && first == i) {
      unique[3 * id] = pos[3 * i];
      unique[3 * id + 1] = pos[3 * i + 1];
      unique[3 * id + 2] = pos[3 * i + 2];
    }
  }
}

__global__ __launch_bounds__(kThreads) void k_census(const uint32_t *__restrict__ w, uint64_t T,
                                                     unsigned long long *keys, uint32_t *count, uint64_t mask,
                                                     unsigned long long *result) {
  int bnd = 0, nm = 0;
  for (uint64_t t0 = uint64_t(blockIdx.x) * kThreads; t0 < T; t0 += uint64_t(gridDim.x) * kThreads) {
    const uint64_t t = t0 + threadIdx.x;
    if (t >= T) continue;
    const uint32_t a = w[3 * t], b = w[3 * t + 1], c = w[3 * t + 2];
    if (a == b || b == c || c == a) continue;
    edge_insert(a, b, keys, count, mask, bnd, nm);
    edge_insert(b, c, keys, count, mask, bnd, nm);
    edge_insert(c, a, keys, count, mask, bnd, nm);
  }
  add_counts(bnd, nm, result);
}

__global__ __launch_bounds__(kThreads) void k_iota(uint32_t *__restrict__ v, uint64_t n) {
  for (uint64_t i = uint64_t(blockIdx.x) * kThreads + threadIdx.x; i < n; i += uint64_t(gridDim.x) * kThreads)
    v[i] = static_cast<uint32_t>(i);
}

// Slot numbers are 32 bits: with 2^31 positions and more the table fills further, never up.
uint64_t weld_slots(uint64_t n) { return std::min<uint64_t>(pow2_at_least(2 * n), 1ull << 32); }
uint64_t edge_slots(uint64_t T) { return pow2_at_least(4 * T); }

}  // namespace

namespace sdfb {

cudaError_t iota_device(uint32_t *v, uint64_t n, int num_sms, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  k_iota<<<grid_for(n, num_sms), kThreads, 0, st>>>(v, n);
  note_launch();
  return cudaGetLastError();
}

// Layout: slot | flag | number | table, scan scratch.
size_t weld_temp_bytes(uint64_t n) {
  return 2 * align256(n * 4) + align256((n + 1) * 8) + align256(weld_slots(n) * 4) + scan_scratch_bytes(n);
}

cudaError_t weld_enqueue(const float *pos, uint64_t n, float cell, uint32_t *welded, float *unique, void *temp,
                         size_t temp_bytes, const uint64_t **num_unique, int num_sms, cudaStream_t st) {
  if (n == 0 || n >= (1ull << 32)) return cudaErrorInvalidValue;
  if (temp_bytes < weld_temp_bytes(n)) return cudaErrorMemoryAllocation;
  char *p = static_cast<char *>(temp);
  auto take = [&](size_t bytes) {
    char *r = p;
    p += align256(bytes);
    return r;
  };
  uint32_t *slot = reinterpret_cast<uint32_t *>(take(n * 4));
  uint32_t *flag = reinterpret_cast<uint32_t *>(take(n * 4));
  uint64_t *number = reinterpret_cast<uint64_t *>(take((n + 1) * 8));
  const uint64_t slots = weld_slots(n);
  uint32_t *tab = reinterpret_cast<uint32_t *>(take(slots * 4));
  const Scratch scratch{p, temp_bytes - size_t(p - static_cast<char *>(temp))};
  cudaError_t e = cudaMemsetAsync(tab, 0xff, slots * 4, st);
  if (e != cudaSuccess) return e;
  k_weld<<<grid_for(n, num_sms), kThreads, 0, st>>>(pos, n, cell, tab, static_cast<uint32_t>(slots - 1), slot);
  note_launch();
  k_first<<<grid_for(n, num_sms), kThreads, 0, st>>>(tab, n, slot, flag);
  note_launch();
  if ((e = exclusive_scan_u32(flag, number, n, scratch, st)) != cudaSuccess) return e;
  k_assign<<<grid_for(n, num_sms), kThreads, 0, st>>>(pos, n, tab, slot, number, welded, unique);
  note_launch();
  *num_unique = number + n;
  return cudaGetLastError();
}

cudaError_t weld_device(const float *pos, uint64_t n, float cell, uint32_t *welded, void *temp, size_t temp_bytes,
                        uint32_t *num_unique, int num_sms, cudaStream_t st) {
  *num_unique = 0;
  if (n == 0) return cudaSuccess;
  const uint64_t *d_count = nullptr;
  cudaError_t e = weld_enqueue(pos, n, cell, welded, nullptr, temp, temp_bytes, &d_count, num_sms, st);
  if (e != cudaSuccess) return e;
  uint64_t total = 0;
  if ((e = cudaMemcpyAsync(&total, d_count, 8, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
  *num_unique = static_cast<uint32_t>(total);
  return cudaSuccess;
}

// Layout: two counters | keys | counts, all cleared to ~0 by one call.
size_t watertight_temp_bytes(uint64_t T) { return 256 + edge_slots(T) * 12; }

cudaError_t watertight_enqueue(const uint32_t *welded, uint64_t T, void *temp, size_t temp_bytes,
                               const unsigned long long **counts, int num_sms, cudaStream_t st) {
  if (T == 0) return cudaErrorInvalidValue;
  if (temp_bytes < watertight_temp_bytes(T)) return cudaErrorMemoryAllocation;
  const uint64_t slots = edge_slots(T);
  unsigned long long *result = static_cast<unsigned long long *>(temp);
  unsigned long long *keys = result + 32;
  uint32_t *count = reinterpret_cast<uint32_t *>(keys + slots);
  cudaError_t e = cudaMemsetAsync(temp, 0xff, watertight_temp_bytes(T), st);
  if (e != cudaSuccess) return e;
  k_census<<<grid_for(T, num_sms), kThreads, 0, st>>>(welded, T, keys, count, slots - 1, result);
  note_launch();
  *counts = result;
  return cudaGetLastError();
}

cudaError_t watertight_device(const uint32_t *welded, uint64_t T, void *temp, size_t temp_bytes, uint64_t *boundary,
                              uint64_t *nonmanifold, int num_sms, cudaStream_t st) {
  *boundary = *nonmanifold = 0;
  if (T == 0) return cudaSuccess;
  const unsigned long long *counts = nullptr;
  cudaError_t e = watertight_enqueue(welded, T, temp, temp_bytes, &counts, num_sms, st);
  if (e != cudaSuccess) return e;
  unsigned long long h[2];
  if ((e = cudaMemcpyAsync(h, counts, sizeof h, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
  *boundary = h[0] + 1;
  *nonmanifold = h[1] + 1;
  return cudaSuccess;
}

}  // namespace sdfb

// The meshes go through the gate in runs of consecutive ones whose tables fit kGateRoom together (or of one
// mesh), one run after the other in the same memory: without it the tables of a batch, 48 to 96 B a triangle
// and 12 to 20 B a vertex, were held all at once. A batch of 10M triangles is one run; another costs three
// launches and a memset.
constexpr size_t kGateRoom = size_t(1) << 30;

sdfb_status device_gate(sdfb_ctx *ctx, const std::vector<PlanMesh *> &ms, cudaStream_t st, size_t *bad,
                        const std::function<sdfb_status()> &meanwhile) {
  // Records first (uploaded), then the results and bounds and the tables, which start at ~0, and the slots of
  // the vertices.
  const size_t n = ms.size();
  if (n == 0) return SDFB_OK;
  struct Run {
    size_t first, count, cleared;  // meshes, bytes of their tables
    uint32_t vblocks, tblocks;
  };
  std::vector<GateRec> recs(n);
  std::vector<Run> runs;
  const size_t o_result = align256(n * sizeof(GateRec)), o_bounds = o_result + align256(n * 24);
  const size_t o_tables = o_bounds + align256(n * 24);
  size_t total = o_tables;
  for (size_t first = 0; first < n;) {
    uint64_t vblocks = 0, tblocks = 0;
    size_t end = first, tables = 0, slots = 0;
    for (; end < n; ++end) {
      const PlanMesh &p = *ms[end];
      GateRec &r = recs[end];
      const uint64_t vs = weld_slots(p.V), es = edge_slots(p.T);
      const uint64_t vb = vblocks + (uint64_t(p.V) + kVertsPerBlock - 1) / kVertsPerBlock;
      const uint64_t tb = tblocks + (uint64_t(p.T) + kTrisPerBlock - 1) / kTrisPerBlock;
      const size_t need = align256(es * 8) + align256(es * 4) + align256(vs * 4);
      const size_t need_slots = align256(size_t(p.V) * 4);
      if (end > first && (tables + need + slots + need_slots > kGateRoom || vb >= (1ull << 31) || tb >= (1ull << 31))) break;
      r.verts = p.verts;
      r.idx = p.idx;
      r.V = p.V;
      r.T = p.T;
      r.vblock = static_cast<uint32_t>(vblocks);
      r.tblock = static_cast<uint32_t>(tblocks);
      r.vmask = static_cast<uint32_t>(vs - 1);
      r.emask = es - 1;
      // offsets until the buffer is known
      r.ekeys = reinterpret_cast<unsigned long long *>(o_tables + tables);
      r.ecount = reinterpret_cast<uint32_t *>(o_tables + tables + align256(es * 8));
      r.vtab = reinterpret_cast<uint32_t *>(o_tables + tables + align256(es * 8) + align256(es * 4));
      r.slot = reinterpret_cast<uint32_t *>(slots);  // past the run's tables
      tables += need;
      slots += need_slots;
      vblocks = vb;
      tblocks = tb;
    }
    for (size_t m = first; m < end; ++m)
      recs[m].slot = reinterpret_cast<uint32_t *>(reinterpret_cast<size_t>(recs[m].slot) + o_tables + tables);
    runs.push_back(Run{first, end - first, tables, static_cast<uint32_t>(vblocks), static_cast<uint32_t>(tblocks)});
    total = std::max(total, o_tables + tables + slots);
    first = end;
  }
  if (!ctx->weld_tmp.ensure(total))
    return ctx_fail(ctx, SDFB_ERR_OUT_OF_MEMORY, "cannot allocate %zu bytes of device memory", total);
  if (!ctx->gate_pin.ensure(n * sizeof(GateRec) + n * 24)) return ctx_fail(ctx, SDFB_ERR_OUT_OF_MEMORY, "pinned staging");
  char *d = static_cast<char *>(ctx->weld_tmp.p);
  auto fix = [&](auto *&p) { p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(d + reinterpret_cast<size_t>(p)); };
  for (size_t m = 0; m < n; ++m) {
    GateRec &r = recs[m];
    fix(r.ekeys);
    fix(r.ecount);
    fix(r.vtab);
    fix(r.slot);
    r.result = reinterpret_cast<unsigned long long *>(d + o_result + m * 24);
    r.bounds = reinterpret_cast<uint32_t *>(d + o_bounds + m * 24);
  }
  std::memcpy(ctx->gate_pin.p, recs.data(), n * sizeof(GateRec));
  unsigned long long *h = reinterpret_cast<unsigned long long *>(static_cast<char *>(ctx->gate_pin.p) + n * sizeof(GateRec));
  cudaError_t e = cudaMemcpyAsync(d, ctx->gate_pin.p, n * sizeof(GateRec), cudaMemcpyHostToDevice, st);
  for (const Run &run : runs) {
    const GateRec *dr = reinterpret_cast<const GateRec *>(d) + run.first;
    const int k = static_cast<int>(run.count);
    // The first memset takes the results and bounds of all meshes with it.
    const size_t at = run.first == 0 ? o_result : o_tables;
    if (e == cudaSuccess) e = cudaMemsetAsync(d + at, 0xff, o_tables + run.cleared - at, st);
    if (e != cudaSuccess) return ctx_cuda(ctx, e, "gate set-up");
    k_gate_bounds<<<run.vblocks, kThreads, 0, st>>>(dr, k);
    note_launch();
    k_gate_weld<<<run.vblocks, kThreads, 0, st>>>(dr, k);
    note_launch();
    k_gate_edges<<<run.tblocks, kThreads, 0, st>>>(dr, k);
    note_launch();
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, d + o_result, n * 24, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaEventRecord(ctx->gate_done, st);
  const sdfb_status early = meanwhile && e == cudaSuccess ? meanwhile() : SDFB_OK;
  if (e == cudaSuccess) e = cudaEventSynchronize(ctx->gate_done);
  if (early != SDFB_OK) return early;
  if (e != cudaSuccess) return ctx_cuda(ctx, e, "watertight gate");
  for (size_t m = 0; m < n; ++m) {
    if (h[3 * m + 2] != ~0ull) {
      *bad = m;
      return ctx_fail(ctx, SDFB_ERR_BAD_MESH, "triangle index out of range");
    }
    ms[m]->watertight = (h[3 * m] + 1 == 0 && h[3 * m + 1] + 1 == 0) ? 1 : 0;
  }
  return SDFB_OK;
}
