// Expansion of per-triangle work into items (candidate cells or columns) without a device-wide scan.
//
// A thread block takes 256 consecutive triangles (32 of a small mesh): a thread sets up one triangle and
// counts its items, the block scans the counts in shared memory, and its threads take the items in order, each
// finding the owner by binary search in the shared starts and reading the triangle from shared
// memory. A triangle with more than kWarpItems items goes to a list instead; a second kernel gives each
// of those a warp, one with more than kBlockItems a block, or several while there are few, and one with more than
// kGridItems the grid.
// (A block takes as long as its triangles have items: with the list from 4096 items on, the occupancy
// stage of 1280 triangles at 128^3 and 256^3 took 179 and 891 us, now 27 and 45.)
//
// Before, a kernel counted, three launches scanned the counts of all triangles and threads walked the
// device-wide starts from owner to owner: a walk over the empty triangles of a mesh much finer than
// its grid is a serial chain of loads (1M triangles on 128^2 columns 241 us, 157k triangles of a
// mixed batch 260 us, for the column test alone). Now the whole bake of the former takes 6.90 ms for
// 7.10, a 32^3 bake of 960 triangles 291 us for 327 and a 256^3 occupancy grid of 4k triangles 76 us
// for 97.
//
// An Op describes the work:
//   Op::Tri                       the triangle as its items need it, trivially copyable, whole words
//   op.setup(B, t, tri) -> count  the triangle (global index t) and its number of items
//   op.item(B, tri, k)            item k
//   op.finish(B, items)           at the end, by every thread; over the threads, items adds up to those run
// Every thread has its own copy of the op, so item() may keep sums in it for finish().
#pragma once

#include <cstdint>

#include "common.cuh"
#include "kernels.h"

namespace sdfb {

constexpr int kExpandThreads = 256;
// A warp's worth of items and more go to a warp (16: 81,920 triangles at 256^3 37 -> 49 us, 64: eight mixed
// meshes 43 -> 49 us), from 512 to a block (2048: 320 triangles at 128^3 31 -> 48 us).
constexpr uint64_t kWarpItems = 48, kBlockItems = 512, kGridItems = 1 << 18;
constexpr uint64_t kGridList = 1024;
// The triangles for a block are cut into parts where they are fewer than twice the blocks, so that none of
// the blocks is idle and none holds the others up. One block a triangle, parts for one, two, four times the
// blocks, and a device-wide scan of all items as it was once: occupancy stage of a turned box of 12 triangles at
// 128^3 387, 43, 45, 47 and 52 us, of 80 triangles at 256^3 191, 69, 63, 62 and 76, of 200 as large as the grid
// at 128^3 439, 235, 166, 143 and 164, of 320 at 128^3 31, 29, 30, 33 and 29; crossings of the box at 400^3 127,
// 25, 27, 29 and 54.
constexpr unsigned long long kBlockShare = 2;

// Triangles left to the second kernel: those for a warp from the front of `tris`, those for a block from
// its end, those for the grid in a list of their own (as far as it holds them). counts: zero before the
// first kernel.
struct BigList {
  unsigned long long *counts;  // warp, block, grid
  uint64_t *grid;              // kGridList entries
  uint64_t *tris;              // n entries
  uint64_t n;
};

template <class Op, int OWN>
__global__ __launch_bounds__(kExpandThreads) void k_expand(BatchDev B, uint64_t n, BigList big, Op op) {
  using Tri = typename Op::Tri;
  constexpr int kWords = sizeof(Tri) / 4;
  static_assert(sizeof(Tri) % 4 == 0, "a triangle is whole words");
  __shared__ uint32_t s_tri[kWords][OWN];
  __shared__ uint32_t s_start[OWN + 1];
  __shared__ uint32_t s_warp[kExpandThreads / kWarp];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t t = uint64_t(blockIdx.x) * OWN + threadIdx.x;
  uint32_t count = 0;
  if (threadIdx.x < OWN && t < n) {
    Tri tri;
    const uint64_t c = op.setup(B, t, tri);
    if (c > kWarpItems) {
      unsigned long long at = kGridList;
      if (c > kGridItems && (at = atomicAdd(big.counts + 2, 1ull)) < kGridList) big.grid[at] = t;
      if (at >= kGridList) {
        const bool block = c > kBlockItems;
        at = atomicAdd(big.counts + (block ? 1 : 0), 1ull);
        big.tris[block ? n - 1 - at : at] = t;
      }
    } else if (c) {
      count = static_cast<uint32_t>(c);
      const uint32_t *w = reinterpret_cast<const uint32_t *>(&tri);
#pragma unroll
      for (int k = 0; k < kWords; ++k) s_tri[k][threadIdx.x] = w[k];
    }
  }
  uint32_t incl = count;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t x = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += x;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  uint32_t before = 0;
  for (int w = 0; w < warp; ++w) before += s_warp[w];
  if (threadIdx.x < OWN) s_start[threadIdx.x + 1] = before + incl;
  if (threadIdx.x == 0) s_start[0] = 0;
  __syncthreads();
  const uint32_t total = s_start[OWN];
  for (uint32_t w = threadIdx.x; w < total; w += kExpandThreads) {
    int j = 0;  // the last triangle that starts at or before w (an empty one starts where the next does)
#pragma unroll
    for (int step = OWN / 2; step; step >>= 1)
      if (s_start[j + step] <= w) j += step;
    Tri tri;
    uint32_t *x = reinterpret_cast<uint32_t *>(&tri);
#pragma unroll
    for (int k = 0; k < kWords; ++k) x[k] = s_tri[k][j];
    op.item(B, tri, uint64_t(w - s_start[j]));
  }
  __syncwarp();
  op.finish(B, threadIdx.x == 0 ? total : 0);
}

template <class Op>
__global__ __launch_bounds__(kExpandThreads) void k_expand_big(BatchDev B, BigList big, Op op) {
  constexpr int kWarps = kExpandThreads / kWarp;
  const unsigned long long nwarp = big.counts[0], nblock = big.counts[1];
  const unsigned long long ngrid = min(big.counts[2], static_cast<unsigned long long>(kGridList));
  const int lane = threadIdx.x & 31;
  const unsigned long long warp = blockIdx.x * (unsigned long long)kWarps + (threadIdx.x >> 5);
  unsigned long long items = 0;  // of the first lane, or thread, that ran them
  for (unsigned long long i = warp; i < nwarp; i += gridDim.x * (unsigned long long)kWarps) {
    typename Op::Tri tri;
    const uint64_t c = op.setup(B, big.tris[i], tri);
    for (uint64_t k = lane; k < c; k += kWarp) op.item(B, tri, k);
    if (lane == 0) items += c;
  }
  const unsigned long long share = nblock ? max(1ull, kBlockShare * gridDim.x / nblock) : 1;
  for (unsigned long long i = blockIdx.x; i < nblock * share; i += gridDim.x) {
    const unsigned long long t = i / share, part = i - t * share;
    typename Op::Tri tri;
    const uint64_t c = op.setup(B, big.tris[big.n - 1 - t], tri);
    for (uint64_t k = part * kExpandThreads + threadIdx.x; k < c; k += share * kExpandThreads) op.item(B, tri, k);
    if (threadIdx.x == 0 && part == 0) items += c;
  }
  for (unsigned long long i = 0; i < ngrid; ++i) {
    typename Op::Tri tri;
    const uint64_t c = op.setup(B, big.grid[i], tri);
    const uint64_t stride = uint64_t(gridDim.x) * kExpandThreads;
    const uint64_t first = uint64_t(blockIdx.x) * kExpandThreads + threadIdx.x;
    for (uint64_t k = first; k < c; k += stride) op.item(B, tri, k);
    if (first == 0) items += c;
  }
  __syncwarp();
  op.finish(B, items);
}

// Bytes of a list for n triangles, and the list in that memory (counts first; the caller clears them).
inline size_t big_list_bytes(uint64_t n) { return 256 + kGridList * 8 + ((n * 8 + 255) & ~size_t(255)); }
inline BigList big_list(void *mem, uint64_t n) {
  char *p = static_cast<char *>(mem);
  return BigList{reinterpret_cast<unsigned long long *>(p), reinterpret_cast<uint64_t *>(p + 256),
                 reinterpret_cast<uint64_t *>(p + 256 + kGridList * 8), n};
}

template <class Op>
cudaError_t expand(const BatchDev &B, uint64_t n, const BigList &big, const Op &op, int num_sms, cudaStream_t st) {
  // 32 triangles a block where 256 would leave SMs with one block or none: the occupancy stage of 4,096
  // triangles at 64^3 37 -> 20 us.
  if (n < uint64_t(num_sms) * 2 * kExpandThreads)
    k_expand<Op, 32><<<static_cast<unsigned>((n + 31) / 32), kExpandThreads, 0, st>>>(B, n, big, op);
  else
    k_expand<Op, kExpandThreads>
        <<<static_cast<unsigned>((n + kExpandThreads - 1) / kExpandThreads), kExpandThreads, 0, st>>>(B, n, big, op);
  note_launch();
  k_expand_big<Op><<<static_cast<unsigned>(num_sms * 4), kExpandThreads, 0, st>>>(B, big, op);
  note_launch();
  return cudaGetLastError();
}

}  // namespace sdfb
