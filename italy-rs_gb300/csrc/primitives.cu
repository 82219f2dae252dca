// Device-wide primitives used by the bake: exclusive scan and a stable LSD radix sort.
//
// Scan: tiles of 4096 counts (256 threads x 16), scanned per block, tile sums scanned
// recursively, then added back.
//
// Radix sort: digits of at most 8 bits, of equal width over the key's bits, in one of two ways.
//   Up to kSmallSort pairs: one launch of one thread block that holds them in registers and trades
//   them through shared memory, pass after pass.
//   More: one launch counts all digits of all keys, and one launch a pass does the rest: a thread
//   block ranks a tile of 2048 pairs, publishes its digit counts, adds up the tiles before it from
//   theirs (decoupled look-back, Merrill and Garland 2016), and writes the pairs, ordered in shared
//   memory first, as runs. The order is the same either way: both are stable.
// A pass reads and writes 24 B a pair, 0.3 us for 82k pairs at the copy rate: what costs is launches
// and the latency inside them. Before, a pass was five launches (counts, three for the scan of their
// matrix, scatter).
#include <algorithm>
#include <cstdint>
#include <utility>

#include "common.cuh"
#include "kernels.h"

namespace sdfb {
namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr size_t kScanTile = size_t(kScanThreads) * kScanItems;

constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;
constexpr size_t kSortTile = size_t(kSortThreads) * kSortItems;
constexpr int kSmallThreads = 1024;
constexpr int kSmallItems = 8;
constexpr size_t kSmallSort = size_t(kSmallThreads) * kSmallItems;
constexpr int kDigits = 256;
constexpr int kMaxPasses = 8;
constexpr int kLookBack = 4;       // tiles whose counts a thread reads at once
constexpr int kMaxPolls = 1 << 16;

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

struct Bump {
  char *p;
  size_t left;
  template <typename T> T *take(size_t count) {
    const size_t b = align256(count * sizeof(T));
    if (b > left) return nullptr;
    T *r = reinterpret_cast<T *>(p);
    p += b;
    left -= b;
    return r;
  }
};

// Block-wide exclusive scan of one uint64 per thread; returns the block total in *total.
__device__ __forceinline__ uint64_t block_exclusive_scan(uint64_t v, uint64_t *total) {
  __shared__ uint64_t warp_tot[kScanThreads / kWarp];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t n = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += n;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint64_t w = lane < kScanThreads / kWarp ? warp_tot[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t n = __shfl_up_sync(kFull, w, o);
      if (lane >= o) w += n;
    }
    if (lane < kScanThreads / kWarp) warp_tot[lane] = w;  // inclusive warp prefix
  }
  __syncthreads();
  const uint64_t warp_base = warp ? warp_tot[warp - 1] : 0;
  *total = warp_tot[kScanThreads / kWarp - 1];
  return warp_base + incl - v;
}

template <typename Tin>
__global__ __launch_bounds__(kScanThreads) void k_scan_tiles(const Tin *__restrict__ in, uint64_t *__restrict__ out,
                                                             uint64_t *__restrict__ tile_sums, size_t n) {
  const size_t base = size_t(blockIdx.x) * kScanTile + size_t(threadIdx.x) * kScanItems;
  uint64_t v[kScanItems];
  uint64_t sum = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    const size_t k = base + i;
    v[i] = k < n ? static_cast<uint64_t>(in[k]) : 0;
    sum += v[i];
  }
  uint64_t total;
  uint64_t run = block_exclusive_scan(sum, &total);
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    const size_t k = base + i;
    if (k < n) out[k] = run;
    run += v[i];
  }
  if (threadIdx.x == 0) {
    if (tile_sums) tile_sums[blockIdx.x] = total;
    if (gridDim.x == 1) out[n] = total;
  }
}

__global__ void k_add_tile_offsets(uint64_t *__restrict__ out, const uint64_t *__restrict__ offs, size_t n,
                                   size_t ntiles) {
  const size_t stride = size_t(gridDim.x) * blockDim.x;
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) out[i] += offs[i / kScanTile];
  if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = offs[ntiles];
}

template <typename Tin>
cudaError_t scan_impl(const Tin *in, uint64_t *out, size_t n, Bump &b, cudaStream_t st) {
  if (n == 0) return cudaMemsetAsync(out, 0, sizeof(uint64_t), st);
  const size_t ntiles = (n + kScanTile - 1) / kScanTile;
  if (ntiles == 1) {
    k_scan_tiles<Tin><<<1, kScanThreads, 0, st>>>(in, out, nullptr, n);
    note_launch();
    return cudaGetLastError();
  }
  uint64_t *sums = b.take<uint64_t>(ntiles);
  uint64_t *offs = b.take<uint64_t>(ntiles + 1);
  if (!sums || !offs) return cudaErrorMemoryAllocation;
  k_scan_tiles<Tin><<<static_cast<unsigned>(ntiles), kScanThreads, 0, st>>>(in, out, sums, n);
  note_launch();
  cudaError_t e = scan_impl<uint64_t>(sums, offs, ntiles, b, st);
  if (e != cudaSuccess) return e;
  const unsigned blocks = static_cast<unsigned>(std::min<size_t>((n + 255) / 256, 4096));
  k_add_tile_offsets<<<blocks, 256, 0, st>>>(out, offs, n, ntiles);
  note_launch();
  return cudaGetLastError();
}

// ---- radix sort -------------------------------------------------------------------------------

// Ranks a warp's digit (kDigits: no pair) among the digits that the warp took before it, in counts
// (the warp's own kDigits counters). A vote for each bit finds the lanes with the same digit; with
// __match_any_sync k_sort_small took 29 us for 25 at 5520 pairs.
__device__ __forceinline__ uint32_t warp_rank(uint32_t digit, uint32_t *counts) {
  const int lane = threadIdx.x & 31;
  uint32_t peers = kFull;
#pragma unroll
  for (int b = 0; b < 9; ++b) {
    const bool set = (digit >> b) & 1u;
    const uint32_t vote = __ballot_sync(kFull, set);
    peers &= set ? vote : ~vote;
  }
  uint32_t before = 0;
  if (digit < kDigits) before = counts[digit];
  __syncwarp();
  if (digit < kDigits && __ffs(peers) - 1 == lane) counts[digit] = before + __popc(peers);
  __syncwarp();
  return before + __popc(peers & ((1u << lane) - 1u));
}

// Exclusive scan of one uint32 a thread over the block's first kDigits threads; warp_tot: kDigits / 32
// words of shared memory. Every thread of the block calls it.
__device__ __forceinline__ uint32_t digit_scan(uint32_t v, uint32_t *warp_tot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t n = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += n;
  }
  if (lane == 31 && warp < kDigits / kWarp) warp_tot[warp] = incl;
  __syncthreads();
  uint32_t base = 0;
  for (int w = 0; w < min(warp, kDigits / kWarp); ++w) base += warp_tot[w];
  return base + incl - v;
}

struct SmallSort {
  uint64_t key[kSmallSort];
  uint32_t val[kSmallSort];
  uint32_t cnt[kSmallThreads / kWarp][kDigits];
  uint32_t part[kSmallThreads / kDigits][kDigits];
  uint32_t warp_tot[kDigits / kWarp];
};

// Every warp owns consecutive pairs, `rounds` of 32, so that all warps share a small sort. Bound by
// the latency of its steps: 30-bit keys (4 passes), 1280 pairs 12 us, 5520 pairs 25 us. The other way
// takes about 40 us at any size up to 100k pairs; before, 75 to 90 us.
__global__ __launch_bounds__(kSmallThreads) void k_sort_small(uint64_t *__restrict__ keys, uint32_t *__restrict__ vals,
                                                              uint32_t n, int bits, int digit_bits) {
  extern __shared__ __align__(16) unsigned char smem[];
  SmallSort &S = *reinterpret_cast<SmallSort *>(smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rounds = static_cast<int>((n + kSmallThreads - 1) / kSmallThreads);
  const uint32_t first = static_cast<uint32_t>(warp * rounds * kWarp + lane);
  const uint32_t mask = (1u << digit_bits) - 1u;
  uint64_t key[kSmallItems];
  uint32_t val[kSmallItems], rank[kSmallItems];
#pragma unroll
  for (int r = 0; r < kSmallItems; ++r) {
    const uint32_t pos = first + r * kWarp;
    const bool mine = r < rounds && pos < n;
    key[r] = mine ? keys[pos] : 0;
    val[r] = mine ? vals[pos] : 0;
  }
  for (int shift = 0; shift < bits; shift += digit_bits) {
    uint32_t *flat = &S.cnt[0][0];
#pragma unroll
    for (int k = 0; k < kDigits / kWarp; ++k) flat[k * kSmallThreads + tid] = 0;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSmallItems; ++r) {
      if (r >= rounds) break;
      const bool mine = first + r * kWarp < n;
      rank[r] = warp_rank(mine ? static_cast<uint32_t>(key[r] >> shift) & mask : kDigits, S.cnt[warp]);
    }
    __syncthreads();
    // Counts to starts: a thread takes one digit of a quarter of the warps.
    constexpr int kParts = kSmallThreads / kDigits, kRun = kSmallThreads / kWarp / kParts;
    const int digit = tid & (kDigits - 1), part = tid / kDigits;
    uint32_t c[kRun], sum = 0;
#pragma unroll
    for (int k = 0; k < kRun; ++k) {
      c[k] = S.cnt[part * kRun + k][digit];
      sum += c[k];
    }
    S.part[part][digit] = sum;
    __syncthreads();
    uint32_t total = 0, before = 0;
#pragma unroll
    for (int k = 0; k < kParts; ++k) {
      const uint32_t x = S.part[k][digit];
      total += x;
      if (k < part) before += x;
    }
    __syncthreads();
    const uint32_t start = digit_scan(total, S.warp_tot);
    if (part == 0) S.part[0][digit] = start;
    __syncthreads();
    uint32_t run = S.part[0][digit] + before;
#pragma unroll
    for (int k = 0; k < kRun; ++k) {
      S.cnt[part * kRun + k][digit] = run;
      run += c[k];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSmallItems; ++r) {
      if (r >= rounds || first + r * kWarp >= n) break;
      const uint32_t to = S.cnt[warp][static_cast<uint32_t>(key[r] >> shift) & mask] + rank[r];
      S.key[to] = key[r];
      S.val[to] = val[r];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSmallItems; ++r) {
      const uint32_t pos = first + r * kWarp;
      if (r >= rounds || pos >= n) break;
      key[r] = S.key[pos];
      val[r] = S.val[pos];
    }
  }
#pragma unroll
  for (int r = 0; r < kSmallItems; ++r) {
    const uint32_t pos = first + r * kWarp;
    if (r >= rounds || pos >= n) break;
    keys[pos] = key[r];
    vals[pos] = val[r];
  }
}

// Counts of every digit of every pass: totals[pass][digit].
__global__ __launch_bounds__(kSortThreads) void k_sort_count(const uint64_t *__restrict__ keys, size_t n, int passes,
                                                             int digit_bits, unsigned long long *__restrict__ totals) {
  __shared__ uint32_t cnt[kMaxPasses][kDigits];
  for (int p = 0; p < passes; ++p) cnt[p][threadIdx.x] = 0;
  __syncthreads();
  const uint32_t mask = (1u << digit_bits) - 1u;
  const size_t stride = size_t(gridDim.x) * kSortThreads;
  for (size_t i = size_t(blockIdx.x) * kSortThreads + threadIdx.x; i < n; i += stride) {
    uint64_t key = keys[i];
    for (int p = 0; p < passes; ++p, key >>= digit_bits) atomicAdd(&cnt[p][static_cast<uint32_t>(key) & mask], 1u);
  }
  __syncthreads();
  for (int p = 0; p < passes; ++p) {
    const uint32_t c = cnt[p][threadIdx.x];
    if (c) atomicAdd(totals + p * kDigits + threadIdx.x, static_cast<unsigned long long>(c));
  }
}

// A tile's published count of a digit: (tag << 48) | count. The tag names the pass, and whether the
// count is the tile's own (2 pass + 1) or that of all tiles up to it (2 pass + 2); what an earlier pass
// left has a smaller one. Tag and count travel in one word, so no fence orders them.
constexpr int kTagShift = 48;

// Pairs of the digit in the tiles before `tile`. Tiles take their numbers from a counter, so those
// before it have started and publish without waiting for anything; should one not be seen within
// kMaxPolls looks all the same, the thread counts that tile and those before it in the keys
// themselves, which this pass only reads.
__device__ __forceinline__ uint64_t look_back(const uint64_t *__restrict__ kin, const volatile uint64_t *status,
                                              size_t tile, uint32_t digit, int pass, int shift, uint32_t mask) {
  const uint64_t own = 2 * pass + 1, all = own + 1;
  uint64_t sum = 0;
  int polls = 0;
  size_t t = tile;  // tiles below t are still to be added
  while (t > 0) {
    uint64_t w[kLookBack];
#pragma unroll
    for (int k = 0; k < kLookBack; ++k) w[k] = t > size_t(k) ? status[(t - 1 - k) * kDigits + digit] : 0;
#pragma unroll
    for (int k = 0; k < kLookBack; ++k) {
      const uint64_t tag = w[k] >> kTagShift;
      if (tag < own) break;
      sum += w[k] & ((uint64_t(1) << kTagShift) - 1);
      if (tag == all) return sum;
      --t;
    }
    if (++polls > kMaxPolls) {
      for (size_t i = 0; i < t * kSortTile; ++i) sum += (static_cast<uint32_t>(kin[i] >> shift) & mask) == digit ? 1 : 0;
      return sum;
    }
  }
  return sum;
}

__global__ __launch_bounds__(kSortThreads) void k_sort_pass(const uint64_t *__restrict__ kin,
                                                            const uint32_t *__restrict__ vin,
                                                            uint64_t *__restrict__ kout, uint32_t *__restrict__ vout,
                                                            size_t n, int pass, int digit_bits,
                                                            const unsigned long long *__restrict__ totals,
                                                            unsigned long long *ticket, uint64_t *status) {
  constexpr int kWarps = kSortThreads / kWarp;
  static_assert(kSortThreads == kDigits && kSortThreads == kScanThreads, "a thread per digit");
  __shared__ uint64_t s_key[kSortTile];
  __shared__ uint32_t s_val[kSortTile];
  __shared__ uint32_t s_cnt[kWarps][kDigits];
  __shared__ uint32_t s_start[kDigits];
  __shared__ uint64_t s_out[kDigits];
  __shared__ uint32_t s_tot[kDigits / kWarp];
  __shared__ unsigned long long s_tile;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int shift = pass * digit_bits;
  const uint32_t mask = (1u << digit_bits) - 1u;
  if (tid == 0) s_tile = atomicAdd(ticket, 1ull);
#pragma unroll
  for (int w = 0; w < kWarps; ++w) s_cnt[w][tid] = 0;
  __syncthreads();
  const size_t tile = s_tile;
  const size_t base = tile * kSortTile;
  const uint32_t count = static_cast<uint32_t>(n - base < kSortTile ? n - base : kSortTile);
  const uint32_t first = static_cast<uint32_t>(warp * kSortItems * kWarp + lane);
  uint64_t key[kSortItems];
  uint32_t val[kSortItems], rank[kSortItems];
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const uint32_t pos = first + r * kWarp;
    key[r] = pos < count ? kin[base + pos] : 0;
    val[r] = pos < count ? vin[base + pos] : 0;
  }
#pragma unroll
  for (int r = 0; r < kSortItems; ++r)
    rank[r] = warp_rank(first + r * kWarp < count ? static_cast<uint32_t>(key[r] >> shift) & mask : kDigits, s_cnt[warp]);
  __syncthreads();
  uint32_t total = 0;  // of digit tid
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    const uint32_t c = s_cnt[w][tid];
    s_cnt[w][tid] = total;
    total += c;
  }
  volatile uint64_t *mine = status + tile * kDigits + tid;
  if (tile) *mine = (uint64_t(2 * pass + 1) << kTagShift) | total;
  const uint64_t before = look_back(kin, status, tile, tid, pass, shift, mask);
  *mine = (uint64_t(2 * pass + 2) << kTagShift) | (before + total);
  const uint32_t start = digit_scan(total, s_tot);
  uint64_t all;
  const uint64_t digit_base = block_exclusive_scan(totals[pass * kDigits + tid], &all);
  s_start[tid] = start;
  s_out[tid] = digit_base + before - start;  // of the digit's first pair, less its place in the tile
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    if (first + r * kWarp >= count) break;
    const uint32_t digit = static_cast<uint32_t>(key[r] >> shift) & mask;
    const uint32_t to = s_start[digit] + s_cnt[warp][digit] + rank[r];
    s_key[to] = key[r];
    s_val[to] = val[r];
  }
  __syncthreads();
  for (uint32_t i = tid; i < count; i += kSortThreads) {
    const uint64_t k = s_key[i];
    const uint64_t to = s_out[static_cast<uint32_t>(k >> shift) & mask] + i;
    kout[to] = k;
    vout[to] = s_val[i];
  }
}

}  // namespace

size_t scan_scratch_bytes(size_t n) {
  size_t total = 0;
  size_t m = n;
  while (m > kScanTile) {
    const size_t t = (m + kScanTile - 1) / kScanTile;
    total += align256(t * sizeof(uint64_t)) + align256((t + 1) * sizeof(uint64_t));
    m = t;
  }
  return total + 1024;
}

cudaError_t exclusive_scan_u32(const uint32_t *in, uint64_t *out, size_t n, Scratch s, cudaStream_t st) {
  Bump b{static_cast<char *>(s.ptr), s.bytes};
  return scan_impl<uint32_t>(in, out, n, b, st);
}

// Scratch of a sort of more than kSmallSort pairs: the passes' tile counters, the digits' totals and
// the tiles' published counts.
constexpr size_t kSortTotals = size_t(kMaxPasses) * kDigits * 8;

size_t sort_scratch_bytes(size_t n) {
  const size_t ntiles = (n + kSortTile - 1) / kSortTile;
  return 256 + kSortTotals + ntiles * kDigits * 8;
}

cudaError_t radix_sort_pairs(uint64_t *keys, uint32_t *vals, uint64_t *keys_alt, uint32_t *vals_alt, size_t n,
                             int bits, Scratch s, cudaStream_t st) {
  if (n <= 1 || bits <= 0) return cudaSuccess;
  const int passes = (bits + 7) / 8, digit_bits = (bits + passes - 1) / passes;
  if (n <= kSmallSort) {
    cudaError_t e = cudaFuncSetAttribute(k_sort_small, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(SmallSort));
    if (e != cudaSuccess) return e;
    k_sort_small<<<1, kSmallThreads, sizeof(SmallSort), st>>>(keys, vals, static_cast<uint32_t>(n), bits, digit_bits);
    note_launch();
    return cudaGetLastError();
  }
  if (passes > kMaxPasses) return cudaErrorInvalidValue;
  const size_t bytes = sort_scratch_bytes(n), ntiles = (n + kSortTile - 1) / kSortTile;
  if (bytes > s.bytes) return cudaErrorMemoryAllocation;
  char *p = static_cast<char *>(s.ptr);
  unsigned long long *tickets = reinterpret_cast<unsigned long long *>(p);
  unsigned long long *totals = reinterpret_cast<unsigned long long *>(p + 256);
  uint64_t *status = reinterpret_cast<uint64_t *>(p + 256 + kSortTotals);
  cudaError_t e = cudaMemsetAsync(p, 0, bytes, st);
  if (e != cudaSuccess) return e;
  k_sort_count<<<static_cast<unsigned>(std::min<size_t>(ntiles, 608)), kSortThreads, 0, st>>>(keys, n, passes,
                                                                                              digit_bits, totals);
  note_launch();
  uint64_t *ka = keys, *kb = keys_alt;
  uint32_t *va = vals, *vb = vals_alt;
  for (int pass = 0; pass < passes; ++pass) {
    k_sort_pass<<<static_cast<unsigned>(ntiles), kSortThreads, 0, st>>>(ka, va, kb, vb, n, pass, digit_bits, totals,
                                                                        tickets + pass, status);
    note_launch();
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    std::swap(ka, kb);
    std::swap(va, vb);
  }
  if (passes & 1) {
    e = cudaMemcpyAsync(keys, ka, n * sizeof(uint64_t), cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return e;
    return cudaMemcpyAsync(vals, va, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st);
  }
  return cudaSuccess;
}

}  // namespace sdfb
