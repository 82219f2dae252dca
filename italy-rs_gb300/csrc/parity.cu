// Exact +z ray parity for watertight meshes (the reference's first parity ray is +z,
// src/render/kernels/sdf_bake.cu:53-69; there it is stepped with a 1e-4 epsilon and voted over 5
// rays, here it is one exact ray per column).
//
// Every cell of a column (x, y) shares the line through the column's FP32 centre, so the bake
// finds, once per column, the heights at which that line crosses the mesh; a cell is inside when
// an odd number of crossings lie above its centre. Whether the line crosses a triangle is decided
// with exact orientation predicates and simulation of simplicity (common.cuh), so a line through
// a shared edge or vertex is counted exactly once and the parity is exact for every column.
//
// Parity meshes keep a bit a cell, layers along a word: a crossing at height z flips the inside bit of
// every cell below it, so it toggles one bit, that of the highest such layer, and a cell is inside when
// an odd number of toggles lie at or above it (the distance kernel counts them). One pass over the
// (triangle, column) items (expand.cuh), one XOR a crossing, 1/32 of the distance grid's size.
//
// Winding-number meshes need every crossing's height and orientation: a first pass counts them per
// column, a scan gives the columns their slots and a second pass fills them, in any order. (Parity
// meshes took these three steps too, and the distance kernel compared every cell with every height of
// its column.)
#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "expand.cuh"
#include "kernels.h"

namespace sdfb {
namespace {

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

struct TriCols {
  f3 a, b, c;
  int x0, x1, y0, y1;
  int mesh;
};

__device__ __forceinline__ f3 vload(const float *v, uint32_t i) {
  return {__ldg(v + 3ull * i), __ldg(v + 3ull * i + 1), __ldg(v + 3ull * i + 2)};
}

// Column index range [lo, hi] whose centres o + (i + 0.5) v may fall inside [mn, mx], widened by
// a margin far above the FP32 error of the index arithmetic.
__device__ __forceinline__ void col_range(float mn, float mx, float o, float v, int n, int &lo, int &hi) {
  const float a = (mn - o) / v - 0.5f, b = (mx - o) / v - 0.5f;
  const float eps = 0.01f + 2e-6f * fmaxf(fabsf(a), fabsf(b));
  const float fa = ceilf(a - eps), fb = floorf(b + eps);
  lo = fa < 0.0f ? 0 : (fa > float(n - 1) ? n : static_cast<int>(fa));
  hi = fb < 0.0f ? -1 : (fb > float(n - 1) ? n - 1 : static_cast<int>(fb));
}

// Parity triangle t (global over the parity meshes) and its candidate columns.
__device__ __forceinline__ TriCols tri_cols(const BatchDev &B, uint64_t t) {
  TriCols r;
  r.mesh = find_mesh(B.ptri_starts, B.num_meshes, t);
  const MeshRec &M = B.recs[r.mesh];
  const uint64_t lt = t - B.ptri_starts[r.mesh];
  const uint32_t V = M.pnum_verts;
  const uint32_t i0 = __ldg(M.pidx + 3 * lt), i1 = __ldg(M.pidx + 3 * lt + 1), i2 = __ldg(M.pidx + 3 * lt + 2);
  r.a = vload(M.pverts, i0 < V ? i0 : 0);
  r.b = vload(M.pverts, i1 < V ? i1 : 0);
  r.c = vload(M.pverts, i2 < V ? i2 : 0);
  const bool ok = isfinite(r.a.x + r.a.y + r.b.x + r.b.y + r.c.x + r.c.y + r.a.z + r.b.z + r.c.z);
  const GridDev &g = M.g;
  col_range(fminf(fminf(r.a.x, r.b.x), r.c.x), fmaxf(fmaxf(r.a.x, r.b.x), r.c.x), g.ox, g.voxel, g.nx, r.x0, r.x1);
  col_range(fminf(fminf(r.a.y, r.b.y), r.c.y), fmaxf(fmaxf(r.a.y, r.b.y), r.c.y), g.oy, g.voxel, g.ny, r.y0, r.y1);
  if (!ok || r.x1 < r.x0 || r.y1 < r.y0) {
    r.x0 = r.y0 = 0;
    r.x1 = r.y1 = -1;
  }
  return r;
}

// Layers whose cell centres are below z, of nz. The estimate is corrected against the centres
// themselves, which do not decrease with the layer.
__device__ __forceinline__ int layers_below(const GridDev &g, float z) {
  const float f = (z - g.oz) / g.voxel + 0.5f;
  int k = f > 0.0f ? (f < float(g.nz) ? static_cast<int>(f) : g.nz) : 0;
  while (k > 0 && !(cell_center(g.oz, k - 1, g.voxel) < z)) --k;
  while (k < g.nz && cell_center(g.oz, k, g.voxel) < z) ++k;
  return k;
}

// FILL: the winding-number meshes' second pass; else their count, and the parity meshes' bits.
template <bool FILL> struct ColumnOp {
  using Tri = TriCols;
  uint32_t *col_count, *bits;
  const uint64_t *col_start;
  float *col_z;
  int8_t *col_s;
  uint64_t capacity;
  unsigned long long *crossings;
  uint32_t *err;
  uint32_t found = 0;

  // Candidate columns, as a 64-bit count (a triangle across a wide, flat grid can cover more than 2^32).
  __device__ __forceinline__ uint64_t setup(const BatchDev &B, uint64_t t, Tri &tri) const {
    tri = tri_cols(B, t);
    if (tri.x1 < tri.x0 || (FILL && B.recs[tri.mesh].sign != kSignGwn)) return 0;
    return uint64_t(tri.x1 - tri.x0 + 1) * uint64_t(tri.y1 - tri.y0 + 1);
  }
  __device__ __forceinline__ void item(const BatchDev &B, const Tri &tri, uint64_t k) {
    const MeshRec &M = B.recs[tri.mesh];
    const GridDev &g = M.g;
    const uint32_t sx = tri.x1 - tri.x0 + 1;
    const uint64_t row = (k >> 32) == 0 ? static_cast<uint32_t>(k) / sx : k / sx;
    const int x = tri.x0 + static_cast<int>(k - row * sx), y = tri.y0 + static_cast<int>(row);
    const float px = cell_center(g.ox, x, g.voxel), py = cell_center(g.oy, y, g.voxel);
    float z;
    int sgn;
    const bool hit = column_crossing(tri.a, tri.b, tri.c, px, py, z, sgn);
    if (!hit) return;
    ++found;
    if (!FILL && M.sign == kSignParity) {
      const int below = layers_below(g, z);
      if (below > 0) {
        const uint64_t words = (uint64_t(g.nz) + 31) / 32;
        atomicXor(bits + M.bit_base + (uint64_t(y) * g.nx + x) * words + (below - 1) / 32, 1u << ((below - 1) & 31));
      }
      return;
    }
    const uint64_t col = M.col_base + uint64_t(y) * g.nx + x;
    const uint32_t slot = atomicAdd(col_count + col, 1u);
    if (FILL) {
      const uint64_t at = col_start[col] + slot;
      if (at < capacity) {
        col_z[at] = z;
        col_s[at] = static_cast<int8_t>(sgn);
      } else {
        atomic_or_err(err, kErrCrossingOverflow);
      }
    }
  }
  __device__ __forceinline__ void finish(const BatchDev &, unsigned long long) const {
    if (FILL) return;
    const uint32_t sum = __reduce_add_sync(kFull, found);
    if (sum && (threadIdx.x & 31) == 0) atomicAdd(crossings, static_cast<unsigned long long>(sum));
  }
};

struct ParTemp {
  void *big;
  uint32_t *col_count;
  void *scratch;
  size_t scratch_bytes;
};

size_t par_layout(uint64_t T, uint64_t ncols, char *base, ParTemp *o) {
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char *p = base ? base + off : nullptr;
    off += align256(bytes);
    return p;
  };
  ParTemp x;
  x.big = take(big_list_bytes(T));
  x.col_count = reinterpret_cast<uint32_t *>(take(ncols * 4 + 4));
  x.scratch_bytes = scan_scratch_bytes(ncols);
  x.scratch = take(x.scratch_bytes);
  if (o) *o = x;
  return off;
}

}  // namespace

size_t parity_temp_bytes(uint64_t total_ptris, uint64_t total_cols) {
  return par_layout(total_ptris, total_cols, nullptr, nullptr);
}

cudaError_t parity_columns(const BatchDev &B, uint32_t *bits, uint64_t *col_start, float *col_z, int8_t *col_s,
                           uint64_t capacity, void *temp, size_t temp_bytes, unsigned long long *counters,
                           uint32_t *err, int num_sms, cudaStream_t st) {
  const uint64_t T = B.total_ptris, ncols = B.total_cols;
  ParTemp o;
  if (par_layout(T, ncols, static_cast<char *>(temp), &o) > temp_bytes) return cudaErrorMemoryAllocation;
  if (T == 0) return cudaErrorInvalidValue;
  BigList big = big_list(o.big, T);
  unsigned long long *const second = big.counts;
  big.counts = counters + 1;
  cudaError_t e = cudaSuccess;
  if (B.total_bit_words) e = cudaMemsetAsync(bits, 0, B.total_bit_words * 4, st);
  if (e == cudaSuccess && ncols) e = cudaMemsetAsync(o.col_count, 0, ncols * 4, st);
  if (e != cudaSuccess) return e;
  e = expand(B, T, big, ColumnOp<false>{o.col_count, bits, nullptr, nullptr, nullptr, 0, counters, err, 0}, num_sms, st);
  if (e != cudaSuccess || ncols == 0) return e;
  if ((e = exclusive_scan_u32(o.col_count, col_start, ncols, Scratch{o.scratch, o.scratch_bytes}, st)) != cudaSuccess ||
      (e = cudaMemsetAsync(o.col_count, 0, ncols * 4, st)) != cudaSuccess ||
      (e = cudaMemsetAsync(second, 0, 24, st)) != cudaSuccess)
    return e;
  big.counts = second;
  return expand(B, T, big, ColumnOp<true>{o.col_count, nullptr, col_start, col_z, col_s, capacity, nullptr, err, 0}, num_sms,
                st);
}

}  // namespace sdfb
