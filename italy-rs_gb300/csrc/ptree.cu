// Packed 32-ary tree over the triangles of a batch of meshes, for the distance walk (it takes the
// place of the OptiX GAS build of src/convert/sdf_baker.cpp:170-193).
//
// The triangles of a mesh are sorted along a Hilbert curve and cut into blocks of 2, 4 or 8
// consecutive triangles; 32 consecutive blocks are a level-1 node, 32 consecutive level-1 nodes a
// level-2 node, and so on up to one root. Nothing is linked: node i of level l covers nodes
// [32 i, 32 i + 32) of level l - 1. A warp tests all 32 children of a node at once from coalesced
// loads (distance.cu), and the build is a sort, one pass over the triangles and a reduction per
// level, without per-node atomics. The Hilbert curve has no jumps (a Morton curve's make blocks
// that straddle them: 10-25% more point-triangle pairs in the walk on the measured meshes).
//
//   k_prep      checks indices and finiteness, reduces per-mesh centroid bounds
//   k_keys      key = (mesh << 30) | 30-bit Hilbert index of the box centre in its mesh's bounds
//   radix sort  (key, triangle) pairs, stable
//   k_pack      per triangle the 80-byte frame record (DistTri, in planes of float4 so that
//               consecutive triangles coalesce); per block an oriented box; per level-1 node its
//               axis-aligned box
//   k_upper     the boxes of the levels above, one thread block per mesh and block size
//
// A block's oriented box follows its patch of surface: normal axis from the triangles' area
// vectors, in-plane axes from the vertices' covariance. Where a surface runs obliquely to the axes
// an axis-aligned box of eight triangles stands out of it by about half the patch size, which is
// what kept thousands of nearly equidistant triangles alive in the interior of a closed mesh.
#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "kernels.h"

namespace sdfb {
namespace {

constexpr int kThreads = 256;
static_assert(kThreads == kTreePad, "one thread block packs one padding unit");

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }
inline unsigned blocks_for(size_t n) { return static_cast<unsigned>((n + kThreads - 1) / kThreads); }

__device__ __forceinline__ float3 load3(const float *v, uint32_t i) {
  return make_float3(__ldg(v + 3ull * i), __ldg(v + 3ull * i + 1), __ldg(v + 3ull * i + 2));
}

// Corners of local triangle lt; an index out of range reads vertex 0 (and is reported once, by k_prep).
__device__ __forceinline__ bool corners(const MeshRec &M, uint64_t lt, float3 &a, float3 &b, float3 &c) {
  const uint32_t V = M.num_verts;
  const uint32_t i0 = __ldg(M.idx + 3 * lt), i1 = __ldg(M.idx + 3 * lt + 1), i2 = __ldg(M.idx + 3 * lt + 2);
  a = load3(M.verts, i0 < V ? i0 : 0);
  b = load3(M.verts, i1 < V ? i1 : 0);
  c = load3(M.verts, i2 < V ? i2 : 0);
  return i0 < V && i1 < V && i2 < V;
}

__device__ __forceinline__ float3 box_mid(float3 a, float3 b, float3 c) {
  return make_float3(0.5f * (fminf(fminf(a.x, b.x), c.x) + fmaxf(fmaxf(a.x, b.x), c.x)),
                     0.5f * (fminf(fminf(a.y, b.y), c.y) + fmaxf(fmaxf(a.y, b.y), c.y)),
                     0.5f * (fminf(fminf(a.z, b.z), c.z) + fmaxf(fmaxf(a.z, b.z), c.z)));
}

__global__ void k_init_bounds(uint32_t *bounds, int M) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 6 * M) bounds[i] = (i % 6) < 3 ? 0xffffffffu : 0u;
}

__global__ __launch_bounds__(kThreads) void k_prep(BatchDev B, uint32_t *__restrict__ bounds,
                                                   uint32_t *__restrict__ err) {
  const uint64_t t = uint64_t(blockIdx.x) * kThreads + threadIdx.x;
  float cmin[3] = {INFINITY, INFINITY, INFINITY}, cmax[3] = {-INFINITY, -INFINITY, -INFINITY};
  int mesh = -1;
  if (t < B.total_tris) {
    mesh = find_mesh(B.tri_starts, B.num_meshes, t);
    float3 a, b, c;
    if (!corners(B.recs[mesh], t - B.tri_starts[mesh], a, b, c)) atomic_or_err(err, kErrBadIndex);
    const bool finite = isfinite(a.x) && isfinite(a.y) && isfinite(a.z) && isfinite(b.x) && isfinite(b.y) &&
                        isfinite(b.z) && isfinite(c.x) && isfinite(c.y) && isfinite(c.z);
    if (!finite) {
      atomic_or_err(err, kErrNonFinite);
    } else {
      const float3 m = box_mid(a, b, c);
      cmin[0] = cmax[0] = m.x;
      cmin[1] = cmax[1] = m.y;
      cmin[2] = cmax[2] = m.z;
    }
  }
  // Reduce over the warp when all its lanes hold the same mesh, else per lane.
  const int m0 = __shfl_sync(kFull, mesh, 0);
  if (__all_sync(kFull, mesh == m0)) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        cmin[a] = fminf(cmin[a], __shfl_xor_sync(kFull, cmin[a], o));
        cmax[a] = fmaxf(cmax[a], __shfl_xor_sync(kFull, cmax[a], o));
      }
    }
    if ((threadIdx.x & 31) != 0) mesh = -1;
  }
  if (mesh >= 0 && cmin[0] <= cmax[0]) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      atomicMin(bounds + 6 * mesh + a, float_to_ordered(cmin[a]));
      atomicMax(bounds + 6 * mesh + 3 + a, float_to_ordered(cmax[a]));
    }
  }
}

// 30-bit index of a 10-bit lattice point along a 3-D Hilbert curve (Skilling 2004, "Programming the
// Hilbert curve": the transpose form, then the bits interleaved).
__device__ __forceinline__ uint32_t hilbert30(uint32_t x, uint32_t y, uint32_t z) {
  uint32_t X[3] = {x, y, z};
#pragma unroll
  for (uint32_t q = 512; q > 1; q >>= 1) {
    const uint32_t p = q - 1;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      if (X[i] & q) {
        X[0] ^= p;
      } else {
        const uint32_t t = (X[0] ^ X[i]) & p;
        X[0] ^= t;
        X[i] ^= t;
      }
    }
  }
  X[1] ^= X[0];
  X[2] ^= X[1];
  uint32_t t = 0;
#pragma unroll
  for (uint32_t q = 512; q > 1; q >>= 1)
    if (X[2] & q) t ^= q - 1;
  uint32_t key = 0;
#pragma unroll
  for (int b = 9; b >= 0; --b)
#pragma unroll
    for (int i = 0; i < 3; ++i) key = (key << 1) | (((X[i] ^ t) >> b) & 1u);
  return key;
}

__global__ __launch_bounds__(kThreads) void k_keys(BatchDev B, const uint32_t *__restrict__ bounds,
                                                   uint64_t *__restrict__ keys, uint32_t *__restrict__ vals) {
  const uint64_t t = uint64_t(blockIdx.x) * kThreads + threadIdx.x;
  if (t >= B.total_tris) return;
  const int mesh = find_mesh(B.tri_starts, B.num_meshes, t);
  float3 a, b, c;
  corners(B.recs[mesh], t - B.tri_starts[mesh], a, b, c);
  const float3 m = box_mid(a, b, c);
  const float mid[3] = {m.x, m.y, m.z};
  float lo[3], ext = 0.0f;  // one scale for the three axes: the curve's cells are cubes
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    lo[k] = ordered_to_float(bounds[6 * mesh + k]);
    ext = fmaxf(ext, ordered_to_float(bounds[6 * mesh + 3 + k]) - lo[k]);
  }
  uint32_t q[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float u = ext > 0.0f ? (mid[k] - lo[k]) / ext : 0.5f;
    const float s = fminf(fmaxf(u * 1024.0f, 0.0f), 1023.0f);
    q[k] = isfinite(s) ? static_cast<uint32_t>(s) : 0u;
  }
  keys[t] = (uint64_t(mesh) << 30) | hilbert30(q[0], q[1], q[2]);
  vals[t] = static_cast<uint32_t>(t);
}

// Sum, minimum and maximum over aligned groups of n lanes (n a power of two).
__device__ __forceinline__ float group_sum(float v, int n) {
  for (int o = 1; o < n; o <<= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}
__device__ __forceinline__ float group_min(float v, int n) {
  for (int o = 1; o < n; o <<= 1) v = fminf(v, __shfl_xor_sync(kFull, v, o));
  return v;
}
__device__ __forceinline__ float group_max(float v, int n) {
  for (int o = 1; o < n; o <<= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, o));
  return v;
}

__device__ __forceinline__ float3 sub(float3 a, float3 b) { return make_float3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float dot(float3 a, float3 b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, a.z * b.z)); }
__device__ __forceinline__ float3 cross(float3 a, float3 b) {
  return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ float3 scaled(float3 a, float s) { return make_float3(a.x * s, a.y * s, a.z * s); }

// Oriented box of the n triangles in an aligned group of n lanes, written by the group's first
// lane as four float4s: (centre, half0), (axis0, half1), (axis1, half2), (axis2, diagonal).
// The half extents are measured along the axes as rounded to FP32 and widened by 1e-6 of the
// box's size, several times the rounding of a point's coordinates in that frame and of the
// point-triangle distance itself: a triangle whose computed distance is below a bound is never
// behind a box distance above it (see the margins in distance.cu).
__device__ __forceinline__ void put_obb(float3 a, float3 b, float3 c, int n, float4 *obb, uint32_t block,
                                        bool lead) {
  float3 cr = cross(sub(b, a), sub(c, a));
  const int first = (threadIdx.x & 31) & ~(n - 1);
  const float3 ref = make_float3(__shfl_sync(kFull, cr.x, first), __shfl_sync(kFull, cr.y, first),
                                 __shfl_sync(kFull, cr.z, first));
  if (dot(cr, ref) < 0.0f) cr = scaled(cr, -1.0f);
  float3 nv = make_float3(group_sum(cr.x, n), group_sum(cr.y, n), group_sum(cr.z, n));
  const float big = fmaxf(fmaxf(fabsf(nv.x), fabsf(nv.y)), fabsf(nv.z));
  // Unit normal; scaling by the largest component first keeps tiny triangles out of underflow. A
  // patch without area takes any frame.
  if (big > 1e-37f && isfinite(big)) {
    nv = scaled(nv, 1.0f / big);
    nv = scaled(nv, rsqrtf(dot(nv, nv)));
  } else {
    nv = make_float3(0.0f, 0.0f, 1.0f);
  }
  const float inv = 1.0f / (3.0f * float(n));
  const float3 mid = make_float3(group_sum(a.x + b.x + c.x, n) * inv, group_sum(a.y + b.y + c.y, n) * inv,
                                 group_sum(a.z + b.z + c.z, n) * inv);
  float3 u = fabsf(nv.x) < 0.7f ? make_float3(1.0f, 0.0f, 0.0f) : make_float3(0.0f, 1.0f, 0.0f);
  u = sub(u, scaled(nv, dot(u, nv)));
  u = scaled(u, rsqrtf(dot(u, u)));
  float3 w = cross(nv, u);
  // Covariance of the vertices in the (u, w) plane; its larger eigenvector is the first axis.
  float suu = 0.0f, suw = 0.0f, sww = 0.0f, ext = 0.0f;
  const float3 p[3] = {sub(a, mid), sub(b, mid), sub(c, mid)};
#pragma unroll
  for (int k = 0; k < 3; ++k) ext = fmaxf(ext, fmaxf(fabsf(dot(p[k], u)), fabsf(dot(p[k], w))));
  ext = group_max(ext, n);
  const float is = ext > 0.0f && isfinite(ext) ? 1.0f / ext : 0.0f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float x = dot(p[k], u) * is, y = dot(p[k], w) * is;
    suu = fmaf(x, x, suu);
    suw = fmaf(x, y, suw);
    sww = fmaf(y, y, sww);
  }
  suu = group_sum(suu, n);
  suw = group_sum(suw, n);
  sww = group_sum(sww, n);
  const float half = 0.5f * (suu - sww), root = sqrtf(fmaf(half, half, suw * suw));
  float ex = half + root, ey = suw;  // eigenvector (half + root, suw); the other form where it vanishes
  if (half < 0.0f) {
    ex = suw;
    ey = root - half;
  }
  const float len2 = fmaf(ex, ex, ey * ey);
  if (len2 > 1e-12f) {
    const float r = rsqrtf(len2);
    ex *= r;
    ey *= r;
  } else {
    ex = 1.0f;
    ey = 0.0f;
  }
  const float3 ax[3] = {make_float3(u.x * ex + w.x * ey, u.y * ex + w.y * ey, u.z * ex + w.z * ey),
                        make_float3(w.x * ex - u.x * ey, w.y * ex - u.y * ey, w.z * ex - u.z * ey), nv};
  float mn[3], mx[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float d0 = dot(p[0], ax[k]), d1 = dot(p[1], ax[k]), d2 = dot(p[2], ax[k]);
    mn[k] = group_min(fminf(fminf(d0, d1), d2), n);
    mx[k] = group_max(fmaxf(fmaxf(d0, d1), d2), n);
  }
  if (!lead) return;
  float3 cen = mid;
  float h[3], diag = 0.0f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float m = 0.5f * (mn[k] + mx[k]);
    cen = make_float3(fmaf(ax[k].x, m, cen.x), fmaf(ax[k].y, m, cen.y), fmaf(ax[k].z, m, cen.z));
    h[k] = 0.5f * (mx[k] - mn[k]);
    diag += h[k];
  }
  // The centre is rounded to the coordinates' precision: allow for it in every direction.
  const float room = 1e-6f * diag + 2.4e-7f * (fabsf(cen.x) + fabsf(cen.y) + fabsf(cen.z));
  float4 *o = tree_obb(obb, block);
  o[0] = make_float4(cen.x, cen.y, cen.z, h[0] + room);
  o[kObbPlane] = make_float4(ax[0].x, ax[0].y, ax[0].z, h[1] + room);
  o[2 * kObbPlane] = make_float4(ax[1].x, ax[1].y, ax[1].z, h[2] + room);
  o[3 * kObbPlane] = make_float4(ax[2].x, ax[2].y, ax[2].z, diag);
}

// Axis-aligned box as centre and half extent, rounded outward: [c - e, c + e] contains [lo, hi].
__device__ __forceinline__ void put_box(float4 *box, uint32_t node, const float (&lo)[3], const float (&hi)[3]) {
  float c[3], e[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    c[k] = __fmul_rn(0.5f, __fadd_rn(lo[k], hi[k]));
    e[k] = __fmul_ru(fmaxf(__fsub_ru(hi[k], c[k]), __fsub_ru(c[k], lo[k])), 1.0f + 0x1p-22f);
  }
  box[2 * size_t(node)] = make_float4(c[0], c[1], c[2], 0.0f);
  box[2 * size_t(node) + 1] = make_float4(e[0], e[1], e[2], 0.0f);
}

// One thread per triangle slot; slots past a mesh's last triangle repeat it, so every block is full.
// A thread block packs 256 slots of one mesh.
__global__ __launch_bounds__(kThreads) void k_pack(BatchDev B, const PTreeRec *__restrict__ trees,
                                                   const uint64_t *__restrict__ group_starts,
                                                   const uint32_t *__restrict__ vals) {
  __shared__ float s_lo[kThreads / kWarp][3], s_hi[kThreads / kWarp][3];
  const int mesh = find_mesh(group_starts, B.num_meshes, blockIdx.x);
  const PTreeRec &R = trees[mesh];
  const uint32_t slot = static_cast<uint32_t>(blockIdx.x - group_starts[mesh]) * kThreads + threadIdx.x;
  const uint64_t base = B.tri_starts[mesh];
  const uint32_t pos = min(slot, R.num_tris - 1);
  const uint64_t lt = (B.total_tris > 1 ? uint64_t(__ldg(vals + base + pos)) : 0) - base;
  float3 a, b, c;
  corners(B.recs[mesh], lt, a, b, c);
  {
    const DistTri t = make_dist_tri(a, b, c);
    float4 *o = tree_tri(R.tri, slot);
    o[0] = t.q0;
    o[kTriPlane] = t.q1;
    o[2 * kTriPlane] = t.q2;
    o[3 * kTriPlane] = t.q3;
    o[4 * kTriPlane] = t.q4;
  }
#pragma unroll
  for (int k = 0; k < kTreeSizes; ++k) {
    if (!R.obb[k]) continue;
    const int n = 2 << k;
    put_obb(a, b, c, n, R.obb[k], slot >> (k + 1), (threadIdx.x & (n - 1)) == 0);
  }
  float lo[3] = {fminf(fminf(a.x, b.x), c.x), fminf(fminf(a.y, b.y), c.y), fminf(fminf(a.z, b.z), c.z)};
  float hi[3] = {fmaxf(fmaxf(a.x, b.x), c.x), fmaxf(fmaxf(a.y, b.y), c.y), fmaxf(fmaxf(a.z, b.z), c.z)};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    lo[k] = group_min(lo[k], kWarp);
    hi[k] = group_max(hi[k], kWarp);
    if ((threadIdx.x & 31) == 0) {
      s_lo[threadIdx.x >> 5][k] = lo[k];
      s_hi[threadIdx.x >> 5][k] = hi[k];
    }
  }
  __syncthreads();
  // Level-1 nodes: 32 blocks of 2, 4, 8 triangles are 2, 4, 8 warps.
  const int k = threadIdx.x >> 5, j = threadIdx.x & 31;  // block size index, node within this thread block
  if (k >= kTreeSizes || !R.obb[k] || j >= (4 >> k)) return;
  const uint32_t nodes = tree_level_count(R.num_tris, k + 1, 1);
  const uint32_t first = (blockIdx.x - static_cast<uint32_t>(group_starts[mesh])) * (4u >> k) + j;
  if (first >= nodes) return;
  for (int w = j * (2 << k); w < (j + 1) * (2 << k); ++w)
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      if (w == j * (2 << k)) {
        lo[x] = s_lo[w][x];
        hi[x] = s_hi[w][x];
      } else {
        lo[x] = fminf(lo[x], s_lo[w][x]);
        hi[x] = fmaxf(hi[x], s_hi[w][x]);
      }
    }
  put_box(R.box[k], first, lo, hi);
}

// Levels 2 and up of one mesh (blockIdx.x) and block size (blockIdx.y): a warp reduces 32 children.
__global__ __launch_bounds__(1024) void k_upper(const PTreeRec *__restrict__ trees) {
  const PTreeRec &R = trees[blockIdx.x];
  const int k = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  if (!R.obb[k]) return;
  float4 *box = R.box[k];
  uint32_t from = 0, n = tree_level_count(R.num_tris, k + 1, 1);
  while (n > 1) {
    const uint32_t up = (n + 31) / 32, to = from + n;
    for (uint32_t i = warp; i < up; i += warps) {
      const uint32_t ch = min(i * 32 + lane, n - 1);
      const float4 c = box[2 * size_t(from + ch)], e = box[2 * size_t(from + ch) + 1];
      float lo[3] = {__fsub_rd(c.x, e.x), __fsub_rd(c.y, e.y), __fsub_rd(c.z, e.z)};
      float hi[3] = {__fadd_ru(c.x, e.x), __fadd_ru(c.y, e.y), __fadd_ru(c.z, e.z)};
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        lo[x] = group_min(lo[x], kWarp);
        hi[x] = group_max(hi[x], kWarp);
      }
      if (lane == 0) put_box(box, to + i, lo, hi);
    }
    __syncthreads();
    from = to;
    n = up;
  }
}

struct BuildTemp {
  uint64_t *keys, *keys_alt;
  uint32_t *vals, *vals_alt, *bounds;
  void *scratch;
  size_t scratch_bytes;
};

size_t temp_layout(uint64_t T, int M, char *base, BuildTemp *t) {
  const size_t n = std::max<uint64_t>(T, 1);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char *p = base ? base + off : nullptr;
    off += align256(bytes);
    return p;
  };
  BuildTemp x;
  x.keys = reinterpret_cast<uint64_t *>(take(n * 8));
  x.keys_alt = reinterpret_cast<uint64_t *>(take(n * 8));
  x.vals = reinterpret_cast<uint32_t *>(take(n * 4));
  x.vals_alt = reinterpret_cast<uint32_t *>(take(n * 4));
  x.bounds = reinterpret_cast<uint32_t *>(take(size_t(M) * 24));
  x.scratch_bytes = sort_scratch_bytes(n);
  x.scratch = take(x.scratch_bytes);
  if (t) *t = x;
  return off;
}

}  // namespace

size_t ptree_temp_bytes(uint64_t total_tris, int num_meshes) {
  return temp_layout(total_tris, num_meshes, nullptr, nullptr);
}

size_t ptree_layout(uint32_t T, int mask, char *base, PTreeRec *out) {
  PTreeRec r{};
  r.num_tris = T;
  r.slots = static_cast<uint32_t>((uint64_t(T) + kTreePad - 1) / kTreePad * kTreePad);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char *p = base ? base + off : nullptr;
    off += align256(bytes);
    return p;
  };
  r.tri = reinterpret_cast<float4 *>(take(size_t(r.slots) * sizeof(DistTri)));
  for (int k = 0; k < kTreeSizes; ++k) {
    if (!(mask >> k & 1)) continue;
    r.obb[k] = reinterpret_cast<float4 *>(take(size_t(r.slots >> (k + 1)) * 64));
    size_t nodes = 0;
    for (int l = 1;; ++l) {
      const uint32_t n = tree_level_count(T, k + 1, l);
      nodes += n;
      if (n <= 1) break;
    }
    r.box[k] = reinterpret_cast<float4 *>(take(nodes * 32));
  }
  if (out) *out = r;
  return off;
}

cudaError_t ptree_build(const BatchDev &B, const PTreeRec *trees, const uint64_t *group_starts, uint64_t groups,
                        void *temp, size_t temp_bytes, uint32_t *err, cudaStream_t st) {
  const uint64_t T = B.total_tris;
  const int M = B.num_meshes;
  if (T == 0 || M == 0 || T >= (1ull << 31)) return cudaErrorInvalidValue;
  BuildTemp t;
  if (temp_layout(T, M, static_cast<char *>(temp), &t) > temp_bytes) return cudaErrorMemoryAllocation;
  k_init_bounds<<<(6 * M + 255) / 256, 256, 0, st>>>(t.bounds, M);
  note_launch();
  k_prep<<<blocks_for(T), kThreads, 0, st>>>(B, t.bounds, err);
  note_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (T > 1) {
    k_keys<<<blocks_for(T), kThreads, 0, st>>>(B, t.bounds, t.keys, t.vals);
    note_launch();
    int mesh_bits = 0;
    while ((1 << mesh_bits) < M) ++mesh_bits;
    if ((e = radix_sort_pairs(t.keys, t.vals, t.keys_alt, t.vals_alt, T, 30 + mesh_bits,
                              Scratch{t.scratch, t.scratch_bytes}, st)) != cudaSuccess)
      return e;
  }
  k_pack<<<static_cast<unsigned>(groups), kThreads, 0, st>>>(B, trees, group_starts, t.vals);
  note_launch();
  k_upper<<<dim3(M, kTreeSizes), 1024, 0, st>>>(trees);
  note_launch();
  return cudaGetLastError();
}

}  // namespace sdfb
