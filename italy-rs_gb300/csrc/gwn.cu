// Generalized winding number sign for meshes that are not watertight (replaces the 5-ray parity
// vote of src/render/kernels/sdf_bake.cu:53-69, which assumes a closed mesh).
//
// w(q) = sum of triangle solid angles / 4 pi (Jacobson, Kavan & Sorkine-Hornung 2013); a cell is
// inside when |w| > 0.5. It is evaluated through an exact decomposition: the bake closes every
// boundary loop of the mesh with a small fan cap (caps.cu), so mesh + caps has no boundary
// and its winding number W(q) is an integer, namely the signed count of +z crossings above q
// (parity.cu stores each crossing's orientation). Then
//     w(q) = W(q) - w_caps(q),
// and only the caps -- small triangles hugging the holes -- need solid angles. A cap subtree far
// from q is replaced by its dipole term with a rigorous error bound (the far field of Barill et al.
// 2018, "Fast Winding Numbers for Soups and Clouds", with a Taylor bound of our own): a triangle
// of area a and unit normal n subtends the integral over it of f(x) = (x - q) . n / |x - q|^3,
// whose gradient is at most 2 / |x - q|^3 in length. For a cluster inside the ball of radius rho
// about c, at r = |c - q| > rho,
//     Omega = D . (c - q) / r^3  +/-  A * 2 rho / (r - rho)^3,    D = sum a_i n_i,  A = sum a_i,
// with (D, A) stored per node (lbvh.cu) and (c, rho) the child box's centre and half diagonal. A
// subtree is taken as its dipole when that bound is at most tau, and a cell is decided as soon as
// the summed bounds cannot move |w| across 0.5.
//
// A group of cells (a warp's tile, or 32 listed cells) is walked together: the lanes stand for nodes
// of the caps' hierarchy, and a subtree is taken for the whole group with the group's centre in
// place of q, which only adds the group's radius to rho (both the cluster's and the cell's offset
// move the argument of f): Omega(q) = D . (c - q0) / r^3 +/- A * 2 (rho + rho_g) / (r - rho - rho_g)^3.
// The lanes' sums are added up once; only leaves too close for that are measured by every cell.
// (Cells as lanes took 22,000 instructions a tile of 128 cells: pass 1 at 512^3 24.8 -> 7.7 ms; the
// band's two passes and the direct sum 20.5 -> 4.5 ms.)
//
// Precision split:
//   pass 1 (FP32, every cell of every winding-number mesh, warp tiles of 4 x 4 x 8, four cells
//     of a column per lane): cells outside the band (|d| > band_voxels * voxel) whose interval
//     [c - e, c + e] lies on one side of |w| = 0.5 get their sign; the band and undecided cells
//     go to a refine list.
//   pass 2 (FP64 accumulation, 32 listed cells a warp): first with coarse subtrees (kTau64) and the
//     near caps' solid angles in FP32 with a bound on their rounding error (solid_angle_bounded),
//     then the cells that stay undecided twice more with fine subtrees (kTau64Fine, kTau64Finest), a
//     warp to a cell and solid angles in FP64; a cell still undecided goes to
//   pass 3 (FP64 sum over every cap triangle of its mesh, one block per cell), which takes the coarse
//     pass's cells at once when they and the caps are few.
// A sign is only given where the summed bounds prove it, so the FP32 solid angles of pass 2 change
// none: they filter the cells that need FP64 ones (FP64 runs at 1/64 of the FP32 rate here).
#include <algorithm>
#include <cstdint>

#include "api_internal.h"
#include "common.cuh"

using namespace sdfb;

namespace {

constexpr int kThreads = 256;
constexpr int kMinBlocks = 3;  // 80 registers: sign stage of the 512^3 scene 11.6 ms at 2, 10.1 at 3, 11.5 at 4
constexpr int kWarps = kThreads / kWarp;
constexpr double kInv4Pi = 0.07957747154594767;
// Largest far-field error bound (sr) taken for one cap subtree. A cell is decided once the summed
// bounds cannot move |w| across 0.5, and most cells have a margin near 0.5, so pass 1 takes coarse
// subtrees. The band's bound is finer: what it leaves costs a warp a cell. The few cells near the
// level set itself are walked with ever finer subtrees before the direct sum (~7 us a cell) gets what
// is left. Sign stage of five 500k-triangle scenes at 512^3 (1.6 M cells in the band): kTau64 0.3
// 12-132 ms (where components overlap many bounds add up), 0.1 12-89, 3e-2 11.7-13.4, 1e-2 12.2-15.0,
// 3e-3 14-19. One fine pass instead of two, on the first scene: 1e-2 21.2 ms (1,674 cells summed
// directly), 1e-3 14.0 ms (466), 1e-4 14.0 ms (143), 1e-5 21.2 ms (26); 1e-3 then 2e-5 12.0 ms (55).
constexpr float kTau32 = 1e-1f;
constexpr float kTau64 = 2e-2f;
constexpr float kTau64Fine = 1e-3f;
constexpr float kTau64Finest = 2e-5f;

template <typename T> struct V3 {
  T x, y, z;
};

// Exact solid angle of triangle (a, b, c) seen from the origin (Van Oosterom & Strackee 1983).
template <typename T>
__device__ __forceinline__ T solid_angle(V3<T> a, V3<T> b, V3<T> c) {
  const T la = sqrt(a.x * a.x + a.y * a.y + a.z * a.z);
  const T lb = sqrt(b.x * b.x + b.y * b.y + b.z * b.z);
  const T lc = sqrt(c.x * c.x + c.y * c.y + c.z * c.z);
  const T det = a.x * (b.y * c.z - b.z * c.y) - a.y * (b.x * c.z - b.z * c.x) + a.z * (b.x * c.y - b.y * c.x);
  const T ab = a.x * b.x + a.y * b.y + a.z * b.z, bc = b.x * c.x + b.y * c.y + b.z * c.z,
          ca = c.x * a.x + c.y * a.y + c.z * a.z;
  const T den = la * lb * lc + ab * lc + bc * la + ca * lb;
  return T(2) * atan2(det, den);
}

// The same in FP32 with a bound on its error. With u = 2^-24, lengths la, lb, lc of the three rounded
// differences and L = la lb lc: the determinant carries at most 16 u L (3 u from the differences,
// 6 u from its operations, times sqrt(3) for the sum of the products' magnitudes) and the
// denominator 50 u L (11 u in the product of lengths, 9 u in each of the other three terms, 3 u of
// the partial sums), so the vector (den, det) of length R moves by at most 53 u L and the angle 2 atan2
// by at most 2.2 * 53 u L / R while that is below a quarter, plus the rounding of atan2f and of the
// sum, unless the move takes the vector across the cut of atan2 (den < 0, det = 0: the point lies in the
// triangle, to rounding), where the angle jumps by 4 pi. There, otherwise, and for a NaN, nothing is known:
// |Omega| <= 2 pi on both sides. L / R is taken from det and den over L, whose squares stay in range where
// those of the cubes det and den do not (from lengths of 2.6e6 on). Lengths whose own squares or products come
// near the ends of FP32's range are not known either: den is at most 4 L, and what underflows is below 1e-12
// of L.
__device__ __forceinline__ float solid_angle_bounded(V3<float> a, V3<float> b, V3<float> c, float &err) {
  const float aa = a.x * a.x + a.y * a.y + a.z * a.z, bb = b.x * b.x + b.y * b.y + b.z * b.z,
              cc = c.x * c.x + c.y * c.y + c.z * c.z;
  const float la = sqrtf(aa), lb = sqrtf(bb), lc = sqrtf(cc);
  const float det = a.x * (b.y * c.z - b.z * c.y) - a.y * (b.x * c.z - b.z * c.x) + a.z * (b.x * c.y - b.y * c.x);
  const float ab = a.x * b.x + a.y * b.y + a.z * b.z, bc = b.x * c.x + b.y * c.y + b.z * c.z,
              ca = c.x * a.x + c.y * a.y + c.z * a.z;
  const float L = la * lb * lc;
  const float den = L + ab * lc + bc * la + ca * lb;
  const float s = 1.0f / L, x = den * s, y = det * s;
  const float rel = rsqrtf(x * x + y * y);
  const bool in_range = L < 8e37f && fminf(L, fminf(aa, fminf(bb, cc))) > 1e-32f;
  const bool cut = x < 4e-6f && fabsf(y) < 2e-6f;  // 50 u and 16 u are 3e-6 and 1e-6
  err = in_range && !cut && rel < 7e4f ? fmaf(8e-6f, rel, 2e-6f) : 13.0f;
  return 2.0f * atan2f(det, den);
}

// Up to 32 of a tile's cells left to pass 2, from the (32 part)-th on: bit l of cells[v] is lane l's
// cell v. A part is a warp's work there: whole tiles leave the last warps with four walks each (10k
// triangles at res 100: k_gwn64 199 us for 96).
struct TileCells {
  uint64_t tile_part;  // tile | part << kPartShift
  uint32_t cells[kGwnCellsPerLane];
};
constexpr int kPartShift = 56;

struct GwnArgs {
  BatchDev batch;  // each GWN mesh record names its caps hierarchy
  const uint64_t *col_start;
  const float *col_z;
  const int8_t *col_s;
  uint64_t capacity;  // of col_z and col_s
  float band_voxels;
  TileCells *tiles;  // pass 1 -> pass 2 (coarse): tiles' parts with cells to refine
  unsigned long long *listed_tiles, *refine_count;  // their number, and their cells'
  uint64_t *cells;  // pass 2 (coarse) -> pass 2 (fine): global cells
  unsigned long long *cell_count;
  unsigned long long *tile_counter;
  uint32_t most_caps;  // of a mesh
  uint32_t *err;
};

// Whether the cells that the coarse pass left are summed directly. The two fine passes take at least
// the latency of one cell's walk each, 100 and 190 us at 600 caps and 0.35 ms at 3600, however few the
// cells; the direct sum takes about 75 cycles of an SM a cap and cell, 0.5 ms at the bound. Sign stage
// with the fine passes and without: 50 cells, 600 caps 0.60-0.77 -> 0.37-0.44 ms; 200 cells, 3600 caps
// 1.66-1.80 -> 0.92-0.97 ms.
constexpr unsigned long long kDirectWork = 1 << 21;  // caps times cells
__device__ __forceinline__ bool few(const GwnArgs &a) { return *a.cell_count * a.most_caps <= kDirectWork; }

// A column's crossings in the lists: [s0, s1). Where the lists are too short for all crossings the columns'
// starts pass their end: what is beyond it was not written, and is not read (the bake is repeated).
__device__ __forceinline__ void column_list(const GwnArgs &a, const MeshRec &M, int vx, int vy, uint64_t &s0,
                                            uint64_t &s1) {
  const uint64_t col = M.col_base + uint64_t(vy) * M.g.nx + vx;
  s0 = __ldg(a.col_start + col);
  s1 = min(__ldg(a.col_start + col + 1), a.capacity);
}

// Signed crossings of the column above height pz (the integer winding number of mesh + caps).
__device__ __forceinline__ int column_winding(const GwnArgs &a, const MeshRec &M, int vx, int vy, float pz) {
  uint64_t s0, s1;
  column_list(a, M, vx, vy, s0, s1);
  int w = 0;
  for (uint64_t k = s0; k < s1; ++k)
    if (__ldg(a.col_z + k) > pz) w += __ldg(a.col_s + k);
  return w;
}

// The same for V heights of one column, reading its crossings once.
template <int V>
__device__ __forceinline__ void column_windings(const GwnArgs &a, const MeshRec &M, int vx, int vy,
                                                const float (&pz)[V], int (&w)[V]) {
  uint64_t s0, s1;
  column_list(a, M, vx, vy, s0, s1);
#pragma unroll
  for (int v = 0; v < V; ++v) w[v] = 0;
  for (uint64_t k = s0; k < s1; ++k) {
    const float z = __ldg(a.col_z + k);
    const int s = __ldg(a.col_s + k);
#pragma unroll
    for (int v = 0; v < V; ++v) w[v] += z > pz[v] ? s : 0;
  }
}

// (D, A) of a leaf's cap triangles (D = half the sum of their edge cross products, A = half the
// sum of their lengths, which the records hold).
__device__ __forceinline__ float4 leaf_moment(const TriRec *tr, int count) {
  float4 m = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (int j = 0; j < count; ++j) {
    const float4 r3 = __ldg(&tr[j].r3);
    m.x += 0.5f * r3.x;
    m.y += 0.5f * r3.y;
    m.z += 0.5f * r3.z;
    m.w += 0.5f * r3.w;
  }
  return m;
}

// The far field of a cap cluster -- moment m = (D, A), inside the child box of centre c and half
// extent e (so inside the ball of radius |e| about c) -- seen from every point within rho_g of q:
// false when they are too close (r <= 2 (|e| + rho_g)) or the error bound exceeds tau; else
// val = D . (c - q) / r^3 and err bounds |Omega - val|. One reciprocal square root per distance and
// one approximate reciprocal for the bound (each within 2 ulp, far inside the 1e-5 margin that the
// bound carries); the acceptance test err <= tau is taken as A 2 rho <= tau g^3 with a 1e-6 margin. g^3 has
// to lie where both stay normal: __fdividef gives 0 for divisors above 2^126.
__device__ __forceinline__ bool far_field(float qx, float qy, float qz, float rho_g, const float4 &n0,
                                          const float4 &n1, const float4 &n2, int which, const float4 &m, float tau,
                                          float &val, float &err) {
  const float cx = which ? n1.z : n0.x, cy = which ? n1.w : n0.y, cz = which ? n2.x : n0.z;
  const float ex = which ? n2.y : n0.w, ey = which ? n2.z : n1.x, ez = which ? n2.w : n1.y;
  const float dx = cx - qx, dy = cy - qy, dz = cz - qz;
  const float r2 = dx * dx + dy * dy + dz * dz;
  const float rho2 = ex * ex + ey * ey + ez * ez;
  const float rho = (rho2 > 0.0f ? rho2 * rsqrtf(rho2) : 0.0f) + rho_g;
  if (!(r2 > 4.0f * rho * rho)) return false;
  const float ir = rsqrtf(r2);
  const float g = r2 * ir - rho;
  const float g3 = g * g * g;
  const float lim = m.w * 2.0f * rho;
  if (!(g3 > 1e-30f && g3 < 8e37f) || !(lim <= tau * (1.0f - 1e-6f) * g3)) return false;
  val = (m.x * dx + m.y * dy + m.z * dz) * (ir * ir * ir);
  constexpr float kRel = 1e-5f;
  err = __fdividef(lim, g3) * (1.0f + kRel) + kRel * fabsf(val);
  return true;
}

// Shared memory of one warp's walk. The stack never overflows: when it is nearly full nodes are taken
// one at a time, depth first, which needs one entry a level (a radix tree over 64-bit keys and 32-bit
// positions has at most 96 levels).
constexpr int kStack = 512, kStackRoom = 128, kLeaves = 96;
struct CapMem {
  int stack[kStack];
  int2 leaf[kLeaves];  // node, child
};

// Caps of one mesh seen from the cells of a warp: V cells a lane in one column (q = (qx, qy, qz[v])),
// all active ones within rho_g of (gx, gy, gz). wex receives their summed solid angle, eps the error
// bound. T is the accumulation type; with LEAF64 the near caps' solid angles are FP64, else FP32 with
// their bound added to eps. q and the caps' vertices are FP32 values. SINGLE: the lanes all hold the
// same cell (V = 1, rho_g = 0), and share out the leaves too.
template <typename T, bool LEAF64, bool SINGLE, int V>
__device__ void caps_walk(const MeshRec &M, CapMem &mem, const bool (&active)[V], float qx, float qy,
                          const float (&qz)[V], float gx, float gy, float gz, float rho_g, float tau, T (&wex)[V],
                          T (&eps)[V], bool &corrupt) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  int sp = 1, nl = 0;
  float sval = 0.0f, serr = 0.0f;
  T tval = T(0), terr = T(0);
  __syncwarp();
  if (lane == 0) mem.stack[0] = M.cap_root;
  __syncwarp();

  // Leaves that are not far for the whole group: far for every cell, or exact.
  auto near_leaves = [&]() {
    if (SINGLE) {
      for (int i = lane; i < nl; i += kWarp) {
        const int2 lf = mem.leaf[i];
        const int4 n3 = __ldg(&(M.cap_nodes + lf.x)->n3);
        const TriRec *tr = M.cap_trec + (lf.y ? n3.y : n3.x);
        const int cnt = lf.y ? n3.w : n3.z;
        for (int j = 0; j < cnt; ++j) {
          const float4 r0 = __ldg(&tr[j].r0), r1 = __ldg(&tr[j].r1), r2 = __ldg(&tr[j].r2);
          tval += solid_angle<T>({T(r0.x) - T(qx), T(r0.y) - T(qy), T(r0.z) - T(qz[0])},
                                 {T(r1.x) - T(qx), T(r1.y) - T(qy), T(r1.z) - T(qz[0])},
                                 {T(r2.x) - T(qx), T(r2.y) - T(qy), T(r2.z) - T(qz[0])});
        }
      }
      __syncwarp();
      nl = 0;
      return;
    }
    for (int i = 0; i < nl; ++i) {
      const int2 lf = mem.leaf[i];
      const Node *np = M.cap_nodes + lf.x;
      const float4 n0 = __ldg(&np->n0), n1 = __ldg(&np->n1), n2 = __ldg(&np->n2);
      const int4 n3 = __ldg(&np->n3);
      const int ref = lf.y ? n3.y : n3.x, cnt = lf.y ? n3.w : n3.z;
      const TriRec *tr = M.cap_trec + ref;
      const float4 mom = leaf_moment(tr, cnt);
      float val[V], err[V];
      bool need = false;
#pragma unroll
      for (int v = 0; v < V; ++v) {
        val[v] = err[v] = 0.0f;
        need |= active[v] && !far_field(qx, qy, qz[v], 0.0f, n0, n1, n2, lf.y, mom, tau, val[v], err[v]);
      }
      if (!__any_sync(kFull, need)) {
#pragma unroll
        for (int v = 0; v < V; ++v) {
          wex[v] += T(val[v]);
          eps[v] += T(err[v]);
        }
        continue;
      }
      for (int j = 0; j < cnt; ++j) {
        const float4 r0 = __ldg(&tr[j].r0), r1 = __ldg(&tr[j].r1), r2 = __ldg(&tr[j].r2);
#pragma unroll
        for (int v = 0; v < V; ++v) {
          if (LEAF64) {
            const V3<T> a{T(r0.x) - T(qx), T(r0.y) - T(qy), T(r0.z) - T(qz[v])},
                b{T(r1.x) - T(qx), T(r1.y) - T(qy), T(r1.z) - T(qz[v])},
                c{T(r2.x) - T(qx), T(r2.y) - T(qy), T(r2.z) - T(qz[v])};
            wex[v] += solid_angle<T>(a, b, c);
          } else {
            const V3<float> a{r0.x - qx, r0.y - qy, r0.z - qz[v]}, b{r1.x - qx, r1.y - qy, r1.z - qz[v]},
                c{r2.x - qx, r2.y - qy, r2.z - qz[v]};
            float e;
            wex[v] += T(solid_angle_bounded(a, b, c, e));
            eps[v] += T(e);
          }
        }
      }
    }
    __syncwarp();
    nl = 0;
  };

  const long long step_limit = 2ll * M.cap_nodes_n + 64;
  for (long long steps = 0; sp > 0; ++steps) {
    if (steps > step_limit) {
      corrupt = true;
      break;
    }
    const int n = min(min(kWarp, sp), max(1, kStack - kStackRoom - sp));
    sp -= n;
    const bool have = lane < n;
    const int node = have ? mem.stack[sp + lane] : M.cap_root;
    __syncwarp();
    const bool ok = node >= 0 && node < M.cap_nodes_n;
    corrupt |= !ok;
    const Node *np = M.cap_nodes + (ok ? node : M.cap_root);
    const float4 n0 = __ldg(&np->n0), n1 = __ldg(&np->n1), n2 = __ldg(&np->n2);
    const int4 n3 = __ldg(&np->n3);
    const int refs[2] = {n3.x, n3.y}, cnts[2] = {n3.z, n3.w};
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      bool down = false, leaf = false;
      if (have && ok && cnts[k] >= 0) {
        float4 mom = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        bool sound = true;
        if (cnts[k] == 0) {
          sound = refs[k] >= 0 && refs[k] < M.cap_inner_n;
          if (sound) mom = __ldg(M.cap_moment + refs[k]);
        } else {
          sound = refs[k] >= 0 && cnts[k] <= M.cap_recs_n - refs[k];
          if (sound) mom = leaf_moment(M.cap_trec + refs[k], cnts[k]);
        }
        corrupt |= !sound;
        float val, err;
        if (sound) {
          if (far_field(gx, gy, gz, rho_g, n0, n1, n2, k, mom, tau, val, err)) {
            sval += val;
            serr += err;
          } else {
            down = cnts[k] == 0;
            leaf = !down;
          }
        }
      }
      const unsigned md = __ballot_sync(kFull, down), ml = __ballot_sync(kFull, leaf);
      if (down) mem.stack[sp + __popc(md & below)] = refs[k];
      if (leaf) mem.leaf[nl + __popc(ml & below)] = make_int2(node, k);
      sp += __popc(md);
      nl += __popc(ml);
      __syncwarp();
      if (nl > kLeaves - kWarp) near_leaves();
    }
    if (sizeof(T) == 8) {  // FP64 accumulation: fold the lanes' few FP32 terms in step by step
      tval += T(sval);
      terr += T(serr);
      sval = serr = 0.0f;
    }
  }
  if (nl > 0) near_leaves();
  tval += T(sval);
  terr += T(serr);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    tval += __shfl_xor_sync(kFull, tval, o);
    terr += __shfl_xor_sync(kFull, terr, o);
  }
#pragma unroll
  for (int v = 0; v < V; ++v) {
    wex[v] += tval;
    eps[v] += terr;
  }
}

// A warp's tile of 4 x 4 x kGwnTileZ cells: kGwnCellsPerLane cells a lane, two layers apart.
struct GwnTile {
  int mesh, x0, y0, z0;
  __device__ __forceinline__ GwnTile(const BatchDev &B, unsigned long long tile) {
    mesh = find_mesh(B.gwn_tile_starts, B.num_meshes, tile);
    const GridDev &g = B.recs[mesh].g;
    const unsigned long long local = tile - B.gwn_tile_starts[mesh];
    const int tiles_x = (g.nx + 3) / 4, tiles_y = (g.ny + 3) / 4;
    const unsigned long long rest = local / tiles_x;
    x0 = static_cast<int>(local % tiles_x) * 4;
    y0 = static_cast<int>(rest % tiles_y) * 4;
    z0 = static_cast<int>(rest / tiles_y) * kGwnTileZ;
  }
  __device__ __forceinline__ int vx(int lane) const { return x0 + lane % 4; }
  __device__ __forceinline__ int vy(int lane) const { return y0 + (lane / 4) % 4; }
  __device__ __forceinline__ int vz(int lane, int v) const { return z0 + lane / 16 + 2 * v; }
  // The tile's centre, and its half diagonal with room for the cell centres' rounding.
  __device__ __forceinline__ float centre(const GridDev &g, float &gx, float &gy, float &gz) const {
    gx = g.ox + (float(x0) + 2.0f) * g.voxel;
    gy = g.oy + (float(y0) + 2.0f) * g.voxel;
    gz = g.oz + (float(z0) + 0.5f * kGwnTileZ) * g.voxel;
    constexpr float rx = 1.5f, rz = 0.5f * (kGwnTileZ - 1);
    return 1.0001f * g.voxel * sqrtf(2.0f * rx * rx + rz * rz) +
           1e-6f * (fabsf(g.ox) + fabsf(g.oy) + fabsf(g.oz) + fabsf(gx) + fabsf(gy) + fabsf(gz));
  }
};

// Pass 1: FP32 over the tiles of the winding-number meshes.
__global__ __launch_bounds__(kThreads, kMinBlocks) void k_gwn32(GwnArgs a) {
  constexpr int V = kGwnCellsPerLane;
  const int lane = threadIdx.x & 31;
  const BatchDev &B = a.batch;
  bool corrupt = false;
  __shared__ CapMem s_mem[kWarps];
  CapMem &mem = s_mem[threadIdx.x >> 5];
  for (;;) {
    unsigned long long tile = 0;
    if (lane == 0) tile = atomicAdd(a.tile_counter, 1ull);
    tile = __shfl_sync(kFull, tile, 0);
    if (tile >= B.total_gwn_tiles) break;
    const GwnTile t(B, tile);
    const MeshRec &M = B.recs[t.mesh];
    const GridDev g = M.g;
    const int vx = t.vx(lane), vy = t.vy(lane);
    bool active[V];
    float qz[V], wex[V], eps[V];
    bool any_active = false;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      active[v] = vx < g.nx && vy < g.ny && t.vz(lane, v) < g.nz;
      any_active |= active[v];
      qz[v] = cell_center(g.oz, t.vz(lane, v), g.voxel);
      wex[v] = 0.0f;
      eps[v] = 0.0f;
    }
    if (M.cap_root >= 0) {
      float gx, gy, gz;
      const float rho_g = t.centre(g, gx, gy, gz);
      caps_walk<float, false, false, V>(M, mem, active, cell_center(g.ox, vx, g.voxel), cell_center(g.oy, vy, g.voxel),
                                        qz, gx, gy, gz, rho_g, kTau32, wex, eps, corrupt);
    }
    int W[V];
    if (any_active) column_windings<V>(a, M, vx, vy, qz, W);
    uint32_t left[V];
    int count = 0;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      bool refine = false;
      if (active[v]) {
        const uint64_t cell = (uint64_t(t.vz(lane, v)) * g.ny + vy) * g.nx + vx;
        const float d = M.dist[cell];
        const float c = fabsf(float(W[v]) - wex[v] * float(kInv4Pi));
        const float e = eps[v] * float(kInv4Pi) + 1e-5f * (1.0f + fabsf(wex[v]));
        const bool band = d <= a.band_voxels * g.voxel;
        if (!band && c - e > 0.5f) M.dist[cell] = -d;
        else refine = band || !(c + e < 0.5f);
      }
      left[v] = __ballot_sync(kFull, refine);
      count += __popc(left[v]);
    }
    if (count) {
      const int parts = (count + kWarp - 1) / kWarp;
      unsigned long long at = 0;
      if (lane == 0) {
        at = atomicAdd(a.listed_tiles, static_cast<unsigned long long>(parts));
        atomicAdd(a.refine_count, static_cast<unsigned long long>(count));
      }
      at = __shfl_sync(kFull, at, 0);
      if (lane < parts) {
        TileCells &o = a.tiles[at + lane];
        o.tile_part = tile | uint64_t(lane) << kPartShift;
#pragma unroll
        for (int v = 0; v < V; ++v) o.cells[v] = left[v];
      }
    }
  }
  if (corrupt) atomic_or_err(a.err, kErrCorruptTree);
}

// Gives an FP64 interval's sign to a cell; true when it does not decide.
__device__ __forceinline__ bool undecided64(const MeshRec &M, uint64_t cell, int W, double wex, double eps) {
  const double c = fabs(double(W) - wex * kInv4Pi);
  const double e = eps * kInv4Pi + 1e-12 * (1.0 + fabs(wex)) + 1e-6;  // 1e-6: the far field's FP32 sums
  if (c - e > 0.5) {
    M.dist[cell] = -fabsf(M.dist[cell]);
    return false;
  }
  return !(c + e < 0.5);
}

// Pass 2, coarse: a listed tile's cells, 32 a warp. The list lengths are read on the device, so no
// pass needs a host round trip.
__global__ __launch_bounds__(kThreads, kMinBlocks) void k_gwn64(GwnArgs a) {
  const unsigned long long n = *a.listed_tiles;
  const int lane = threadIdx.x & 31;
  const BatchDev &B = a.batch;
  bool corrupt = false;
  __shared__ CapMem s_mem[kWarps];
  CapMem &mem = s_mem[threadIdx.x >> 5];
  for (unsigned long long k = blockIdx.x * (unsigned long long)kWarps + (threadIdx.x >> 5); k < n;
       k += (unsigned long long)gridDim.x * kWarps) {
    const TileCells &in = a.tiles[k];
    const GwnTile t(B, in.tile_part & ((1ull << kPartShift) - 1));
    const MeshRec &M = B.recs[t.mesh];
    const GridDev g = M.g;
    float gx, gy, gz;
    const float rho_g = t.centre(g, gx, gy, gz);
    int total = 0;
#pragma unroll
    for (int v = 0; v < kGwnCellsPerLane; ++v) total += __popc(in.cells[v]);
    // this lane's cell: the (base + lane)-th listed one of the tile
    const int base = static_cast<int>(in.tile_part >> kPartShift) * kWarp;
    const bool active = base + lane < total;
    int rank = active ? base + lane : base, v = 0;
#pragma unroll
    for (int j = 0; j < kGwnCellsPerLane - 1; ++j) {
      const int c = __popc(in.cells[j]);
      if (v == j && rank >= c) {
        rank -= c;
        ++v;
      }
    }
    const int src = __fns(in.cells[v], 0, rank + 1);
    const int vx = t.vx(src), vy = t.vy(src), vz = t.vz(src, v);
    const float qz[1] = {cell_center(g.oz, vz, g.voxel)};
    const bool act[1] = {active};
    double wex[1] = {0.0}, eps[1] = {0.0};
    if (M.cap_root >= 0)
      caps_walk<double, false, false, 1>(M, mem, act, cell_center(g.ox, vx, g.voxel), cell_center(g.oy, vy, g.voxel),
                                         qz, gx, gy, gz, rho_g, kTau64, wex, eps, corrupt);
    const uint64_t cell = (uint64_t(vz) * g.ny + vy) * g.nx + vx;
    const bool left = active && undecided64(M, cell, column_winding(a, M, vx, vy, qz[0]), wex[0], eps[0]);
    const unsigned mask = __ballot_sync(kFull, left);
    if (mask) {
      unsigned long long at = 0;
      if (lane == 0) at = atomicAdd(a.cell_count, static_cast<unsigned long long>(__popc(mask)));
      at = __shfl_sync(kFull, at, 0) + __popc(mask & ((1u << lane) - 1u));
      if (left) a.cells[at] = B.cell_starts[t.mesh] + cell;
    }
  }
  if (corrupt) atomic_or_err(a.err, kErrCorruptTree);
}

__device__ __forceinline__ void cell_of(const BatchDev &B, uint64_t gcell, int &mesh, int &vx, int &vy, int &vz,
                                        uint64_t &cell) {
  mesh = find_mesh(B.cell_starts, B.num_meshes, gcell);
  const GridDev &g = B.recs[mesh].g;
  cell = gcell - B.cell_starts[mesh];
  vx = static_cast<int>(cell % uint64_t(g.nx));
  vy = static_cast<int>((cell / uint64_t(g.nx)) % uint64_t(g.ny));
  vz = static_cast<int>(cell / (uint64_t(g.nx) * g.ny));
}

// Pass 2, fine: a warp per listed cell, its lanes sharing the walk and the FP64 solid angles. Cells
// that stay undecided go from `in` to `out`.
__global__ __launch_bounds__(kThreads) void k_gwn64_fine(GwnArgs a, float tau, const uint64_t *__restrict__ in,
                                                         const unsigned long long *in_count, uint64_t *out,
                                                         unsigned long long *out_count) {
  if (few(a)) return;
  const unsigned long long n = *in_count;
  const int lane = threadIdx.x & 31;
  const BatchDev &B = a.batch;
  bool corrupt = false;
  __shared__ CapMem s_mem[kWarps];
  CapMem &mem = s_mem[threadIdx.x >> 5];
  for (unsigned long long k = blockIdx.x * (unsigned long long)kWarps + (threadIdx.x >> 5); k < n;
       k += (unsigned long long)gridDim.x * kWarps) {
    int mesh, vx, vy, vz;
    uint64_t cell;
    cell_of(B, in[k], mesh, vx, vy, vz, cell);
    const MeshRec &M = B.recs[mesh];
    const GridDev g = M.g;
    const float qx = cell_center(g.ox, vx, g.voxel), qy = cell_center(g.oy, vy, g.voxel);
    const float qz[1] = {cell_center(g.oz, vz, g.voxel)};
    const bool act[1] = {true};
    double wex[1] = {0.0}, eps[1] = {0.0};
    if (M.cap_root >= 0)
      caps_walk<double, true, true, 1>(M, mem, act, qx, qy, qz, qx, qy, qz[0], 0.0f, tau, wex, eps, corrupt);
    if (lane == 0 && undecided64(M, cell, column_winding(a, M, vx, vy, qz[0]), wex[0], eps[0]))
      out[atomicAdd(out_count, 1ull)] = in[k];
  }
  if (corrupt) atomic_or_err(a.err, kErrCorruptTree);
}

// Pass 3: one block per remaining cell, FP64 sum over every cap triangle of its mesh.
__global__ __launch_bounds__(kThreads) void k_gwn_direct(GwnArgs a, unsigned long long *last_count) {
  __shared__ double part[kThreads / kWarp];
  const BatchDev &B = a.batch;
  const uint64_t *__restrict__ in = a.cells;
  unsigned long long n;
  if (few(a)) {
    n = *a.cell_count;
    if (blockIdx.x == 0 && threadIdx.x == 0) *last_count = n;
  } else {
    n = *last_count;
  }
  for (unsigned long long k = blockIdx.x; k < n; k += gridDim.x) {
    int mesh, vx, vy, vz;
    uint64_t cell;
    cell_of(B, in[k], mesh, vx, vy, vz, cell);
    const MeshRec &M = B.recs[mesh];
    const GridDev g = M.g;
    const float fz = cell_center(g.oz, vz, g.voxel);
    const double qx = cell_center(g.ox, vx, g.voxel), qy = cell_center(g.oy, vy, g.voxel), qz = fz;
    double w = 0.0;
    for (uint32_t t = threadIdx.x; t < M.cap_tris; t += kThreads) {
      V3<double> p[3];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const uint32_t i = __ldg(M.cidx + 3ull * t + j);
        p[j] = {double(__ldg(M.cverts + 3ull * i)) - qx, double(__ldg(M.cverts + 3ull * i + 1)) - qy,
                double(__ldg(M.cverts + 3ull * i + 2)) - qz};
      }
      w += solid_angle<double>(p[0], p[1], p[2]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(kFull, w, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = w;
    __syncthreads();
    if (threadIdx.x == 0) {
      double s = 0.0;
      for (int i = 0; i < kThreads / kWarp; ++i) s += part[i];
      const int W = column_winding(a, M, vx, vy, fz);
      if (fabs(double(W) - s * kInv4Pi) > 0.5) M.dist[cell] = -fabsf(M.dist[cell]);
    }
    __syncthreads();
  }
}

}  // namespace

namespace {
// counters | cells of the coarse pass | cells of the fine pass, sharing their room with the tiles' list
// (read by the coarse pass alone; 24 bytes for 32 cells of a tile)
size_t list_bytes(uint64_t gwn_cells) { return (gwn_cells * 8 + 255) & ~size_t(255); }
size_t tile_list_bytes(uint64_t gwn_tiles) {
  return (gwn_tiles * kGwnCellsPerLane * sizeof(TileCells) + 255) & ~size_t(255);
}
}  // namespace

size_t gwn_temp_bytes(uint64_t gwn_cells, uint64_t gwn_tiles) {
  return 256 + list_bytes(gwn_cells) + std::max(list_bytes(gwn_cells), tile_list_bytes(gwn_tiles));
}

cudaError_t gwn_enqueue(const GwnInput &in, void *temp, int num_sms, cudaStream_t st) {
  const BatchDev &B = in.batch;
  if (B.total_gwn_tiles == 0) return cudaSuccess;
  char *base = static_cast<char *>(temp);
  unsigned long long *counters = reinterpret_cast<unsigned long long *>(base);
  GwnArgs a;
  a.batch = B;
  a.col_start = in.col_start;
  a.col_z = in.col_z;
  a.col_s = in.col_s;
  a.capacity = in.capacity;
  a.band_voxels = in.band_voxels;
  a.tile_counter = counters;
  a.refine_count = counters + 1;
  a.listed_tiles = counters + 2;
  a.cell_count = counters + 4;
  unsigned long long *last_count = counters + 3, *fine_count = counters + 5;
  a.cells = reinterpret_cast<uint64_t *>(base + 256);
  a.tiles = reinterpret_cast<TileCells *>(base + 256 + list_bytes(in.gwn_cells));
  uint64_t *fine = reinterpret_cast<uint64_t *>(a.tiles);  // the coarse pass has read the tiles by then (stream order)
  a.most_caps = in.most_caps;
  a.err = in.err;
  cudaError_t e = cudaMemsetAsync(counters, 0, 64, st);
  if (e != cudaSuccess) return e;
  // A whole wave of resident blocks, each kernel at its own occupancy.
  auto resident = [&](auto *kernel) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, 0);
    return static_cast<long long>(num_sms) * std::max(per_sm, 1);
  };
  static const long long wave32 = resident(k_gwn32), wave64 = resident(k_gwn64), wave_fine = resident(k_gwn64_fine);
  const long long blocks = std::min<long long>(wave32, static_cast<long long>((B.total_gwn_tiles + kWarps - 1) / kWarps));
  k_gwn32<<<static_cast<unsigned>(std::max<long long>(blocks, 1)), kThreads, 0, st>>>(a);
  note_launch();
  k_gwn64<<<static_cast<unsigned>(wave64), kThreads, 0, st>>>(a);
  note_launch();
  k_gwn64_fine<<<static_cast<unsigned>(wave_fine), kThreads, 0, st>>>(a, kTau64Fine, a.cells, a.cell_count, fine,
                                                                      fine_count);
  note_launch();
  k_gwn64_fine<<<static_cast<unsigned>(wave_fine), kThreads, 0, st>>>(a, kTau64Finest, fine, fine_count, a.cells,
                                                                      last_count);
  note_launch();
  k_gwn_direct<<<static_cast<unsigned>(num_sms * 4), kThreads, 0, st>>>(a, last_count);
  note_launch();
  return cudaGetLastError();
}

uint64_t *gwn_refine_counter(void *temp) { return reinterpret_cast<uint64_t *>(static_cast<char *>(temp)) + 1; }

uint64_t *gwn_direct_counter(void *temp) { return reinterpret_cast<uint64_t *>(static_cast<char *>(temp)) + 3; }
