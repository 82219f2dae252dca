// Nearest-triangle distance per cell with the sign fused in (replaces the 160-ray estimate of
// src/render/kernels/sdf_bake.cu:39-51 with the exact Euclidean distance).
//
// Work unit: a warp owns a tile of TX x TY x TZ cells (32 lanes, VPL cells per lane stacked in z),
// taken from its block's chunk of neighbouring tiles. It walks the packed 32-ary tree (ptree.cu)
// and changes what its lanes stand for on the way down:
//
//   lanes = children   a node's 32 children (boxes; at the last level the blocks' oriented boxes)
//                      are tested at once, each lane deciding for the whole tile whether its child
//                      can hold a triangle nearer than the bounds found so far;
//   lanes = cells      a block that survives is measured against every cell of the tile by the
//                      distance to its oriented box; the cells that it could improve become
//                      (block, cell) pairs in shared memory;
//   lanes = triangles  pairs are taken 32 / n at a time, n lanes computing the exact distances to a
//                      block's n triangles; the minimum goes to the cell's bound in shared memory. A block
//                      that most cells want is measured by all of them instead, lanes = cells.
//
// Before, all lanes were cells throughout: every node and triangle was tested by 128 cells although
// most die on the first one's answer, 50-70 instructions a triangle. Testing children by lanes costs
// about 4 instructions a child, and the exact test runs only for pairs that need it.
//
// Whole-tile test. Let c be the tile's centre and delta = q - c for a cell q. For a convex child
// (box) with nearest point p to c, e = c - p, d = |e|, n = e / d, the child lies behind the plane
// through p with normal n, so its distance to q is at least d + n . delta; and if its farthest
// point from p is at D, its squared distance is at least d^2 + 2 e . delta + |delta|^2 - K with
// K = D (2 rho - D) for D < rho, else rho^2, rho = max |delta| (|x - p|^2 + 2 delta . (p - x)
// minimised over |x - p| <= D, and |c - x|^2 >= d^2 + |x - p|^2 by the projection onto a convex
// set). On the other side the cells' current bounds u are majorised by planes, u <= a + g . delta
// and u^2 - |delta|^2 <= A + G . delta (g, G fitted, a and A the largest residuals). A child is
// dropped when either lower bound is above its plane over the whole box |delta_k| <= H_k, which is
// one sum of three absolute values each. The first is tight near the surface, the second, where the
// curvature of the distance cancels, for children small against their distance.
//
// Every test keeps a child by a margin above the rounding of both sides and of the exact test, so a
// triangle is dropped only when its computed distance cannot be the minimum: the result is the
// minimum over all triangles of the computed distance, whatever the order of the walk.
//
// Two passes keep one expensive tile from holding the whole GPU. In pass A a walk looks at the
// chunk counter every few steps; once every chunk has been handed out (the tail) it stops, stores
// its cells' bounds (squared distances, upper bounds of the answer) in the output and appends the
// tile to a deferred list. Pass B gives each deferred tile a whole block, which goes down the tree a
// level at a time: its warps take the level's surviving nodes from a shared list, test their children
// and list those that survive for the next level; at the last they measure the blocks against the
// cells, whose bounds they share in shared memory (atomicMin on the float bits, valid for
// non-negative values). A pass starts from bounds that are nearly final, so what it takes is set by
// how evenly the warps share the rest. Before, its 16 warps took the subtrees of one fixed level: bakes
// of 82k triangles at 256^3 went from 5.25 to 5.12 ms, of 1M at 128^3 from 6.90 to 6.30 ms. Handing
// over the first pass's stack instead, few nodes with uneven subtrees, made the passes 4.8 -> 5.2 ms
// and 6.3 -> 7.1 ms. 12 warps, two blocks an SM: against 16 warps and one, both passes over 97 x 61 x
// 43 cells take 201-281 us for 178-240 (8 warps and three: 178-233, but 168 for 160 us at 64^3).
//
// Sign: parity counts the column's crossing bits at and above each cell (parity.cu). Winding-number
// signs are applied afterwards by gwn.cu, which needs the unsigned distance to find the near-surface
// band.
#include <algorithm>
#include <climits>
#include <cstdint>

#include "common.cuh"
#include "kernels.h"

namespace sdfb {
namespace {

// 7 blocks an SM at 72 registers a thread: against 6 blocks at 80, 1 to 3% less time from 64^3 up.
constexpr int kThreadsA = 128;
constexpr int kMinBlocksA = 7;
constexpr int kWarpsPerBlockA = kThreadsA / kWarp;
// Tile order within a mesh: bricks of kBrickX x kBrickY x kBrickZ tiles, x fastest inside a brick
// and across bricks. Tiles of a partial brick beyond the grid have no active cell.
constexpr int kBrickX = 4, kBrickY = 4, kBrickZ = 2, kBrickTiles = kBrickX * kBrickY * kBrickZ;
constexpr int kChunkMax = 32;  // tiles per chunk when there are plenty
constexpr unsigned long long kNoTile = ~0ull;
constexpr int kDispatchSpin = 1 << 22;  // bound on a warp's wait for its block's next chunk
constexpr int kThreads = 384;
constexpr int kMinBlocksB = 2;
constexpr int kWarpsPerBlockB = kThreads / kWarp;
constexpr uint32_t kFrontier = 2048;  // pass B: nodes of a level that the block keeps
constexpr int kMaxLevels = 8;        // 2^31 triangles in blocks of 2 make 6 levels of 32-ary nodes
constexpr int kStackSize = 32 * kMaxLevels;  // a node leaves at most 31 siblings behind on its level
constexpr int kFlushAt = 16;                 // surviving blocks measured against the cells together
constexpr int kSurvivors = kFlushAt + kWarp;
// Cells of a tile of 128 from which on a block is measured by all of them rather than in pairs. Large
// triangles, pairs alone and with 64, 48 and 32 cells: a box of 12 at 256^3 0.32 ms, 0.30 each; 80 at 256^3
// 0.86, 0.68, 0.67, 0.66; 2,000 as large as their box at 128^3 2.8, 1.46, 1.46, 1.45; 82k small ones at 256^3
// 4.38, 4.14, 4.08, 4.07. Smaller tiles keep to pairs: they belong to grids that leave the GPU underfilled, where
// the pairs' shorter chain of loads counts (1,280 triangles at 32^3 59.5 us, 62.3 with 24 of 32 cells).
constexpr uint32_t kDirectCells = 48;
constexpr int kDrainAt = 64;                 // pairs that start a round of exact tests
// Steps of work as sdfb_opts.step_budget counts them, about 8 instructions each.
constexpr int kStepsPerVisit = 16, kStepsPerBlock = 10, kStepsPerRound = 12;
// A search for a seed gives up after as many nodes, and a tile takes its seed from a neighbour whose centre
// lies within this squared distance, in squared half diagonals. A bad seed costs its tile and the ones that
// take theirs from it: 400 visits instead of 48 and 20 instead of 5 took the distance stage of 82k triangles
// at 256^3 from 4.85 to 4.49 ms, of 1M at 128^3 from 5.2 to 4.7 ms and of 490k at 512^3 from 33.2 to 30.3 ms
// (no limit on the distance: 5.0, 5.4 and 31.9; a search in every tile: 4.5, 4.7 and 37.5).
constexpr int kSearchVisits = 400;
constexpr float kCloseTile = 20.0f;
constexpr uint32_t kNoSeed = ~0u;
constexpr float kInf = __builtin_huge_valf();

struct Shape {
  int tx, ty, tz;
};
constexpr Shape kShapes[] = {{4, 4, 2}, {8, 4, 1}, {4, 4, 4}, {8, 4, 2}, {4, 4, 8}, {8, 4, 4}};
constexpr int kNumShapes = sizeof(kShapes) / sizeof(kShapes[0]);

struct WalkStats {
  unsigned long long box_tests = 0, tri_tests = 0, plane_tests = 0, rect_tests = 0;
  bool overflow = false, corrupt = false;
};

// A tile's cells as one lane sees them. A cell beyond the grid stands in for the nearest cell inside
// it, so that every lane holds valid points; only active cells are written.
template <int TX, int TY, int TZ>
struct TileCells {
  static constexpr int kLayer = TX * TY;
  static constexpr int kLanesZ = kWarp / kLayer;
  static constexpr int VPL = TZ / kLanesZ;
  static_assert(kLayer * kLanesZ == kWarp && VPL * kLanesZ == TZ, "tile must cover whole warps");
  const MeshRec *M;
  GridDev g;
  int x0, y0, z0;  // the tile's first cell

  // Returns false for a tile without a cell inside the grid.
  __device__ __forceinline__ bool locate(const BatchDev &B, unsigned long long tile) {
    const int mesh = find_mesh(B.tile_starts, B.num_meshes, tile);
    M = &B.recs[mesh];
    g = M->g;
    const unsigned long long local = tile - B.tile_starts[mesh];
    const int tiles_x = (g.nx + TX - 1) / TX, tiles_y = (g.ny + TY - 1) / TY;
    const int bricks_x = (tiles_x + kBrickX - 1) / kBrickX, bricks_y = (tiles_y + kBrickY - 1) / kBrickY;
    const unsigned long long brick = local / kBrickTiles;
    const int w = static_cast<int>(local % kBrickTiles);
    const unsigned long long rest = brick / bricks_x;
    x0 = (static_cast<int>(brick % bricks_x) * kBrickX + w % kBrickX) * TX;
    y0 = (static_cast<int>(rest % bricks_y) * kBrickY + (w / kBrickX) % kBrickY) * TY;
    z0 = (static_cast<int>(rest / bricks_y) * kBrickZ + w / (kBrickX * kBrickY)) * TZ;
    return x0 < g.nx && y0 < g.ny && z0 < g.nz;
  }
  __device__ __forceinline__ int vx(int lane) const { return x0 + lane % TX; }
  __device__ __forceinline__ int vy(int lane) const { return y0 + (lane / TX) % TY; }
  __device__ __forceinline__ int vz(int lane, int v) const { return z0 + lane / kLayer + v * kLanesZ; }
  __device__ __forceinline__ float px(int lane) const { return cell_center(g.ox, min(vx(lane), g.nx - 1), g.voxel); }
  __device__ __forceinline__ float py(int lane) const { return cell_center(g.oy, min(vy(lane), g.ny - 1), g.voxel); }
  __device__ __forceinline__ float pz(int lane, int v) const {
    return cell_center(g.oz, min(vz(lane, v), g.nz - 1), g.voxel);
  }
  __device__ __forceinline__ bool active(int lane, int v) const {
    return vx(lane) < g.nx && vy(lane) < g.ny && vz(lane, v) < g.nz;
  }
  // Output index of the lane's cell v, or of the cell it stands in for.
  __device__ __forceinline__ uint64_t cell(int lane, int v) const {
    return (uint64_t(min(vz(lane, v), g.nz - 1)) * g.ny + min(vy(lane), g.ny - 1)) * g.nx + min(vx(lane), g.nx - 1);
  }
};

// When a walk may stop early: every `every` steps of work it reads the pass's tile counter, and it stops
// once every tile has been handed out (the pass is in its tail, where a long walk would run
// alone). every = 0: never.
struct TailCheck {
  const unsigned long long *counter;
  unsigned long long total;
  int every;
};

// Bounds of one walk: the most node visits (a walk visits each node at most once) and the usable stack
// entries. The fault-injection bits shrink them so that the error paths behind them can be tested.
struct WalkLimits {
  int visits, stack;
};
__device__ __forceinline__ WalkLimits walk_limits(const DistTree &t, int stack_depth, int fault) {
  WalkLimits l;
  l.visits = static_cast<int>(min(t.num_tris, 0x7ffffff0u - 64u)) + 64;
  l.stack = kStackSize;
  if (fault) {
    if (fault & kFaultStepLimit) l.visits = 0;
    if ((fault & kFaultStackAll) || (stack_depth <= 32 && (fault & kFaultShallowStack))) l.stack = 2;
  }
  return l;
}

// Shared memory of one warp's walk. What is the same for all lanes lives here rather than in
// registers (one broadcast load where it is needed): 80 instead of 120 registers a thread.
struct WarpMem {
  float4 centre;                // the tile's centre; w: rho
  float4 half;                  // half extents of the cell centres about it; w: a
  float4 lin, sq;               // (g, -) and (G, A): the planes above the bounds
  DistTree t;
  float z[8];                   // z of the tile's layers
  uint32_t level_n[kMaxLevels], level_off[kMaxLevels];  // nodes of each level, first node in t.box
  uint32_t stack[kStackSize];   // (level << 28) | node
  uint32_t blocks[kSurvivors];  // surviving blocks; blocks[0] is the nearest of its node
  uint32_t mesh;                // the mesh that t is of
  uint32_t seed;                // the block that last improved the middle cell of the tile at seed_at
  uint32_t started;             // the block that the tile's bounds were started from
  float seed_at[3];
  uint16_t pairs[kDrainAt + kWarp * 4];  // (index into blocks << 7) | (v << 5) | lane
};
static_assert(kSurvivors <= 512, "a pair packs into 16 bits");

// Exact squared distance from q to a triangle record.
__device__ __forceinline__ float tri_dist2(const float4 &q0, const float4 &q1, const float4 &q2, const float4 &q3,
                                           const float4 &q4, float qx, float qy, float qz) {
  const float ax = qx - q0.x, ay = qy - q0.y, az = qz - q0.z;
  const float h = fmaf(az, q3.z, fmaf(ay, q3.y, ax * q3.x));
  const float u = fmaf(az, q1.z, fmaf(ay, q1.y, ax * q1.x)), w = fmaf(az, q2.z, fmaf(ay, q2.y, ax * q2.x));
  return fmaf(h, h, inplane_dist2(u, w, dist_to_range(u, q0.w), q0.w, q1.w, q2.w, q3.w, q4));
}

template <int TX, int TY, int TZ, bool COUNT>
struct Walker {
  using Cells = TileCells<TX, TY, TZ>;
  static constexpr int VPL = Cells::VPL;
  static constexpr int kMiddle = (VPL / 2) * kWarp + 13;  // a cell about the middle of the tile
  // Relative margin of the cells' bounds in the oriented box test (2e-6 in the distance, several
  // times the rounding of the box distance and of the exact test; the boxes' half extents carry the
  // part that scales with the block's size).
  static constexpr float kKeep = 1.0f + 4e-6f;

  WarpMem &m;
  uint32_t *best;  // squared distance bounds (float bits) of the tile's cells: this warp's, or its block's
  int lane;
  float px, py, pz[VPL], keep[VPL];  // keep: best * kKeep
  int steps = 0;                     // work of the current walk
  WalkStats ws;

  __device__ __forceinline__ Walker(WarpMem &mem, uint32_t *b, int l) : m(mem), best(b), lane(l) {}

  __device__ __forceinline__ void set_tile(const Cells &c) {
    const GridDev &g = c.g;
    px = c.px(lane);
    py = c.py(lane);
#pragma unroll
    for (int v = 0; v < VPL; ++v) pz[v] = c.pz(lane, v);
    if (lane < TZ) m.z[lane] = cell_center(g.oz, min(c.z0 + lane, g.nz - 1), g.voxel);
    const float cx = g.ox + (float(c.x0) + 0.5f * TX) * g.voxel, cy = g.oy + (float(c.y0) + 0.5f * TY) * g.voxel,
                cz = g.oz + (float(c.z0) + 0.5f * TZ) * g.voxel;
    // Half extents of the cell centres about (cx, cy, cz), with room for both sides' rounding.
    const float hx = 0.50001f * (TX - 1) * g.voxel + 3e-7f * (fabsf(g.ox) + fabsf(cx)),
                hy = 0.50001f * (TY - 1) * g.voxel + 3e-7f * (fabsf(g.oy) + fabsf(cy)),
                hz = 0.50001f * (TZ - 1) * g.voxel + 3e-7f * (fabsf(g.oz) + fabsf(cz));
    if (lane == 0) {
      m.centre = make_float4(cx, cy, cz, sqrtf(hx * hx + hy * hy + hz * hz));
      m.half = make_float4(hx, hy, hz, kInf);
      m.lin.w = 1.0f / g.voxel;  // for fit()
    }
    __syncwarp();
  }

  // Nodes per level of the mesh's tree and where each level starts in t.box.
  __device__ __forceinline__ void set_tree(const DistTree &tree, uint32_t mesh) {
    if (lane < kMaxLevels) {
      m.level_n[lane] = tree_level_count(tree.num_tris, tree.block_log2, lane);
      uint32_t off = 0;
      for (int l = 1; l < lane; ++l) off += tree_level_count(tree.num_tris, tree.block_log2, l);
      m.level_off[lane] = off;
    }
    if (lane == 0) {
      m.t = tree;
      m.seed = m.started = kNoSeed;
      *const_cast<volatile uint32_t *>(&m.mesh) = mesh;
    }
    __syncwarp();
  }
  __device__ __forceinline__ uint32_t root() const {
    int l = 1;
    while (l < kMaxLevels - 1 && m.level_n[l] > 1) ++l;
    return static_cast<uint32_t>(l) << 28;
  }

  // Sum and maximum over the warp.
  static __device__ __forceinline__ float wsum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
  }
  static __device__ __forceinline__ float wmax(float v) {
    return ordered_to_float(__reduce_max_sync(kFull, float_to_ordered(v)));
  }

  // Reads the bounds and fits the planes above them: g and G are the least squares slopes over the
  // tile (the cells' offsets from the centre sum to about zero), taken about a middle cell's value. The
  // sums take the offsets in voxels, so that they hold nothing larger than a squared length, as the bounds
  // themselves. Where one passes FP32's range all the same its plane becomes +inf, which drops nothing.
  __device__ __forceinline__ void fit() {
    float su = 0.0f, sw = 0.0f, sz = 0.0f, swz = 0.0f, u[VPL], w[VPL];
    const float4 c = m.centre;
    const float n = m.lin.w;  // 1 / voxel
    const float dx = px - c.x, dy = py - c.y, dxy = dx * dx + dy * dy;
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      const float b = __uint_as_float(best[v * kWarp + lane]);
      const float dz = pz[v] - c.z;
      keep[v] = b * kKeep;
      u[v] = sqrtf(b);
      w[v] = b - fmaf(dz, dz, dxy);
    }
    const float u0 = __shfl_sync(kFull, u[kMiddle / kWarp], kMiddle % kWarp),
                w0 = __shfl_sync(kFull, w[kMiddle / kWarp], kMiddle % kWarp);
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      const float kz = (pz[v] - c.z) * n, du = u[v] - u0, dw = w[v] - w0;
      su += du;
      sw += dw;
      sz = fmaf(du, kz, sz);
      swz = fmaf(dw, kz, swz);
    }
    const float kx = dx * n, ky = dy * n;
    constexpr float kCells = 12.0f / (VPL * kWarp);  // over the sum of squared offsets, but for the axes' cell counts
    const float ix = n * (kCells / (TX * TX - 1)), iy = n * (kCells / (TY * TY - 1)),
                iz = TZ > 1 ? n * (kCells / (TZ > 1 ? TZ * TZ - 1 : 1)) : 0.0f;
    float gx = wsum(su * kx) * ix, gy = wsum(su * ky) * iy, gz = wsum(sz) * iz;
    float Gx = wsum(sw * kx) * ix, Gy = wsum(sw * ky) * iy, Gz = wsum(swz) * iz;
    float ra = -kInf, rA = -kInf;
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      const float dz = pz[v] - c.z;
      ra = fmaxf(ra, u[v] - (gx * dx + gy * dy + gz * dz));
      rA = fmaxf(rA, w[v] - (Gx * dx + Gy * dy + Gz * dz));
    }
    ra = wmax(ra);
    rA = wmax(rA);
    const float4 h = m.half;
    __syncwarp();
    if (lane == 0) {
      if (!(fabsf(gx) + fabsf(gy) + fabsf(gz) + fabsf(ra) < kInf)) {
        gx = gy = gz = 0.0f;
        ra = kInf;
      }
      if (!(fabsf(Gx) + fabsf(Gy) + fabsf(Gz) + fabsf(rA) < kInf)) {
        Gx = Gy = Gz = 0.0f;
        rA = kInf;
      }
      m.half.w = ra + 2e-6f * (fabsf(ra) + h.x * fabsf(gx) + h.y * fabsf(gy) + h.z * fabsf(gz));
      m.lin = make_float4(gx, gy, gz, n);
      m.sq = make_float4(Gx, Gy, Gz,
                         rA + 4e-6f * (fabsf(rA) + h.x * fabsf(Gx) + h.y * fabsf(Gy) + h.z * fabsf(Gz)));
    }
    __syncwarp();
  }

  // Whether a convex child with nearest point c - (ex, ey, ez) to the tile's centre, whose farthest
  // point from there is at sqrt(D2), may hold a triangle nearer than the bounds of some cell. S is
  // the size of the coordinates that e was formed from; a few 1e-7 of it is the error of e. A child
  // that makes a NaN (non-finite vertices, reported elsewhere, or a d2 past FP32) is dropped; a plane never
  // makes one (see fit).
  __device__ __forceinline__ bool near(float rho, float ex, float ey, float ez, float d2, float D2, float S) const {
    const float4 h = m.half, g = m.lin, G = m.sq;
    const float inv = d2 > 0.0f ? rsqrtf(d2) : 0.0f;
    const float d = d2 * inv;
    const float lin = d - h.w - (h.x * fabsf(fmaf(ex, inv, -g.x)) + h.y * fabsf(fmaf(ey, inv, -g.y)) +
                                 h.z * fabsf(fmaf(ez, inv, -g.z)));
    const float D = sqrtf(D2);
    const float K = D < rho ? D * (2.0f * rho - D) : rho * rho;
    const float sq = d2 - K - G.w - (h.x * fabsf(fmaf(2.0f, ex, -G.x)) + h.y * fabsf(fmaf(2.0f, ey, -G.y)) +
                                     h.z * fabsf(fmaf(2.0f, ez, -G.z)));
    return lin <= 2e-6f * S * fmaf(rho, inv, 1.0f) && sq <= 4e-6f * S * (d + rho);
  }

  // Exact distances of the queued pairs, n = 2^block_log2 lanes to a pair.
  __device__ __forceinline__ void drain(int &np) {
    __syncwarp();
    const int lb = m.t.block_log2, sub = lane & ((1 << lb) - 1);
    const float4 *tris = m.t.tri;
    for (int base = 0; base < np; base += kWarp >> lb) {
      const int i = base + (lane >> lb);
      const uint32_t e = m.pairs[min(i, np - 1)];
      const int cl = e & 31, v = (e >> 5) & 3;
      const uint32_t blk = m.blocks[e >> 7];
      const float4 *tri = tree_tri(tris, (size_t(blk) << lb) + sub);
      const float4 q0 = __ldg(tri), q1 = __ldg(tri + kTriPlane), q2 = __ldg(tri + 2 * kTriPlane),
                   q3 = __ldg(tri + 3 * kTriPlane), q4 = __ldg(tri + 4 * kTriPlane);
      float d2 = tri_dist2(q0, q1, q2, q3, q4, __shfl_sync(kFull, px, cl), __shfl_sync(kFull, py, cl),
                           m.z[cl / Cells::kLayer + v * Cells::kLanesZ]);
      for (int o = 1; o < (1 << lb); o <<= 1) d2 = fminf(d2, __shfl_xor_sync(kFull, d2, o));
      if (sub == 0 && i < np) {
        const uint32_t was = atomicMin(best + (e & 127), __float_as_uint(d2));
        if ((e & 127) == kMiddle && __float_as_uint(d2) < was) m.seed = blk;
      }
      if (COUNT) ws.tri_tests += min(np - base, kWarp >> lb) << lb;
    }
    __syncwarp();
#pragma unroll
    for (int v = 0; v < VPL; ++v) keep[v] = __uint_as_float(best[v * kWarp + lane]) * kKeep;
    steps += ((np << lb) >> 5) * kStepsPerRound;
    np = 0;
  }

  // Exact distances of a block's triangles to every cell, lanes = cells: for a block that most cells want.
  __device__ __forceinline__ void direct(uint32_t blk) {
    const int lb = m.t.block_log2;
    float b[VPL];
#pragma unroll
    for (int v = 0; v < VPL; ++v) b[v] = kInf;
    for (int k = 0; k < (1 << lb); ++k) {
      const float4 *tri = tree_tri(m.t.tri, (size_t(blk) << lb) + k);
      const float4 q0 = __ldg(tri), q1 = __ldg(tri + kTriPlane), q2 = __ldg(tri + 2 * kTriPlane),
                   q3 = __ldg(tri + 3 * kTriPlane), q4 = __ldg(tri + 4 * kTriPlane);
#pragma unroll
      for (int v = 0; v < VPL; ++v) b[v] = fminf(b[v], tri_dist2(q0, q1, q2, q3, q4, px, py, pz[v]));
      if (COUNT) ws.tri_tests += kWarp * VPL;
    }
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      const uint32_t was = atomicMin(best + v * kWarp + lane, __float_as_uint(b[v]));
      keep[v] = fminf(b[v], __uint_as_float(was)) * kKeep;
      if (v * kWarp + lane == kMiddle && __float_as_uint(b[v]) < was) m.seed = blk;
    }
    steps += (3 + 5 * VPL) << lb;
    __syncwarp();
  }

  // Measures the surviving blocks against every cell, runs the pairs, refits the planes (not the last time:
  // no node is left that they could drop).
  __device__ __forceinline__ void flush(int &nb, bool last) {
    int np = 0;
    bool any_pair = false;
    const float4 *obb = m.t.obb;
    for (int i = 0; i < nb; ++i) {
      const float4 *o = tree_obb(obb, m.blocks[i]);
      const float4 o0 = __ldg(o), o1 = __ldg(o + kObbPlane), o2 = __ldg(o + 2 * kObbPlane), o3 = __ldg(o + 3 * kObbPlane);
      const float dx = px - o0.x, dy = py - o0.y;
      const float s0 = fmaf(dy, o1.y, dx * o1.x), s1 = fmaf(dy, o2.y, dx * o2.x), s2 = fmaf(dy, o3.y, dx * o3.x);
      bool want[VPL], some = false;
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        const float dz = pz[v] - o0.z;
        const float e0 = fmaxf(fabsf(fmaf(dz, o1.z, s0)) - o0.w, 0.0f);
        const float e1 = fmaxf(fabsf(fmaf(dz, o2.z, s1)) - o1.w, 0.0f);
        const float e2 = fmaxf(fabsf(fmaf(dz, o3.z, s2)) - o2.w, 0.0f);
        want[v] = fmaf(e0, e0, fmaf(e1, e1, e2 * e2)) < keep[v];
        some |= want[v];
      }
      if (COUNT) ws.rect_tests += kWarp * VPL;
      if (!__any_sync(kFull, some)) continue;
      any_pair = true;
      uint32_t masks[VPL], cells = 0;
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        masks[v] = __ballot_sync(kFull, want[v]);
        cells += __popc(masks[v]);
      }
      if (VPL >= 4 && cells >= kDirectCells) {
        direct(m.blocks[i]);
        continue;
      }
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        const uint32_t mask = masks[v];
        if (want[v])
          m.pairs[np + __popc(mask & ((1u << lane) - 1u))] = static_cast<uint16_t>((i << 7) | (v << 5) | lane);
        np += __popc(mask);
      }
      if (np >= kDrainAt) drain(np);
    }
    if (np > 0) drain(np);
    __syncwarp();
    steps += nb * kStepsPerBlock;
    nb = 0;
    if (any_pair && !last) fit();
  }

  // Finds the block to start from: of the blocks nearest to the middle of the last tiles of the
  // block's warps, the one nearest to this tile's centre, if one of those tiles was close by; else a
  // search from the root. (A warp that moves to another mesh meanwhile may leave a block number of
  // that mesh behind: any block of the tree is a valid seed.)
  __device__ __forceinline__ void pick_seed(const WarpMem *mem, int warps) {
    const float4 c = m.centre;
    uint32_t s = 0;
    bool have = false;
    if (lane < warps) {
      const volatile WarpMem *o = mem + lane;
      s = o->seed;
      const float dx = o->seed_at[0] - c.x, dy = o->seed_at[1] - c.y, dz = o->seed_at[2] - c.z;
      have = o->mesh == m.mesh && s < m.level_n[0] && dx * dx + dy * dy + dz * dz < kCloseTile * c.w * c.w;
    }
    if (!__any_sync(kFull, have)) {
      search();
      return;
    }
    const float d2 = have ? obb_dist2(s) : kInf;
    const uint32_t near_key = __reduce_min_sync(kFull, have ? (__float_as_uint(d2) & ~31u) | lane : ~0u);
    s = __shfl_sync(kFull, s, near_key & 31);
    __syncwarp();
    if (lane == 0) m.seed = s;
    __syncwarp();
  }

  // Squared distance of the tile's centre to a block's oriented box.
  __device__ __forceinline__ float obb_dist2(uint32_t blk) const {
    const float4 c = m.centre;
    const float4 *o = tree_obb(m.t.obb, blk);
    const float4 o0 = __ldg(o), o1 = __ldg(o + kObbPlane), o2 = __ldg(o + 2 * kObbPlane), o3 = __ldg(o + 3 * kObbPlane);
    const float dx = c.x - o0.x, dy = c.y - o0.y, dz = c.z - o0.z;
    const float e0 = fmaxf(fabsf(fmaf(dz, o1.z, fmaf(dy, o1.y, dx * o1.x))) - o0.w, 0.0f);
    const float e1 = fmaxf(fabsf(fmaf(dz, o2.z, fmaf(dy, o2.y, dx * o2.x))) - o1.w, 0.0f);
    const float e2 = fmaxf(fabsf(fmaf(dz, o3.z, fmaf(dy, o3.y, dx * o3.x))) - o2.w, 0.0f);
    return e0 * e0 + e1 * e1 + e2 * e2;
  }

  // Nearest block to the tile's centre, or near enough to it: a depth-first search, nearest child
  // first, that gives up after kSearchVisits nodes.
  __device__ __forceinline__ void search() {
    const float4 c = m.centre;
    const int lb = m.t.block_log2, sub = lane & ((1 << lb) - 1);
    uint32_t cur = root(), seed = 0, bound = ~0u;  // bound: float bits of the squared distance found
    int sp = 0;
    for (int visits = 0; visits < kSearchVisits; ++visits) {
      const int level = static_cast<int>(cur >> 28) - 1;
      const uint32_t first = (cur & 0x0fffffffu) * 32, child = first + lane;
      const bool valid = child < m.level_n[level];
      float d2 = kInf;
      if (valid) {
        if (level == 0) {
          d2 = obb_dist2(child);
        } else {
          const float4 *b = m.t.box + 2 * size_t(m.level_off[level] + child);
          const float4 bc = __ldg(b), be = __ldg(b + 1);
          d2 = box_dist2(c.x, c.y, c.z, bc.x, bc.y, bc.z, be.x, be.y, be.z);
        }
      }
      const bool kept = valid && __float_as_uint(d2) < bound;
      const uint32_t mask = __ballot_sync(kFull, kept);
      if (mask) {
        const int nl = __reduce_min_sync(kFull, kept ? (__float_as_uint(d2) & ~31u) | lane : ~0u) & 31;
        const int cnt = __popc(mask), rank = __popc(mask & ((1u << lane) - 1u)) - (lane > nl ? 1 : 0);
        if (level > 0) {
          if (kept && lane != nl && sp + rank < kStackSize) m.stack[sp + rank] = static_cast<uint32_t>(level) << 28 | child;
          sp = min(sp + cnt - 1, kStackSize);
          cur = static_cast<uint32_t>(level) << 28 | (first + nl);
          __syncwarp();
          continue;
        }
        if (kept) m.blocks[lane == nl ? 0 : rank + 1] = child;
        __syncwarp();
        for (int base = 0; base < cnt; base += kWarp >> lb) {
          const uint32_t blk = m.blocks[min(base + (lane >> lb), cnt - 1)];
          const float4 *tri = tree_tri(m.t.tri, (size_t(blk) << lb) + sub);
          const float e = tri_dist2(__ldg(tri), __ldg(tri + kTriPlane), __ldg(tri + 2 * kTriPlane),
                                    __ldg(tri + 3 * kTriPlane), __ldg(tri + 4 * kTriPlane), c.x, c.y, c.z);
          const uint32_t key = __reduce_min_sync(kFull, (__float_as_uint(fminf(e, 1e38f)) & ~31u) | lane);
          if ((key | 31u) < bound) {
            bound = key | 31u;
            seed = __shfl_sync(kFull, blk, key & 31);
          }
        }
        __syncwarp();
      }
      if (sp == 0) break;
      cur = m.stack[--sp];
    }
    __syncwarp();
    if (lane == 0) m.seed = seed;
    __syncwarp();
  }

  // Starts the bounds from the triangles of the seed block (from the first alone: 1% slower).
  __device__ __forceinline__ void start() {
    float b[VPL];
#pragma unroll
    for (int v = 0; v < VPL; ++v) b[v] = kInf;
    const int lb = m.t.block_log2;
    for (int k = 0; k < (1 << lb); ++k) {
      const float4 *tri = tree_tri(m.t.tri, (size_t(m.seed) << lb) + k);
      const float4 q0 = __ldg(tri), q1 = __ldg(tri + kTriPlane), q2 = __ldg(tri + 2 * kTriPlane),
                   q3 = __ldg(tri + 3 * kTriPlane), q4 = __ldg(tri + 4 * kTriPlane);
#pragma unroll
      for (int v = 0; v < VPL; ++v) b[v] = fminf(b[v], tri_dist2(q0, q1, q2, q3, q4, px, py, pz[v]));
      if (COUNT) ws.tri_tests += kWarp * VPL;
    }
#pragma unroll
    for (int v = 0; v < VPL; ++v) best[v * kWarp + lane] = __float_as_uint(b[v]);
    if (lane < 3) m.seed_at[lane] = lane == 0 ? m.centre.x : (lane == 1 ? m.centre.y : m.centre.z);
    if (lane == 3) m.started = m.seed;
    __syncwarp();
  }

  // Whether the lane's child on `level` may matter, and its squared distance to the tile's centre.
  __device__ __forceinline__ bool test(int level, uint32_t child, float &d2) {
    const bool valid = child < m.level_n[level];
    bool kept;
    const float4 c = m.centre;
    if (level > 0) {
      const float4 *b = m.t.box + 2 * size_t(m.level_off[level] + (valid ? child : 0));
      const float4 bc = __ldg(b), be = __ldg(b + 1);
      const float tx = c.x - bc.x, ty = c.y - bc.y, tz = c.z - bc.z;
      const float ax = fabsf(tx), ay = fabsf(ty), az = fabsf(tz);
      const float ex = fmaxf(ax - be.x, 0.0f), ey = fmaxf(ay - be.y, 0.0f), ez = fmaxf(az - be.z, 0.0f);
      const float fx = fminf(ax, be.x) + be.x, fy = fminf(ay, be.y) + be.y, fz = fminf(az, be.z) + be.z;
      d2 = ex * ex + ey * ey + ez * ez;
      kept = near(c.w, copysignf(ex, tx), copysignf(ey, ty), copysignf(ez, tz), d2, fx * fx + fy * fy + fz * fz,
                  ax + ay + az + be.x + be.y + be.z);
      if (COUNT) ws.box_tests += __popc(__ballot_sync(kFull, valid));
    } else {
      const float4 *o = tree_obb(m.t.obb, valid ? child : 0);
      const float4 o0 = __ldg(o), o1 = __ldg(o + kObbPlane), o2 = __ldg(o + 2 * kObbPlane),
                   o3 = __ldg(o + 3 * kObbPlane);
      const float dx = c.x - o0.x, dy = c.y - o0.y, dz = c.z - o0.z;
      const float t0 = fmaf(dz, o1.z, fmaf(dy, o1.y, dx * o1.x)), t1 = fmaf(dz, o2.z, fmaf(dy, o2.y, dx * o2.x)),
                  t2 = fmaf(dz, o3.z, fmaf(dy, o3.y, dx * o3.x));
      const float a0 = fabsf(t0), a1 = fabsf(t1), a2 = fabsf(t2);
      const float e0 = copysignf(fmaxf(a0 - o0.w, 0.0f), t0), e1 = copysignf(fmaxf(a1 - o1.w, 0.0f), t1),
                  e2 = copysignf(fmaxf(a2 - o2.w, 0.0f), t2);
      const float f0 = fminf(a0, o0.w) + o0.w, f1 = fminf(a1, o1.w) + o1.w, f2 = fminf(a2, o2.w) + o2.w;
      d2 = e0 * e0 + e1 * e1 + e2 * e2;
      kept = near(c.w, fmaf(e2, o3.x, fmaf(e1, o2.x, e0 * o1.x)), fmaf(e2, o3.y, fmaf(e1, o2.y, e0 * o1.y)),
                  fmaf(e2, o3.z, fmaf(e1, o2.z, e0 * o1.z)), d2, f0 * f0 + f1 * f1 + f2 * f2,
                  a0 + a1 + a2 + o0.w + o1.w + o2.w);
      if (COUNT) ws.plane_tests += __popc(__ballot_sync(kFull, valid));
    }
    return kept && valid && (level > 0 || child != m.started);
  }

  // Takes the kept blocks into the list, the nearest first.
  __device__ __forceinline__ void take_blocks(bool kept, uint32_t child, uint32_t mask, float d2, int &nb) {
    const int nl = __reduce_min_sync(kFull, kept ? (__float_as_uint(d2) & ~31u) | lane : ~0u) & 31;
    const int rank = __popc(mask & ((1u << lane) - 1u)) - (lane > nl ? 1 : 0);
    if (kept) m.blocks[nb + (lane == nl ? 0 : rank + 1)] = child;
    nb += __popc(mask);
    __syncwarp();
  }

  // Walks below node `cur` ((level << 28) | node). Returns false when the tail check stopped it with
  // work left (the bounds are then upper bounds); a walk past its step limit raises the corrupt flag.
  __device__ __forceinline__ bool walk(uint32_t cur, TailCheck tail, WalkLimits lim) {
    int sp = 0, nb = 0;
    int next_check = tail.every > 0 ? tail.every : INT_MAX;
    steps = 0;
    for (int visits = 0;; ++visits, steps += kStepsPerVisit) {
      if (visits > lim.visits) {
        ws.corrupt = true;
        return true;
      }
      if (steps >= next_check) {
        unsigned long long handed = 0;
        if (lane == 0) handed = *reinterpret_cast<const volatile unsigned long long *>(tail.counter);
        handed = __shfl_sync(kFull, handed, 0);
        if (handed >= tail.total) return false;
        next_check = steps + tail.every;
      }
      const int level = static_cast<int>(cur >> 28) - 1;  // the children's level
      const uint32_t child = (cur & 0x0fffffffu) * 32 + lane;
      float d2;
      const bool kept = test(level, child, d2);
      const uint32_t mask = __ballot_sync(kFull, kept);
      if (mask) {
        if (level > 0) {  // the nearest child is walked next
          const int nl = __reduce_min_sync(kFull, kept ? (__float_as_uint(d2) & ~31u) | lane : ~0u) & 31;
          const int cnt = __popc(mask);
          const int rank = __popc(mask & ((1u << lane) - 1u)) - (lane > nl ? 1 : 0);  // among the others
          if (kept && lane != nl && sp + rank < lim.stack)
            m.stack[sp + rank] = (static_cast<uint32_t>(level) << 28) | child;
          sp += cnt - 1;
          if (sp > lim.stack) {
            ws.overflow = true;
            sp = lim.stack;
          }
          cur = (static_cast<uint32_t>(level) << 28) | ((cur & 0x0fffffffu) * 32 + nl);
          __syncwarp();
          continue;
        }
        take_blocks(kept, child, mask, d2, nb);
      }
      const bool last = sp == 0;
      if (nb >= kFlushAt || (last && nb > 0)) flush(nb, last);
      if (last) return true;
      cur = m.stack[--sp];
    }
  }
};

// Signs (parity) and writes a tile's distances.
template <int TX, int TY, int TZ>
__device__ __forceinline__ void store_cells(const DistanceArgs &a, const TileCells<TX, TY, TZ> &c, int lane,
                                            const uint32_t *best) {
  constexpr int VPL = TileCells<TX, TY, TZ>::VPL;
  const MeshRec &M = *c.M;
  // A cell is inside when an odd number of its column's bits lie at or above its layer. The tile's
  // layers share a word (their first is a multiple of their number, which divides 32).
  static_assert(32 % TZ == 0, "a tile's layers lie in one word");
  uint32_t word = 0, above = 0;
  const int vx = c.vx(lane), vy = c.vy(lane);
  const bool parity = M.sign == kSignParity && vx < c.g.nx && vy < c.g.ny;
  if (parity) {
    const int words = (c.g.nz + 31) / 32;
    const uint32_t *col = a.bits + M.bit_base + (uint64_t(vy) * c.g.nx + vx) * words;
    word = __ldg(col + c.z0 / 32);
    for (int k = c.z0 / 32 + 1; k < words; ++k) above ^= __ldg(col + k);
  }
#pragma unroll
  for (int v = 0; v < VPL; ++v) {
    if (!c.active(lane, v)) continue;
    const float d = sqrtf(__uint_as_float(best[v * kWarp + lane]));
    const bool inside = (__popc(word >> (c.vz(lane, v) & 31)) + __popc(above)) & 1;
    M.dist[c.cell(lane, v)] = inside ? -d : d;
  }
}

template <bool COUNT>
__device__ __forceinline__ void flush_stats(const DistanceArgs &a, const WalkStats &ws, int lane) {
  if (ws.overflow) atomic_or_err(a.err, kErrStackOverflow);
  if (ws.corrupt) atomic_or_err(a.err, kErrCorruptTree);
  if (COUNT && a.work_counters && lane == 0) {
    atomicAdd(a.work_counters, ws.box_tests);
    atomicAdd(a.work_counters + 1, ws.tri_tests);
    atomicAdd(a.work_counters + 3, ws.plane_tests);
    atomicAdd(a.work_counters + 4, ws.rect_tests);
  }
}

// Hands lane 0 of a warp its next tile. *state packs the block's current chunk (high 32 bits)
// and the next index within it (low 32 bits); chunks come from the global counter. The warp that
// draws index == per_chunk moves the block to a new chunk; warps drawing past it wait for that
// (bounded: past the limit the dispatch error is raised and the warp stops). Returns kNoTile when
// every chunk has been handed out.
__device__ unsigned long long next_tile(unsigned long long *state, unsigned long long *chunks,
                                        unsigned long long per_chunk, unsigned long long total_chunks,
                                        unsigned long long total_tiles, uint32_t *err, int fault) {
  // Fault injection: nobody moves the block on, and the waits are short.
  const bool stuck = fault & kFaultDispatch;
  const int spin_limit = stuck ? (1 << 12) : kDispatchSpin;
  for (;;) {
    const unsigned long long old = atomicAdd(state, 1ull);
    const unsigned long long chunk = old >> 32, idx = old & 0xffffffffull;
    if (chunk >= total_chunks) return kNoTile;
    if (idx < per_chunk) {
      const unsigned long long t = chunk * per_chunk + idx;
      if (t < total_tiles) return t;
      continue;  // past the end of the last chunk: draw on until the block moves on
    }
    if (idx == per_chunk && !stuck) {
      atomicExch(state, atomicAdd(chunks, 1ull) << 32);
      continue;
    }
    const volatile unsigned long long *vs = state;
    int spin = 0;
    while ((*vs >> 32) == chunk && spin < spin_limit) ++spin;
    if (spin == spin_limit) {
      atomic_or_err(err, kErrDispatch);
      return kNoTile;
    }
  }
}

// Pass A: warps take tiles from their block's chunk, blocks take chunks from a global counter; a
// tile still walking in the pass's tail (every chunk handed out) is deferred to pass B.
template <int TX, int TY, int TZ, bool COUNT>
__global__ __launch_bounds__(kThreadsA, kMinBlocksA) void k_distance(DistanceArgs a) {
  using W = Walker<TX, TY, TZ, COUNT>;
  constexpr int VPL = W::VPL;
  __shared__ unsigned long long s_state;
  __shared__ WarpMem s_mem[kWarpsPerBlockA];
  __shared__ uint32_t s_best[kWarpsPerBlockA][VPL * kWarp];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const BatchDev &B = a.batch;
  const unsigned long long total_chunks = (B.total_tiles + a.chunk_tiles - 1) / a.chunk_tiles;
  TailCheck tail{a.tile_counter, total_chunks,
                 (a.defer_list && a.step_budget > 0)
                     ? static_cast<int>(min(a.step_budget, 1ll << 30))
                     : 0};
  const TailCheck never{nullptr, 0, 0};
  W w(s_mem[warp], s_best[warp], lane);
  uint32_t mesh = ~0u;
  if (lane == 0) w.m.mesh = ~0u;
  if (threadIdx.x == 0) s_state = atomicAdd(a.tile_counter, 1ull) << 32;
  __syncthreads();

  for (;;) {
    unsigned long long tile = 0;
    if (lane == 0)
      tile = next_tile(&s_state, a.tile_counter, a.chunk_tiles, total_chunks, B.total_tiles, a.err, a.fault);
    tile = __shfl_sync(kFull, tile, 0);
    if (tile == kNoTile) break;
    WalkLimits lim;
    {
      typename W::Cells c;
      if (!c.locate(B, tile)) continue;
      const uint32_t index = static_cast<uint32_t>(c.M - B.recs);
      const bool first = index != mesh;
      if (first) {
        mesh = index;
        w.set_tree(c.M->tree, mesh);
      }
      lim = walk_limits(c.M->tree, a.stack_depth, a.fault);
      w.set_tile(c);
      w.pick_seed(s_mem, kWarpsPerBlockA);
    }
    w.start();
    bool listed = false;
    for (TailCheck check = tail;; check = never) {
      w.fit();
      if (w.walk(w.root(), check, lim)) break;
      unsigned long long slot = 0;
      if (lane == 0) slot = atomicAdd(a.defer_counters, 1ull);
      slot = __shfl_sync(kFull, slot, 0);
      if (slot < a.defer_capacity) {
        if (lane == 0) a.defer_list[slot] = tile;
        listed = true;
        break;
      }
      // The list is full: the tile is finished here, from the bounds found so far.
    }
    // The tile's indices are located again rather than kept in registers across the walk.
    typename W::Cells c;
    c.locate(B, tile);
    __syncwarp();
    if (listed) {
#pragma unroll
      for (int v = 0; v < VPL; ++v)
        if (c.active(lane, v))
          c.M->dist[c.cell(lane, v)] = __uint_as_float(w.best[v * kWarp + lane]);  // pass B starts from these
    } else {
      store_cells<TX, TY, TZ>(a, c, lane, w.best);
    }
    __syncwarp();
  }
  flush_stats<COUNT>(a, w.ws, lane);
}

// Pass B: one block per deferred tile; its warps share the tile's subtrees and bounds.
template <int TX, int TY, int TZ, bool COUNT>
__global__ __launch_bounds__(kThreads, kMinBlocksB) void k_distance_deferred(DistanceArgs a) {
  using W = Walker<TX, TY, TZ, COUNT>;
  constexpr int VPL = W::VPL;
  __shared__ unsigned long long s_tile;
  __shared__ uint32_t s_item, s_count[2], s_nodes[2][kFrontier];
  __shared__ WarpMem s_mem[kWarpsPerBlockB];
  __shared__ uint32_t s_best[VPL * kWarp];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const BatchDev &B = a.batch;
  const unsigned long long count = a.defer_counters[0];
  const unsigned long long total = count < a.defer_capacity ? count : a.defer_capacity;
  W w(s_mem[warp], s_best, lane);
  uint32_t mesh = ~0u;

  for (;;) {
    if (threadIdx.x == 0) {
      const unsigned long long k = atomicAdd(a.defer_counters + 1, 1ull);
      s_tile = k < total ? a.defer_list[k] : ~0ull;
      s_item = 0;
      s_nodes[0][0] = 0;  // the root
      s_count[0] = 1;
      s_count[1] = 0;
    }
    __syncthreads();
    const unsigned long long tile = s_tile;
    if (tile == ~0ull) break;
    typename W::Cells c;
    c.locate(B, tile);
    if (static_cast<uint32_t>(c.M - B.recs) != mesh) {
      mesh = static_cast<uint32_t>(c.M - B.recs);
      w.set_tree(c.M->tree, mesh);
    }
    w.set_tile(c);
    if (warp == 0) {
#pragma unroll
      for (int v = 0; v < VPL; ++v) s_best[v * kWarp + lane] = __float_as_uint(c.M->dist[c.cell(lane, v)]);
    }
    __syncthreads();
    const WalkLimits lim = walk_limits(c.M->tree, a.stack_depth, a.fault);
    w.fit();
    const uint32_t root = w.root();
    int cur = 0, nb = 0;
    for (int level = static_cast<int>(root >> 28); level > 0; --level, cur ^= 1) {
      const uint32_t items = min(s_count[cur], kFrontier);
      for (;;) {
        uint32_t item = 0;
        if (lane == 0) item = atomicAdd(&s_item, 1u);
        item = __shfl_sync(kFull, item, 0);
        if (item >= items) break;
        const uint32_t child = s_nodes[cur][item] * 32 + lane;
        float d2;
        const bool kept = w.test(level - 1, child, d2);
        const uint32_t mask = __ballot_sync(kFull, kept);
        if (!mask) continue;
        if (level == 1) {
          w.take_blocks(kept, child, mask, d2, nb);
          if (nb >= kFlushAt) w.flush(nb, false);
          continue;
        }
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(&s_count[cur ^ 1], static_cast<uint32_t>(__popc(mask)));
        at = __shfl_sync(kFull, at, 0) + __popc(mask & ((1u << lane) - 1u));
        if (kept && at < kFrontier) s_nodes[cur ^ 1][at] = child;
        // No room: the subtree is walked here.
        for (uint32_t over = __ballot_sync(kFull, kept && at >= kFrontier); over; over &= over - 1)
          w.walk((static_cast<uint32_t>(level - 1) << 28) | __shfl_sync(kFull, child, __ffs(over) - 1),
                 TailCheck{nullptr, 0, 0}, lim);
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        s_item = 0;
        s_count[cur] = 0;
      }
      __syncthreads();
    }
    if (nb > 0) w.flush(nb, true);
    __syncthreads();
    if (warp == 0) store_cells<TX, TY, TZ>(a, c, lane, s_best);
    __syncthreads();
  }
  flush_stats<COUNT>(a, w.ws, lane);
}

template <typename K>
int blocks_per_sm(K kernel, int threads) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0);
  return per_sm > 0 ? per_sm : 1;
}

template <int I, bool COUNT>
cudaError_t launch_shape(const DistanceArgs &a, int num_sms, cudaStream_t st) {
  constexpr Shape s = kShapes[I];
  static const int per_sm = blocks_per_sm(k_distance<s.tx, s.ty, s.tz, COUNT>, kThreadsA);
  static const int per_sm_b = blocks_per_sm(k_distance_deferred<s.tx, s.ty, s.tz, COUNT>, kThreads);
  const unsigned long long warps_needed = a.batch.total_tiles;
  unsigned long long blocks = static_cast<unsigned long long>(num_sms) * per_sm;
  blocks = std::min<unsigned long long>(blocks, (warps_needed + kWarpsPerBlockA - 1) / kWarpsPerBlockA);
  if (blocks < 1) blocks = 1;
  // kChunkMax tiles per chunk when there are plenty, fewer when the tiles would not reach every
  // warp several times over.
  DistanceArgs ca = a;
  ca.chunk_tiles = std::max<unsigned long long>(
      1, std::min<unsigned long long>(kChunkMax, a.batch.total_tiles / (blocks * kWarpsPerBlockA * 4)));
  k_distance<s.tx, s.ty, s.tz, COUNT><<<static_cast<unsigned>(blocks), kThreadsA, 0, st>>>(ca);
  note_launch();
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || !a.defer_list || a.step_budget <= 0) return e;
  // Pass B: a persistent grid; the number of deferred tiles is read on the device.
  const unsigned long long blocks_b =
      std::min<unsigned long long>(static_cast<unsigned long long>(num_sms) * per_sm_b, a.defer_capacity);
  k_distance_deferred<s.tx, s.ty, s.tz, COUNT>
      <<<static_cast<unsigned>(std::max<unsigned long long>(blocks_b, 1)), kThreads, 0, st>>>(a);
  note_launch();
  return cudaGetLastError();
}

template <bool COUNT>
cudaError_t launch_any(const DistanceArgs &a, int id, int num_sms, cudaStream_t st) {
  switch (id) {
    case 0: return launch_shape<0, COUNT>(a, num_sms, st);
    case 1: return launch_shape<1, COUNT>(a, num_sms, st);
    case 2: return launch_shape<2, COUNT>(a, num_sms, st);
    case 3: return launch_shape<3, COUNT>(a, num_sms, st);
    case 4: return launch_shape<4, COUNT>(a, num_sms, st);
    default: return launch_shape<5, COUNT>(a, num_sms, st);
  }
}

}  // namespace

int tile_shape_count() { return kNumShapes; }

double distance_work_flops(int tile_id, const unsigned long long *w) {
  int tx, ty, tz;
  tile_shape(tile_id, tx, ty, tz);
  const int vpl = tz / (kWarp / (tx * ty));
  return distance_flops(vpl, double(w[0]), double(w[3]), double(w[4]), double(w[1]));
}

void tile_shape(int id, int &tx, int &ty, int &tz) {
  const Shape s = kShapes[(id < 0 || id >= kNumShapes) ? 0 : id];
  tx = s.tx;
  ty = s.ty;
  tz = s.tz;
}

uint64_t tiles_for(const GridDev &g, int id) {
  int tx, ty, tz;
  tile_shape(id, tx, ty, tz);
  const uint64_t bx = ((g.nx + tx - 1) / tx + kBrickX - 1) / kBrickX;
  const uint64_t by = ((g.ny + ty - 1) / ty + kBrickY - 1) / kBrickY;
  const uint64_t bz = ((g.nz + tz - 1) / tz + kBrickZ - 1) / kBrickZ;
  return bx * by * bz * kBrickTiles;
}

uint64_t defer_capacity_for(uint64_t total_tiles) {
  return std::min<uint64_t>(total_tiles, std::max<uint64_t>(4096, total_tiles / 8));
}

cudaError_t distance_launch(const DistanceArgs &a, int tile_id, int num_sms, cudaStream_t st) {
  if (a.batch.total_tiles == 0) return cudaSuccess;
  if (a.work_counters) return launch_any<true>(a, tile_id, num_sms, st);
  return launch_any<false>(a, tile_id, num_sms, st);
}

}  // namespace sdfb
