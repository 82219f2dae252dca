// Host-side launch interface of the bake kernels. Every launcher enqueues work on the given
// stream and returns the launch error (cudaSuccess when it was enqueued).
//
// All stages work on a batch of meshes at once: triangles, cells, columns and tiles of the meshes
// are numbered consecutively ("global" indices), each kernel finds the mesh of a global index by
// binary search over a prefix table, and a single mesh is simply a batch of one.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace sdfb {

struct TriRec;
struct Node;

// Count of kernel launches issued by this library (every launcher calls note_launch once per
// <<<...>>>); the bake reports the launches of one call in sdfb_stats.
void note_launch();
uint64_t launch_count();

// Device scratch for the device-wide primitives.
struct Scratch {
  void *ptr = nullptr;
  size_t bytes = 0;
};

// ---- primitives.cu ----------------------------------------------------------------------------
// Exclusive scan of n uint32 counts into uint64 starts; out[n] receives the total, so `out` must
// hold n + 1 values. Scratch need: scan_scratch_bytes(n).
size_t scan_scratch_bytes(size_t n);
cudaError_t exclusive_scan_u32(const uint32_t *in, uint64_t *out, size_t n, Scratch s, cudaStream_t st);

// Stable LSD radix sort of (key, value) pairs on bits [0, bits) of the keys; higher bits are zero.
// keys/vals hold the input and receive the result; keys_alt/vals_alt are same-size temporaries.
size_t sort_scratch_bytes(size_t n);
cudaError_t radix_sort_pairs(uint64_t *keys, uint32_t *vals, uint64_t *keys_alt, uint32_t *vals_alt, size_t n,
                             int bits, Scratch s, cudaStream_t st);

// ---- the batch ---------------------------------------------------------------------------------
struct GridDev {
  float ox, oy, oz, voxel;
  int nx, ny, nz;
};

// One mesh's packed tree as the distance walk reads it (ptree.cu).
struct DistTree {
  const float4 *tri;    // DistTri records: groups of kTriPlane triangles, five planes of float4s each
  const float4 *obb;    // oriented boxes of the blocks: groups of kObbPlane boxes, four planes each
  const float4 *box;    // boxes of the nodes above (centre, half extent), level 1 first
  uint32_t num_tris;
  int block_log2;       // a block is 2^block_log2 triangles
};

// First plane of a triangle record or of a block's box; plane p is p * kTriPlane (kObbPlane) float4s
// on, so consecutive records coalesce and one address serves all planes.
constexpr int kTriPlane = 8, kObbPlane = 32;
template <typename F4> __host__ __device__ __forceinline__ F4 *tree_tri(F4 *tri, size_t k) {
  return tri + (k / kTriPlane) * (5 * kTriPlane) + k % kTriPlane;
}
template <typename F4> __host__ __device__ __forceinline__ F4 *tree_obb(F4 *obb, size_t b) {
  return obb + (b / kObbPlane) * (4 * kObbPlane) + b % kObbPlane;
}

constexpr int kTreePad = 256;   // triangle slots of a mesh are padded to this
constexpr int kTreeSizes = 3;   // block sizes that can be built: 2, 4, 8 (index k: 2 << k)

// Nodes of a level of a packed tree: level 0 are the blocks.
__host__ __device__ __forceinline__ uint32_t tree_level_count(uint32_t tris, int block_log2, int level) {
  uint64_t n = (uint64_t(tris) + (1u << block_log2) - 1) >> block_log2;
  for (int l = 0; l < level; ++l) n = (n + 31) >> 5;
  return static_cast<uint32_t>(n);
}

// One mesh's packed tree as the build writes it: obb[k] / box[k] are null for block sizes not built.
struct PTreeRec {
  float4 *tri;
  float4 *obb[kTreeSizes], *box[kTreeSizes];
  uint32_t slots, num_tris;  // triangle slots: num_tris padded to kTreePad
};

enum SignKind : int { kSignNone = 0, kSignParity = 1, kSignGwn = 2 };

// Device-side record of one mesh of a batch.
struct MeshRec {
  const float *verts;     // V x 3, original positions (occupancy, parity and FP64 winding read these)
  const uint32_t *idx;    // T x 3, local vertex indices
  const float *pverts;    // the mesh whose crossings decide parity (== verts unless a welded copy)
  const uint32_t *pidx;
  float *dist;            // cell outputs (either may be null)
  uint8_t *occ;
  uint32_t num_verts, num_tris, pnum_verts, pnum_tris;
  uint64_t tri_base;      // first global triangle = first sorted position of this mesh
  uint64_t cell_base;     // first global cell
  uint64_t col_base;      // first global column (winding-number meshes only)
  uint64_t bit_base;      // first word of the crossing bits (parity meshes only)
  GridDev g;
  int sign;               // SignKind
  int leaf_size;          // 1..16
  int cap_root;           // GWN: virtual root of this mesh's caps in the caps hierarchy, -1 if none
  const float *cverts;    // GWN: vertices of the caps (the parity mesh's vertices + loop centres)
  const uint32_t *cidx;   // GWN: cap triangles
  uint32_t cap_tris;      // GWN: number of cap triangles
  DistTree tree;          // the mesh's packed tree
  // GWN: the hierarchy holding this mesh's caps
  int cap_nodes_n, cap_inner_n, cap_recs_n;
  const Node *cap_nodes;
  const TriRec *cap_trec;
  const float4 *cap_moment;  // per inner cap node: (area-weighted normal sum, total area)
};

// Prefix tables of a batch (device): starts[m] of each numbering, starts[M] = total.
struct BatchDev {
  int num_meshes = 0;
  const MeshRec *recs = nullptr;
  const uint64_t *tri_starts = nullptr;       // triangles (BVH, occupancy)
  const uint64_t *ptri_starts = nullptr;      // triangles of the parity meshes
  const uint64_t *tile_starts = nullptr;      // distance tiles
  const uint64_t *gwn_tile_starts = nullptr;  // winding-number tiles (only GWN meshes have any)
  const uint64_t *cell_starts = nullptr;      // cells
  uint64_t total_tris = 0, total_ptris = 0, total_cells = 0, total_cols = 0, total_tiles = 0, total_gwn_tiles = 0,
           total_bit_words = 0;
};

// Largest m in [0, n) with starts[m] <= x (starts[0] = 0).
__host__ __device__ __forceinline__ int find_mesh(const uint64_t *starts, int n, uint64_t x) {
  int lo = 0, hi = n;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (starts[mid] <= x) lo = mid;
    else hi = mid;
  }
  return lo;
}

// ---- ptree.cu ---------------------------------------------------------------------------------
// The distance hierarchies of a batch: one packed tree per mesh, each in its own region of memory.
size_t ptree_temp_bytes(uint64_t total_tris, int num_meshes);
// Bytes of one mesh's tree with the block sizes of `mask` (bit k: 2 << k triangles); fills `out` with
// its arrays when the region's base address is given.
size_t ptree_layout(uint32_t tris, int mask, char *base, PTreeRec *out);
// trees and group_starts (one entry per mesh and the total; a group is kTreePad slots) are device
// tables beside the batch's.
cudaError_t ptree_build(const BatchDev &batch, const PTreeRec *trees, const uint64_t *group_starts, uint64_t groups,
                        void *temp, size_t temp_bytes, uint32_t *err, cudaStream_t st);

// ---- lbvh.cu ----------------------------------------------------------------------------------
// The winding number's hierarchy over the caps of a batch: every mesh's cap triangles, sorted by
// (mesh, Morton code), under one binary radix tree; each mesh's subtree is entered through its
// virtual root node, stored after the inner nodes.
struct BvhDev {
  TriRec *tris = nullptr;          // T_total records in leaf order
  Node *nodes = nullptr;           // (T_total - 1) inner nodes + M virtual roots
  uint32_t *bounds = nullptr;      // 6 ordered-uint words per mesh: centroid min xyz, max xyz
  float4 *node_moment = nullptr;   // per inner node: (sum of area x unit normal over its triangles,
                                   // their total area)
  int num_inner = 0;               // max(T_total - 1, 0)
  int num_nodes = 0;               // num_inner + M
};

size_t lbvh_temp_bytes(uint64_t total_tris, int num_meshes);
size_t lbvh_bytes(uint64_t total_tris, int num_meshes);
void lbvh_bind(BvhDev &b, void *mem, uint64_t total_tris, int num_meshes);
cudaError_t lbvh_build(const BatchDev &batch, BvhDev &b, void *temp, size_t temp_bytes, uint32_t *err,
                       cudaStream_t st);

// ---- occupancy.cu -----------------------------------------------------------------------------
size_t occupancy_temp_bytes(uint64_t total_tris);
// Clears and fills every mesh's occ grid (meshes with occ == null are skipped). first_tri
// (optional, for a batch of one) receives per cell the smallest triangle index that hits it; err
// (optional) bad indices and non-finite vertices.
cudaError_t occupancy_batch(const BatchDev &batch, uint32_t *first_tri, void *temp, size_t temp_bytes,
                            unsigned long long *sat_tests, uint32_t *err, int num_sms, cudaStream_t st);

// ---- parity.cu --------------------------------------------------------------------------------
// Crossings of the columns' +z lines with the meshes' pverts / pidx. Parity meshes: bits, per column
// ceil(nz / 32) words (total_bit_words in all), toggled at the highest layer below each crossing.
// Winding-number meshes: lists, col_start[total_cols + 1] (uint64 starts), col_z[capacity] heights,
// col_s[capacity] orientations. counters: the number of all crossings, then three of the pass itself;
// all zero before.
size_t parity_temp_bytes(uint64_t total_ptris, uint64_t total_cols);
cudaError_t parity_columns(const BatchDev &batch, uint32_t *bits, uint64_t *col_start, float *col_z, int8_t *col_s,
                           uint64_t capacity, void *temp, size_t temp_bytes, unsigned long long *counters,
                           uint32_t *err, int num_sms, cudaStream_t st);

// ---- distance.cu ------------------------------------------------------------------------------
struct DistanceArgs {
  BatchDev batch;             // each mesh record names its hierarchy and root
  const uint32_t *bits;       // parity: crossing bits
  uint32_t *err;
  unsigned long long *tile_counter;   // pass A's chunk counter, zero before the launch
  unsigned long long chunk_tiles;     // tiles per chunk (set by the launcher)
  unsigned long long *work_counters;  // optional: [0] box, [1] triangle, [3] plane, [4] rectangle tests (lanes)
  // Deferral of long tiles (none when defer_list is null or step_budget <= 0): every step_budget steps
  // (sdfb_opts) a walk checks whether all tiles have been handed out and, if so, defers its
  // tile. The list holds defer_capacity tile indices; defer_counters[0] counts deferred tiles (it
  // may pass the capacity), [1] is the second pass's tile counter. Both are zero before the launch.
  unsigned long long *defer_list;
  unsigned long long defer_capacity;
  unsigned long long *defer_counters;
  long long step_budget;
  int stack_depth;  // sdfb_opts.stack_depth as used: only fault injection looks at it
  int fault;  // sdfb_opts.fault_inject bits (testing only; 0 in normal use)
};

int tile_shape_count();
// FP32 flops of the counted distance work (counters as in DistanceArgs::work_counters).
double distance_work_flops(int tile_id, const unsigned long long *counters);
// tile shape id -> (tx, ty, tz)
void tile_shape(int id, int &tx, int &ty, int &tz);
uint64_t tiles_for(const GridDev &g, int tile_id);
// Deferred-list capacity for a launch of total_tiles tiles.
uint64_t defer_capacity_for(uint64_t total_tiles);
cudaError_t distance_launch(const DistanceArgs &a, int tile_id, int num_sms, cudaStream_t st);

// Every (cell, triangle) pair of a ONE-mesh batch that passes the occupancy rule, as keys
// (cell << tri_bits) | local triangle, appended in no particular order (the mesh's occupancy grid
// is written as well). *hit_count (device) receives the number of hits, also when it exceeds
// `capacity` (then only `capacity` keys are written).
cudaError_t occupancy_hits(const BatchDev &B, void *temp, size_t temp_bytes, uint64_t *keys, uint64_t capacity,
                           unsigned long long *hit_count, int tri_bits, int num_sms, cudaStream_t st);

// ---- weld.cu ----------------------------------------------------------------------------------
// v[i] = i for i < n.
cudaError_t iota_device(uint32_t *v, uint64_t n, int num_sms, cudaStream_t st);
// weldPositions on the device: welded[i] = the first-occurrence number of position i's lattice key
// (cell: the weld lattice, weld_cell in host_mesh.h); unique (optional) gets each number's first
// position. *num_unique points at the count in device memory (valid until temp is reused).
size_t weld_temp_bytes(uint64_t n);
cudaError_t weld_enqueue(const float *pos, uint64_t n, float cell, uint32_t *welded, float *unique, void *temp,
                         size_t temp_bytes, const uint64_t **num_unique, int num_sms, cudaStream_t st);
// The same, waiting for the count.
cudaError_t weld_device(const float *pos, uint64_t n, float cell, uint32_t *welded, void *temp, size_t temp_bytes,
                        uint32_t *num_unique, int num_sms, cudaStream_t st);
// Edge census of a welded triangle list (degenerate triangles skipped). *counts points at two device
// values: boundary edges - 1 and non-manifold edges - 1.
size_t watertight_temp_bytes(uint64_t T);
cudaError_t watertight_enqueue(const uint32_t *welded, uint64_t T, void *temp, size_t temp_bytes,
                               const unsigned long long **counts, int num_sms, cudaStream_t st);
// The same, waiting for the counts.
cudaError_t watertight_device(const uint32_t *welded, uint64_t T, void *temp, size_t temp_bytes, uint64_t *boundary,
                              uint64_t *nonmanifold, int num_sms, cudaStream_t st);

// ---- sparse.cu --------------------------------------------------------------------------------
size_t sparse_temp_bytes(size_t cells, size_t max_out);
// Counts occupied cells (synchronises the stream; *h_total is host memory).
cudaError_t sparse_count(const uint8_t *occ, size_t cells, void *temp, size_t temp_bytes, uint64_t *h_total,
                         cudaStream_t st);
// Writes the occupied cell indices ordered by (first triangle, cell index) into cells_out. counted:
// temp still holds what sparse_count left there.
cudaError_t sparse_emit(const uint8_t *occ, const uint32_t *first_tri, size_t cells, uint64_t total, int tri_bits,
                        bool counted, void *temp, size_t temp_bytes, uint32_t *cells_out, cudaStream_t st);

// x, y and z of n listed cells of a res^3 grid.
cudaError_t sparse_coords(const uint32_t *list, uint64_t n, uint32_t res, int32_t *xyz, cudaStream_t st);

}  // namespace sdfb
