// stq_internal.h - host-side internals shared by the CUDA translation units:
// the context object behind stq_context*, grow-only device buffers and the
// kernel launch wrappers.
#pragma once

#include <atomic>
#include <cstdint>
#include <string>
#include <utility>

#include <cuda_runtime.h>

#include "../../include/stq_abi.h"

namespace stq {

// Grow-only device allocation owned by a context.
struct DevBuf {
  void *ptr = nullptr;
  size_t bytes = 0;
  cudaError_t ensure(size_t want) {
    if (want <= bytes) return cudaSuccess;
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    bytes = 0;
    size_t rounded = (want + 4095) & ~size_t(4095);
    cudaError_t e = cudaMalloc(&ptr, rounded);
    if (e == cudaSuccess) {
      bytes = rounded;
    } else {
      ptr = nullptr;
      (void)cudaGetLastError();  // a refused allocation is no error of the next launch
    }
    return e;
  }
  void release() {
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    bytes = 0;
  }
  template <typename T> T *as() const { return static_cast<T *>(ptr); }
};

// Lets a kernel take more than 48 KB of shared memory; asked once per kernel
// and device.
template <auto Kern>
cudaError_t allow_smem(size_t bytes) {
  static std::atomic<unsigned long long> done{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 64 && (done.load() >> dev & 1ull)) return cudaSuccess;
  e = cudaFuncSetAttribute(Kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
  if (e == cudaSuccess && dev < 64) done.fetch_or(1ull << dev);
  return e;
}

// Launches a kernel that is placed on the device while the last blocks of the one
// before it in the stream end, and waits at its start (after_previous). A pass of a
// small scene is some fifteen kernels of 3 to 15 us, and the gaps between plain
// launches a tenth of it. Whole passes, plain -> so: 2,000 boxes 134 -> 119 us,
// 53,000 boxes 195 -> 166, 477,000 boxes 331 -> 298; large scenes gain 1% (6 M
// boxes) to 3%. Kernels do not let the next one in earlier: its waiting blocks take
// shared memory from the running ones' L1 cache (16 scenes of 500,000 boxes
// 1.38 ms plain, 1.35 so, 1.55 with the next let in at the start). Errors are
// left to cudaGetLastError.
template <typename... P, typename... A>
void launch_after(void (*kern)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, A &&...args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

// Device-side scalars of one sweep: counters, flags and results read back
// by the host in a single copy.
struct DevScalars {
  unsigned long long count;  // pairs found (keeps counting past capacity)
  int work;                  // start-box grab cursor of the sweep kernel
  int flags;                 // kFlag* bits set by kernels
  long long prefix;          // start boxes of the longest prefix that fits
  int axis;                  // sweep axis chosen on the device
  int pad[3];
};

enum : int {
  kFlagNaN = 1,        // a box bound is NaN
  kFlagBadIndex = 2,   // an edge or face index is outside [0, nV)
  kFlagReplicaOverflow = 4,  // cell replicas exceed the replica buffers
};

// Cells per axis of a scene's grid at most (automatic or STQ_OPT_CELLS); cell
// coordinates then fit 11 bits, as the per-box cell records pack them.
constexpr int kMaxGridSide = 2048;

// Cell grid on the two non-sweep axes b, c (the other two axes in increasing
// order). A box is replicated into every cell its [min, max] range touches;
// cell coordinates are a monotone function of the bound, so a pair that
// overlaps shares the cell of its reference point (max of mins on b and c)
// and is emitted there only.
// The policy sets the level-0 grid (nb0 x nc0 cells of the automatic side, or
// the requested grid); a cell of level L is a block of 2^L x 2^L level-0
// cells, and the level is chosen against the replica budget once the box-key
// pass has counted every level's replicas.
struct GridParams {
  int axis;       // sweep axis a
  int nb, nc;     // cells along b and c at the chosen level
  int ncells;     // nb * nc
  float ob, oc;   // grid origin on b and c
  float ib, ic;   // level-0 cells per unit length on b and c
  float Lb, Lc;   // extent of the scene on b and c
  int nb0, nc0;   // level-0 cells along b and c
  int shift;      // cell coordinate = level-0 coordinate >> shift (the chosen
                  // level; kCoordBits when no level fits: one cell)
  float sb, sc;   // code steps (64 per cell of the chosen level) per unit length
  uint32_t key_lo, key_span;  // float keys on the sweep axis: the least minimum, and up to
                              // the largest maximum (long lists, see BatchHeader::exact)
};

constexpr int kGridLevels = 6;  // level L halves the level-0 grid L times
constexpr int kCoordBits = 11;  // level-0 cell coordinates are below 2^11
static_assert(kMaxGridSide <= (1 << kCoordBits), "level-0 cell coordinates fit kCoordBits");

// Sweep-axis codes: 16 bits, 64 segments of 1,024 steps. The inner segments hold
// about the same number of boxes each (their ends are quantiles of a sample), the
// first and the last those before and after the sample, 1 in 256 each: a box far away
// widens the steps of no others. A segment with a gap in it still puts many boxes on
// few steps: batches of few, long lists have keys of more bits (BatchHeader::exact).
constexpr int kSplits = 64;
constexpr int kSplitSteps = 1024;
constexpr int kAxisCodeBits = 16;
static_assert(kSplits * kSplitSteps == 1 << kAxisCodeBits, "16-bit codes");

// One scene of a batch, as computed by the prepare kernels.
struct SceneRecord {
  float split[kSplits];             // sweep-axis codes: lower ends of the segments
  float split_inv[kSplits];         // code steps per unit length in each
  GridParams grid;
};

// Per-scene inputs, written by the host before every prepare.
struct SceneInput {
  int axis_mode;        // -1: largest variance, else the axis
  int cells_opt;        // 0 automatic, 1 no cells, k > 1 a k x k grid
  float cell_scale;     // automatic cell side in median box extents
  int tiles;            // tiles of the scene
};

// Per-scene accumulators of a prepare, on the device: zero before it, and cleared by
// the blocks that read them (uploaded with the inputs, 20,000 scenes were 3 MB to fill
// and copy).
struct SceneSums {
  double s1[3], s2[3];               // sum(min + max), sum(min^2 + max^2)
  unsigned int lo_not[3], hi_key[3]; // order-preserving keys of the bounds: ~ of the least, the largest
  int inverted;                      // some box has min > max on an axis
  unsigned int done;                 // tiles whose statistics are in
  unsigned int keys_done, pad;       // tiles whose box keys are
  unsigned long long level_reps[kGridLevels];  // replicas per grid level
};

// Device-side header of a prepared batch: sizes read by every kernel, so a
// captured graph can be replayed for any batch within its capacities.
struct BatchHeader {
  // what kernels read first, on one line of 128 bytes
  long long n_boxes;        // input: boxes in the batch
  int n_scenes;             // input: scenes
  int n_tiles;              // input: entries of the tile table
  unsigned int replicas;    // R, cell replicas
  unsigned int cells;       // total cells of all scenes
  unsigned int length;      // sweep positions: R + 3 * cells - 1
  unsigned int lists;       // (cell, type) lists: 3 * cells
  int fault;                // a bounded wait between blocks ran out
  int key_bits;             // sweep-axis bits of a replica key (the list id is above)
  int exact;                // they are the leading bits of the minimum's float key above
                            // the scene's least, not of its 16-bit code
  unsigned int passes;      // digits of the replica sort; its input is in buffer passes & 1
  int budget;               // replica budget: replicas <= budget * boxes per scene
  int flags;                // kFlag* bits
  int axis;                 // sweep axis of scene 0
  unsigned int max_list;    // longest (cell, type) list
  // counters
  alignas(128) unsigned long long pairs;  // pairs found by the last sweep
  int work;                 // sweep grab cursor
  unsigned int long_items;  // runs handed from the lane sweep to the warp pass
  unsigned long long long_work;  // warp pass grab cursor
  unsigned long long candidates; // candidates tested by the last sweep
  long long prefix;         // overflow: start positions of the prefix that fits
  unsigned long long used;  // replicas of all scenes at their levels, accumulated
  unsigned int keys_done;   // tiles whose box keys and level counts are in
};

// What the host needs of a prepare's first half, written by the device to
// page-locked memory.
struct FrontInfo {
  unsigned long long replicas;  // replicas and cells that the scenes need
  unsigned long long cells;
  unsigned int passes;          // digits of the replica sort
  int flags;                    // kFlag* bits
};

// A tile of at most kTileBoxes consecutive boxes of one scene (built by the
// host from the scene offsets), so that a block reduces per-scene values once.
constexpr int kTileBoxes = 4096;
// Batches of up to kSmallBatch boxes take tiles of 1,024, so that most SMs get one,
// those of up to kMidBatch tiles of 2,048, and those of up to kTinyBatch tiles of 256,
// one box per thread (the lines are two or four tiles for each of 152 SMs). Whole passes
// with tiles of 1,024 -> 256: 2,000 boxes 118 -> 107 us, 53,000 boxes 167 -> 166, 477,000
// boxes 297 -> 318 (the last block scans the tiles); sweeps with tiles of 1,024, 2,048
// and 4,096: 650,000 boxes 239, 227, 239 us, 1 M 295, 288, 297, 1.2 M 346, 343, 350; 9.1 M
// boxes with 2,048 and 4,096: 3,018, 3,006.
constexpr int kSmallTile = 1024, kMidTile = 2048, kTinyTile = 256;
constexpr int64_t kTinyBatch = 152 * 2 * kTinyTile;
constexpr int64_t kSmallBatch = 152 * 4 * kSmallTile, kMidBatch = 152 * 4 * kMidTile;
constexpr int tile_boxes(int64_t n) {
  return n <= kTinyBatch ? kTinyTile : (n <= kSmallBatch ? kSmallTile : (n <= kMidBatch ? kMidTile : kTileBoxes));
}
// Most tiles of a batch of up to n boxes, but for one more per scene.
constexpr int64_t most_tiles(int64_t n) {
  int64_t t = n / kTileBoxes;
  for (const int64_t v : {kTinyBatch / kTinyTile, kSmallBatch / kSmallTile, kMidBatch / kMidTile}) t = t > v ? t : v;
  return t;
}
struct TileRec {
  long long begin;  // first box of the tile
  int count;        // boxes in the tile (0: the one tile of an empty scene)
  int scene;        // scene of the tile
};

// Sweep shapes (STQ_OPT_SWEEP_SHAPE): a per-warp ring of pending start boxes
// taken by lanes or lane groups, or the flat shape (each warp's 32 starts'
// runs laid end to end, one candidate per lane and step).
constexpr int kShapeRing = 1;
constexpr int kShapeFlat = 2;

// Sweep-kernel tuning (autotuned or set through stq_context_set_option).
struct SweepTuning {
  int shape = kShapeFlat;  // kShapeFlat or kShapeRing
  int lanes = 1;        // lanes sharing one pending start box (1..32)
  int per_lane = 8;     // lanes = 1: candidates a lane tests per step (1, 2, 4, 8)
  int run_cap = 512;    // candidates per start box before the warp pass takes over
  int queue = 64;       // warp queue depth (32, 64, 128)
  int block = 256;      // threads per block (128, 256, 512)
  int chunk = 256;      // start boxes per work grab
};

// One sorted position: what the exact test of a pair reads.
struct PosRec {
  float4 yz;  // (min_b, min_c, max_b, max_c) on the non-sweep axes
  float2 x;   // (min, max) on the sweep axis
  int4 v;     // vertexIds[0..2], id
};

// Sorted scene in HBM, structure of arrays. Every list is followed by one empty
// position (partner = run_end = itself).
struct SortedScene {
  float4 *yz = nullptr;
  float2 *x = nullptr;
  int4 *v = nullptr;
  int *flag = nullptr;        // first-cell bits (0: along b, 1: along c), scene << 2
  uint32_t *scode = nullptr;  // y/z interval in the cell and first-cell bits
                              // (position codes, stq_device.cuh)
  int *partner = nullptr;     // first candidate position of each start position
  int *run_end = nullptr;     // one past its last candidate
  int64_t length = 0;         // sweep positions (boxes; sentinels excluded at the end)
};

// Counters of one sweep launch that runs beside another (a host call's
// windows alternate between two of these), in device memory.
struct WindowCounters {
  unsigned long long pairs;  // pairs found
  int work;                  // grab cursor
  unsigned int long_items;   // runs handed to the warp pass
  unsigned long long long_work;  // warp pass grab cursor
};

// Where one sweep launch keeps its counters and handed-over runs.
struct SweepCursors {
  unsigned long long *count;
  int *work;
  int2 *long_list;
  unsigned int *long_items;
  unsigned long long *long_work;
};

struct SweepParams {
  const float4 *yz;          // bounds on the non-sweep axes
  const float2 *x;           // on the sweep axis
  const int4 *v;             // vertex ids and id
  const int *flag;           // first-cell bits and scene
  const uint32_t *scode;     // position codes
  const int *partner;        // first candidate position of each start position
  const int *run_end;        // one past its last candidate
  int32_t begin, end;        // start positions [begin, min(end, hdr->length))
  int32_t chunk;             // start positions per grab, at most
  int32_t grabs;             // and as many as make this number of grabs (0: chunk)
  stq_pair *pairs;
  long long capacity;
  unsigned long long *count;
  int *work;
  int32_t *box_counts;       // count mode: pairs per start position (k - begin)
  unsigned long long *scene_pairs;  // per-scene pair counters
  const BatchHeader *hdr;    // device sizes (length bounds the sweep range)
  unsigned long long *stats; // candidates tested (may be null)
  int typed;                 // every list holds one box type, so every candidate
                             // pair is V-F, F-V or E-E (is_valid_pair holds)
  int run_cap;               // candidates of one start box a lane (group) tests
                             // before it hands the rest of the run to the warp
                             // pass; 0 = never
  int2 *long_list;           // handed-over runs (start position, next candidate)
  unsigned int *long_items;  // their count
  unsigned long long *long_work;  // warp pass grab cursor
  const DevScalars *sel;     // if set: start positions [begin, begin + sel->prefix),
                             // and none if sel->count pairs fit the capacity
};

// What a sweep does with its pairs.
enum SweepMode {
  kSweepEmit = 0,   // writes them
  kSweepCount = 1,  // counts them per start position
  kSweepBoth = 2,   // both
};

// ---- launch wrappers (each returns the launch error) -------------------------
// points: 2 * nV float4 of scratch for the rounded positions
cudaError_t launch_build_boxes(cudaStream_t s, const double *V0, const double *V1,
                               int64_t nV, const int32_t *E, int64_t nE,
                               const int32_t *F, int64_t nF, float r_up,
                               stq_aabb *out, int *flags, float4 *points);

// ---- batch prepare (scene table) ---------------------------------------------------
// Buffers sized by host capacities; actual sizes come from the BatchHeader.
struct BatchBuffers {
  const stq_aabb *boxes;
  const long long *box_off;     // n_scenes + 1 box offsets
  const TileRec *tiles;         // n_tiles entries
  int tile_cap;
  const SceneInput *inputs;     // n_scenes entries
  SceneSums *sums;              // n_scenes entries, zero between prepares
  unsigned long long *scene_pairs;  // n_scenes pair counters
  SceneRecord *scenes;
  unsigned int *cell_base;      // n_scenes + 1
  BatchHeader *hdr;
  FrontInfo *front;             // page-locked
  uint2 *box_cells;             // per box: cell range and type
                                // (b0 | b1 << 11 | type << 22, c0 | c1 << 11)
  uint32_t *box_q;              // per box: sweep-axis codes of its min | its max << 16 (exact
                                // keys: the max's alone, in the leading bits)
  unsigned long long *tile_reps;  // per tile: replicas of each grid level
  uint32_t *tile_off;           // per tile: first replica
  uint32_t *keys[2];            // replica keys: list id << key_bits | sweep-axis code
  uint32_t *vals[2];            // replica box indices
  uint32_t *seg_scan;           // first sorted replica of each segment (cell x type),
                                // seg_cap + 1 entries
  long long seg_cap;
  long long box_cap;            // capacities
  long long rep_cap;
  int scene_cap;
};
// per-scene statistics; sweep axis, level-0 grid and sweep-axis codes (1 launch)
cudaError_t launch_batch_stats(cudaStream_t s, const BatchBuffers &b);
// level-0 cell ranges, sweep-axis codes and every level's replica count; then the
// level within the replica budget, the cell bases, the key layout and every
// tile's first replica (1 launch). Scenes that need more than rep_cap replicas,
// seg_cap lists or `passes` digits of the replica sort are flagged and left empty
// (no limit: rep_cap -1).
cudaError_t launch_batch_box_keys(cudaStream_t s, const BatchBuffers &b, int64_t rep_cap, int64_t seg_cap, int passes);
// replicas in box order (1 launch)
cudaError_t launch_batch_emit(cudaStream_t s, const BatchBuffers &b);
// list offsets from the sorted keys (and the longest list); the empty position
// after every list and the padding after the last. lists: to launch blocks for
cudaError_t launch_list_offsets(cudaStream_t s, const uint32_t *keys, BatchHeader *hdr, uint32_t *seg_scan,
                                int64_t seg_cap, const SortedScene &scene, int64_t slots_cap, int64_t lists);

cudaError_t launch_gather_cells(cudaStream_t s, const BatchBuffers &b, int64_t replicas, const SortedScene &scene);
// Batched box build: scene s has vertices [voff[s], voff[s+1]) etc.; box ids
// are global (box_off[s] + local), vertex ids local to the scene.
// points: 2 * vert_cap float4 of scratch for the rounded positions
cudaError_t launch_batch_build(cudaStream_t s, const double *V0, const double *V1,
                               const long long *voff, const int32_t *E, const long long *eoff,
                               const int32_t *F, const long long *foff, const long long *box_off,
                               const TileRec *tiles, int tile_cap, BatchHeader *hdr, float r_up, stq_aabb *out,
                               float4 *points, int64_t vert_cap);
// A scene held by the serving loop: its own device mesh and time-step state.
struct MeshRef {
  double *V0, *V1;
  const int32_t *E, *F;
  long long nV, nE, nF;
  unsigned long long seed;
  double sigma;
  int step;   // timestep about to run (0: the submitted positions)
  int pad;
};
cudaError_t launch_advance(cudaStream_t s, const MeshRef *refs, const long long *voff,
                           const BatchHeader *hdr, int64_t vert_cap);
cudaError_t launch_batch_build_refs(cudaStream_t s, const MeshRef *refs, const long long *box_off,
                                    const TileRec *tiles, int tile_cap, BatchHeader *hdr, float r_up, stq_aabb *out);
cudaError_t launch_pair_checksums(cudaStream_t s, const stq_pair *pairs, long long capacity,
                                  const BatchHeader *hdr, const long long *box_off,
                                  unsigned long long *checks, int scene_cap);
cudaError_t launch_reset_sweep(cudaStream_t s, BatchHeader *hdr, unsigned long long *scene_pairs,
                               int scene_cap, const DevScalars *sel = nullptr,
                               long long capacity = 0);
// host_count: device address of page-locked, mapped host memory
cudaError_t launch_window_step(cudaStream_t s, WindowCounters *wc, unsigned long long *host_count);

// Stable LSD radix sorts (8-bit digits). kbuf/vbuf are double buffers.
// fault: device-visible word set to 1 if a bounded wait between blocks ran out
// (the result is then not sorted). d_n (may be null): on the device, the number
// of elements (at most n).
constexpr int kRadixMinTile = 2048;       // keys of the smallest tile of a pass
constexpr int64_t kRadixMinTiles = 1 << 13;  // most tiles of that size
constexpr size_t kRadixHeadBytes = 8704;  // digit counts, cursors
// Workspace of a sort of up to n elements: the head and 256 status words per
// tile. The smallest tiles are used below a fixed size, larger ones (at least
// twice as long) above it.
constexpr size_t radix_workspace_bytes(int64_t n) {
  const size_t tiles = size_t((n > 0 ? n : 1) + kRadixMinTile - 1) / kRadixMinTile;
  const size_t half = (tiles + 1) / 2, small_max = size_t(kRadixMinTiles);
  const size_t small = tiles < small_max ? tiles : small_max;
  return kRadixHeadBytes + sizeof(unsigned long long) * 256 * (small > half ? small : half);
}
// result in kbuf[0], vbuf[0]. d_passes (may be null: 4): on the device, the
// number of low digits to sort by, at most `passes`; the input is then in
// buffer *d_passes & 1, else in buffer 0. likely: the expected number of elements
// (-1: n); the tile size follows it.
cudaError_t radix_sort_u32(cudaStream_t s, uint32_t *const kbuf[2], uint32_t *const vbuf[2], int64_t n, void *workspace,
                           int *fault, int64_t *launches, const unsigned int *d_n = nullptr,
                           const unsigned int *d_passes = nullptr, int passes = 4, int64_t likely = -1);
// by digits; lexicographic by (first, second) as unsigned ids, in place; tmp holds n pairs
cudaError_t radix_sort_pairs(cudaStream_t s, stq_pair *pairs, stq_pair *tmp, int64_t n, void *workspace, int *fault,
                             int64_t *launches);
// What the host needs of a pair sort's histogram, in page-locked memory.
struct PairPlan {
  unsigned int max_first;  // largest first id
  unsigned int fits;       // no bucket was too long: the pairs are sorted
  unsigned int big;        // but for those of these buckets, which take another launch
};
size_t pair_workspace_bytes(int64_t n);
// Lexicographic sort of pairs by buckets of their first id (by digits where ids
// have too many pairs), in place; tmp holds n pairs. May wait for the stream.
// id_bits: bits of the largest first id of earlier sorts, kept for the next.
cudaError_t sort_pairs(cudaStream_t s, stq_pair *pairs, stq_pair *tmp, int64_t n, void *workspace, PairPlan *plan,
                       int *id_bits, int *fault, int64_t *launches);
// Multiprocessors of the current device.
int sm_count();

cudaError_t launch_sweep(cudaStream_t s, const SweepParams &p,
                         const SweepTuning &t, SweepMode mode, int num_sms);
// inclusive scan of box_counts[0..m) and the longest prefix whose pair sum
// is <= capacity -> scalars->prefix; *found (or, with none, more than any
// capacity) -> scalars->count
size_t prefix_workspace_bytes(int64_t m);
cudaError_t launch_prefix_select(cudaStream_t s, const int32_t *box_counts,
                                 int64_t m, long long capacity, void *workspace,
                                 DevScalars *scalars, int64_t *launches,
                                 const unsigned long long *found);
cudaError_t launch_brute_force(cudaStream_t s, const stq_aabb *boxes, int64_t n,
                               stq_pair *pairs, long long capacity,
                               unsigned long long *count);

}  // namespace stq
