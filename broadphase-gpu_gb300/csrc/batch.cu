// batch.cu - prepare kernels of the scene table: per-scene statistics, sweep
// axis and cell grid, cell replicas with their sort keys, and the sorted-scene
// gather with one empty position after every list.
//
// Reference: create_ds (src/sweep.cu:125-161) and the axis choice of
// calc_mean / calc_variance (src/sweep.cu:93-123); the reference sorts one
// scene along x. Here every scene of a batch gets its own sweep axis and
// y/z cell grid, all scenes' cells get global ids, and one sort orders every
// replica by (cell, box type, sweep-axis code). The code is a monotone 16-bit
// image of the minimum (more bits of it where lists are few and long): a list is
// sorted up to boxes of one code, its runs hold every candidate of a code that can
// overlap, and the sweep tests the sweep axis exactly for the pairs that pass its
// filter. So the whole key fits 24 or 32 bits, and the boxes need no sort of their own.
//
// All sizes are read from the BatchHeader on the device, so one captured
// graph serves any batch within the buffer capacities.
#include <mutex>
#include <utility>
#include <vector>

#include "stq_device.cuh"
#include "stq_internal.h"

namespace stq {

namespace {

constexpr int kBlock = 256;
constexpr int kHistBias = 40;  // extent bucket = binary exponent + 40
constexpr int kSampleBoxes = 1024;
constexpr int kSampleMins = 256;  // of these, for the sweep-axis code segments

__device__ __forceinline__ void axes_bc(int a, int &b, int &c) {
  b = a == 0 ? 1 : 0;
  c = a == 2 ? 1 : 2;
}

// Block sums of K values per thread with one shared-memory exchange; out[k]
// is valid in thread 0.
template <typename T, int K>
__device__ void block_sums(const T (&v)[K], T (&out)[K], T (*red)[K]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    T x = v[k];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(kFullMask, x, o);
    if (lane == 0) red[warp][k] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      T t = 0;
      for (int w = 0; w < kBlock / 32; ++w) t += red[w][k];
      out[k] = t;
    }
  }
}

// Exclusive scan of one value per thread of the block; *total in every thread.
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t *total, uint32_t *scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFullMask, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();  // scratch may be in use
  if (lane == 31) scratch[warp] = x;
  __syncthreads();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < kBlock / 32; ++w) {
    before += w < warp ? scratch[w] : 0u;
    all += scratch[w];
  }
  *total = all;
  return before + x - v;
}

__device__ int grid_side(float L, float h) {
  if (!(L > 0.f) || !(h > 0.f) || !isfinite(L)) return 1;
  const float s = ceilf(L / h);
  return s > float(kMaxGridSide) ? kMaxGridSide : (s < 1.f ? 1 : int(s));
}

__device__ __forceinline__ float inv_side(int n, float L) { return n > 1 ? float(n) / L : 0.f; }

// ---- 2. policy of a scene, by the block that finished its statistics ---------------
// Sweep axis of largest corner variance (x, then y, preferred on ties, as
// src/simulation.cu:630-635) unless fixed; level-0 cell side = cell_scale x
// median box extent (from a strided sample of the scene's boxes), at most
// 2048 cells per axis and at most max(1, n / max(16, 8 x cell_scale)) cells.
__device__ __forceinline__ void
scene_policy(const stq_aabb *__restrict__ boxes, long long b0, long long n, const SceneInput &in, SceneSums &sums,
             SceneRecord &r, int scene, BatchHeader *hdr) {
  // the accumulators were written by other blocks' atomics: read them from L2
  uint32_t lo_key[3], hi_key[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) lo_key[k] = ~__ldcg(&sums.lo_not[k]), hi_key[k] = __ldcg(&sums.hi_key[k]);
  const bool inverted = __ldcg(&sums.inverted) != 0;
  int axis = in.axis_mode;
  if (axis < 0) {
    __shared__ double var[3];
    if (threadIdx.x < 3) {
      const double m = n > 0 ? 2.0 * double(n) : 1.0;
      const double mean = __ldcg(&sums.s1[threadIdx.x]) / m;
      var[threadIdx.x] = __ldcg(&sums.s2[threadIdx.x]) - m * mean * mean;
    }
    __syncthreads();
    axis = 0;
    if (var[1] > var[axis]) axis = 1;
    if (var[2] > var[axis]) axis = 2;
  }
  auto key_of = [&](const uint32_t (&k)[3], int a) { return a == 0 ? k[0] : (a == 1 ? k[1] : k[2]); };
  int b, c;
  axes_bc(axis, b, c);
  __shared__ unsigned hist[2][64];
  __shared__ __align__(16) float sample[kSampleMins];
  __shared__ float sorted[kSampleMins];
  __shared__ float median[2];
  for (int i = threadIdx.x; i < 128; i += kBlock) (&hist[0][0])[i] = 0u;
  static_assert(kSampleMins == kBlock, "one sampled minimum per thread");
  sample[threadIdx.x] = INFINITY;
  __syncthreads();
  const bool automatic = in.cells_opt == 0 && !inverted && n > 1;
  {
    const long long step = n > kSampleBoxes ? n / kSampleBoxes : 1;
    // every fourth sample gives a minimum on the sweep axis (all of them in
    // scenes of fewer boxes than minima wanted)
    constexpr int kPer = kSampleBoxes / kBlock;
    const int every = n > kSampleMins ? kPer : 1;
    const int ax[2] = {b, c};
    float mins[kPer], ext[kPer][2];  // all loads first
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const long long i = (long long)(u * kBlock + threadIdx.x) * step;
      if (i < n) {
        const stq_aabb &x = boxes[b0 + i];
        mins[u] = x.min[axis];
        for (int q = 0; q < 2; ++q) ext[u][q] = x.max[ax[q]] - x.min[ax[q]];
      }
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int i = u * kBlock + threadIdx.x;
      if (i * step >= n) continue;
      if (i % every == 0 && i / every < kSampleMins) sample[i / every] = mins[u];
      if (!automatic) continue;
      for (int q = 0; q < 2; ++q) {
        int bucket = 0;
        if (ext[u][q] > 0.f) {
          int e;
          frexpf(ext[u][q], &e);
          bucket = min(63, max(1, e + kHistBias));
        }
        atomicAdd(&hist[q][bucket], 1u);
      }
    }
  }
  __syncthreads();
  // the sampled minima in order: each thread counts those before its own
  // (missing ones are +inf, at the end)
  {
    const float mine = sample[threadIdx.x];
    int rank = 0;
#pragma unroll 8
    for (int i = 0; i < kSampleMins; i += 4) {
      const float4 v = *reinterpret_cast<const float4 *>(&sample[i]);
      rank += (v.x < mine || (v.x == mine && i < int(threadIdx.x))) + (v.y < mine || (v.y == mine && i + 1 < int(threadIdx.x))) +
              (v.z < mine || (v.z == mine && i + 2 < int(threadIdx.x))) + (v.w < mine || (v.w == mine && i + 3 < int(threadIdx.x)));
    }
    // (a NaN bound, rejected later, may leave a place empty)
    sorted[threadIdx.x] = INFINITY;
    __syncthreads();
    sorted[min(rank, kSampleMins - 1)] = mine;
  }
  __syncthreads();
  // median extents: one warp per axis, two buckets per lane
  if (threadIdx.x < 64) {
    const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned h0 = hist[q][2 * lane], h1 = hist[q][2 * lane + 1];
    unsigned run = h0 + h1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(kFullMask, run, o);
      if (lane >= o) run += y;
    }
    const unsigned total = __shfl_sync(kFullMask, run, 31);
    // first bucket whose running count reaches half
    const unsigned m = __ballot_sync(kFullMask, total > 0 && 2 * run >= total);
    if (lane == 0) median[q] = 0.f;
    __syncwarp();
    if (m && lane == __ffs(m) - 1) {
      const int k = 2 * (run - h1) >= total ? 2 * lane : 2 * lane + 1;
      median[q] = k == 0 ? 0.f : 0.75f * exp2f(float(k - kHistBias));
    }
  }
  // sweep-axis code segments: the ends of the inner ones are quantiles of the sample;
  // the first and the last reach from it to the scene's bounds
  if (threadIdx.x >= 64 && threadIdx.x < 64 + kSplits) {
    const int i = threadIdx.x - 64;
    // samples taken: above
    const int m = n > kSampleMins ? int(min(n, (long long)kSampleBoxes) + 3) / 4 : max(int(n), 1);
    static_assert(kSampleBoxes / kBlock == 4, "every fourth sample gives a minimum");
    constexpr int kInner = kSplits - 2;
    const float s0 = i == 0 ? key_float(key_of(lo_key, axis)) : sorted[(i - 1) * (m - 1) / kInner];
    const float s1 = i == kSplits - 1 ? key_float(key_of(hi_key, axis)) : sorted[i * (m - 1) / kInner];
    const float w = s1 - s0;
    r.split[i] = s0;
    r.split_inv[i] = w > 0.f && isfinite(w) ? float(kSplitSteps) / w : 0.f;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int k = 0; k < 3; ++k) {  // for the next prepare
    sums.s1[k] = sums.s2[k] = 0.0;
    sums.lo_not[k] = sums.hi_key[k] = 0u;
  }
  sums.inverted = 0;
  sums.done = 0u;
  const float lob = key_float(key_of(lo_key, b)), hib = key_float(key_of(hi_key, b));
  const float loc = key_float(key_of(lo_key, c)), hic = key_float(key_of(hi_key, c));
  const float Lb = hib - lob, Lc = hic - loc;
  int nb = 1, nc = 1;
  if (in.cells_opt > 1 && !inverted && n > 1) {
    nb = nc = in.cells_opt;
  } else if (automatic) {
    float w[2] = {median[0], median[1]};
    if (!(w[0] > 0.f)) w[0] = Lb / 1024.f;
    if (!(w[1] > 0.f)) w[1] = Lc / 1024.f;
    nb = grid_side(Lb, in.cell_scale * w[0]);
    nc = grid_side(Lc, in.cell_scale * w[1]);
    // at least max(16, 8 * scale) boxes per cell on average: dense scenes of
    // small boxes would otherwise be cut into lists of a few boxes, and their
    // prepare would outweigh the sweep (the buffers are sized for n / 16 cells)
    const long long per_cell = max(16ll, (long long)(8.f * in.cell_scale));
    const long long max_cells = max(1ll, min(1ll << 20, n / per_cell));
    while ((long long)nb * nc > max_cells) {
      if (nb >= nc) nb = (nb + 1) / 2;
      else nc = (nc + 1) / 2;
    }
  }
  if (!(Lb > 0.f) || !isfinite(Lb)) nb = 1;
  if (!(Lc > 0.f) || !isfinite(Lc)) nc = 1;
  GridParams &g = r.grid;
  g.axis = axis;
  g.key_lo = key_of(lo_key, axis);
  g.key_span = max(key_of(hi_key, axis), g.key_lo) - g.key_lo;
  g.ob = lob;
  g.oc = loc;
  g.Lb = Lb;
  g.Lc = Lc;
  g.ib = inv_side(nb, Lb);
  g.ic = inv_side(nc, Lc);
  g.nb0 = g.ib == 0.f ? 1 : nb;
  g.nc0 = g.ic == 0.f ? 1 : nc;
  if (scene == 0) hdr->axis = axis;
}

// ---- 1. statistics: one tile (one scene) per block ------------------------------
__global__ void __launch_bounds__(kBlock)
batch_stats_kernel(const stq_aabb *__restrict__ boxes, const TileRec *__restrict__ tiles,
                   const long long *__restrict__ box_off, const SceneInput *__restrict__ inputs, SceneSums *sums,
                   SceneRecord *scenes, BatchHeader *hdr) {
  after_previous();
  if (int(blockIdx.x) >= hdr->n_tiles) return;
  const TileRec t = tiles[blockIdx.x];
  if (threadIdx.x == 0) want_l2(&sums[t.scene]);
  // moments about the tile's first box centre, in fp32 per thread (fp64 is
  // slow on this part); the block combines them in fp64 and shifts them back
  float c[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float m = t.count > 0 ? 0.5f * (boxes[t.begin].min[k] + boxes[t.begin].max[k]) : 0.f;
    c[k] = isfinite(m) ? m : 0.f;
  }
  float s1[3] = {0.f, 0.f, 0.f}, s2[3] = {0.f, 0.f, 0.f};
  uint32_t lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[3] = {0u, 0u, 0u};
  bool inverted = false, nan = false;
  // thread i takes boxes i, i + kBlock, ...: each warp load instruction covers
  // 32 consecutive boxes, and the unrolled loop keeps several boxes in flight
  const stq_aabb *tb = boxes + t.begin;
#pragma unroll 4
  for (int i = threadIdx.x; i < t.count; i += kBlock) {
    const stq_aabb &x = tb[i];
    float l[3], h[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) l[k] = x.min[k], h[k] = x.max[k];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      nan |= (l[k] != l[k]) | (h[k] != h[k]);
      inverted |= l[k] > h[k];
      const float dl = l[k] - c[k], dh = h[k] - c[k];
      s1[k] += dl + dh;
      s2[k] += dl * dl + dh * dh;
      lo[k] = min(lo[k], float_key(l[k]));
      hi[k] = max(hi[k], float_key(h[k]));
    }
  }
  // warp sums in fp32 (a fixed shuffle tree); the 8 warp sums of each moment
  // are combined in fp64 by one lane each, and each value reaches the scene
  // record with one atomic per block (fp64 and same-address atomics are slow)
  constexpr int kWarps = kBlock / 32;
  __shared__ float wsum[6][kWarps];
  __shared__ uint32_t wkey[6][kWarps];
  __shared__ int wflag[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float m[6] = {s1[0], s1[1], s1[2], s2[0], s2[1], s2[2]};
#pragma unroll
  for (int k = 0; k < 6; ++k)
    for (int o = 16; o > 0; o >>= 1) m[k] += __shfl_down_sync(kFullMask, m[k], o);
  uint32_t kk[6];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    kk[k] = __reduce_min_sync(kFullMask, lo[k]);
    kk[3 + k] = __reduce_max_sync(kFullMask, hi[k]);
  }
  const int fl = (__any_sync(kFullMask, inverted) ? 1 : 0) | (__any_sync(kFullMask, nan) ? 2 : 0);
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < 6; ++k) wsum[k][warp] = m[k], wkey[k][warp] = kk[k];
    wflag[warp] = fl;
  }
  __syncthreads();
  SceneSums &r = sums[t.scene];
  __shared__ bool last;
  if (warp == 0) {
    double tot = 0.0;  // lane k < 6: moment k of the block
    uint32_t key = lane < 3 ? 0xffffffffu : 0u;  // lanes 0-2 minima, 3-5 maxima
    int flags = 0;
    if (lane < 6) {
      for (int w = 0; w < kWarps; ++w) {
        tot += double(wsum[lane][w]);
        key = lane < 3 ? min(key, wkey[lane][w]) : max(key, wkey[lane][w]);
        flags |= wflag[w];
      }
    }
    // sum(l + h) = S1 + 2 n c; sum(l^2 + h^2) = S2 + 2 c S1 + 2 n c^2
    const double a1 = __shfl_sync(kFullMask, tot, lane < 3 ? lane : lane - 3);
    if (lane < 6) {
      const int k = lane < 3 ? lane : lane - 3;
      const double ck = k == 0 ? c[0] : (k == 1 ? c[1] : c[2]), n = double(t.count);
      if (lane < 3) {
        atomicAdd(&r.s1[k], tot + 2.0 * n * ck);
        atomicMax(&r.lo_not[k], ~key);
      } else {
        atomicAdd(&r.s2[k], tot + 2.0 * ck * a1 + 2.0 * n * ck * ck);
        atomicMax(&r.hi_key[k], key);
      }
    }
    if (lane == 0 && (flags & 1)) atomicOr(&r.inverted, 1);
    if (lane == 0 && (flags & 2)) atomicOr(&hdr->flags, kFlagNaN);
    // the block whose tile is the scene's last goes on to its policy
    __threadfence();
    __syncwarp();
    if (lane == 0) last = atomicAdd(&r.done, 1u) + 1u == unsigned(inputs[t.scene].tiles);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const long long first = box_off[t.scene];
  scene_policy(boxes, first, box_off[t.scene + 1] - first, inputs[t.scene], r, scenes[t.scene], t.scene, hdr);
}

struct Range {
  int b0, b1, c0, c1;
};

__device__ __forceinline__ Range cell_range(const stq_aabb &x, int a, float ob, float ib, int nb,
                                            float oc, float ic, int nc) {
  int b, c;
  axes_bc(a, b, c);
  Range r;
  // (a box in a grid has min <= max, or a NaN bound, which is refused: cell 0)
  r.b0 = cell_coord(x.min[b], ob, ib, nb);
  r.b1 = max(cell_coord(x.max[b], ob, ib, nb), r.b0);
  r.c0 = cell_coord(x.min[c], oc, ic, nc);
  r.c1 = max(cell_coord(x.max[c], oc, ic, nc), r.c0);
  return r;
}

// ---- 4. the finest level of a scene within the replica budget, by one thread of the
// block that finished the scene's box keys; returns its replicas
__device__ __forceinline__ unsigned long long choose_level(const SceneInput &in, const unsigned long long (&level_reps)[kGridLevels],
                                                           GridParams &g, long long n, long long budget) {
  int level = kCoordBits;  // none fits: every coordinate shifts to cell 0
  unsigned long long used = (unsigned long long)n;  // one cell: each box once
  if (in.cells_opt > 1) {
    level = 0;  // a requested grid is kept as is
    used = level_reps[0];
  } else {
#pragma unroll
    for (int l = kGridLevels - 1; l >= 0; --l)
      if ((long long)level_reps[l] <= budget * n) {
        level = l;
        used = level_reps[l];
      }
  }
  g.shift = level;
  g.nb = ((g.nb0 - 1) >> level) + 1;
  g.nc = ((g.nc0 - 1) >> level) + 1;
  g.ncells = g.nb * g.nc;
  // 64 code steps per cell of the chosen level; a cell is 2^level level-0
  // cells, of which there are nb0 over Lb (one cell: the whole extent)
  const float steps = 64.f / float(1 << level);
  g.sb = g.Lb > 0.f && isfinite(g.Lb) ? (level >= kCoordBits ? 64.f : steps * float(g.nb0)) / g.Lb : 0.f;
  g.sc = g.Lc > 0.f && isfinite(g.Lc) ? (level >= kCoordBits ? 64.f : steps * float(g.nc0)) / g.Lc : 0.f;
  return used;
}

// Exclusive scan, by the block, of value(0 .. n - 1) into out; returns the total. Each
// thread takes several consecutive values where there are more than threads: their
// loads are in flight together, and one scan serves them all.
template <typename Value>
__device__ __forceinline__ uint32_t scan_into(int n, uint32_t *out, uint32_t *scratch, const Value &value) {
  constexpr int kMost = 8;
  const int per = min(kMost, (n + kBlock - 1) / kBlock);
  uint32_t carry = 0;
  for (int base = 0; base < n; base += kBlock * per) {
    const int i0 = base + int(threadIdx.x) * per;
    uint32_t v[kMost], sum = 0, total;
#pragma unroll
    for (int u = 0; u < kMost; ++u) v[u] = u < per && i0 + u < n ? value(i0 + u) : 0u;
#pragma unroll
    for (int u = 0; u < kMost; ++u) sum += v[u];
    uint32_t at = carry + block_exclusive(sum, &total, scratch);
#pragma unroll
    for (int u = 0; u < kMost; ++u)
      if (u < per && i0 + u < n) {
        out[i0 + u] = at;
        at += v[u];
      }
    carry += total;
  }
  return carry;
}

// What choose_level found, kept in the block for a batch of one scene.
struct OneScene {
  unsigned long long used;
  uint32_t cells;
  int level;
};

// Cell bases, the tiles' first replicas and the key layout, by the block that finished
// the box keys. (20,000 scenes of 20 boxes: the keys stage took 1,172 us with the levels
// chosen here, one scene per thread.)
__device__ __forceinline__ void
lay_out(const TileRec *__restrict__ tiles, const SceneRecord *scenes, const OneScene &one, unsigned int *cell_base,
        const unsigned long long *tile_reps, uint32_t *tile_off, BatchHeader *hdr, FrontInfo *front, long long rep_cap,
        long long seg_cap, int max_passes) {
  __shared__ uint32_t scratch[kBlock / 32];
  const int S = hdr->n_scenes;
  const uint32_t carry = scan_into(S, cell_base, scratch, [&](int s) {
    return S == 1 ? one.cells : uint32_t(__ldcg(&scenes[s].grid.ncells));
  });
  // every tile's first replica, at its scene's level
  scan_into(hdr->n_tiles, tile_off, scratch, [&](int t) {
    const int level = S == 1 ? one.level : __ldcg(&scenes[tiles[t].scene].grid.shift);
    return level < kGridLevels ? uint32_t(__ldcg(&tile_reps[size_t(t) * kGridLevels + level])) : uint32_t(tiles[t].count);
  });
  if (threadIdx.x == 0) {
    cell_base[S] = carry;
    const unsigned long long R = S == 1 ? one.used : __ldcg(&hdr->used), lists = 3ull * carry;
    // key: list id above the top bits of the sweep-axis code, 24 bits in all (three
    // digits) where that leaves the code 9 bits or more, else 32. At 10 bits the
    // 6 M-box scene (14 bits of lists) tests 9% more candidates and sorts a digit
    // less: sort + sweep 0.22 + 1.26 ms against 0.29 + 1.19 with 32 bits. With 15
    // bits of lists, 200,000 boxes (9 bits of code): 44 + 28 -> 36 + 28 us; with 16,
    // 256 scenes (8): the sweep's loss outweighs the digit by 50 us.
    // Batches of few, long lists (one cell: plain sweeps, inverted boxes, boxes on a line)
    // have what the list id leaves of 32 bits: where a 16-bit code is shared by a part
    // of a list, that part is tested all with all. 300,000 boxes of one cell in 200
    // clusters: 65.8 M candidates with codes, 0.8 M so, whole sweep 207 -> 148 us; evenly
    // spread, where codes are as good, the fourth digit costs 20 us (136 -> 157).
    // Shorter lists lose less than the digit costs.
    int seg_bits = 0;
    while (seg_bits < 32 && (1ull << seg_bits) < lists) ++seg_bits;
    const bool exact = seg_bits <= 8 && R >= 4096ull * lists;
    const int code_bits = min(kAxisCodeBits, seg_bits <= 15 ? 24 - seg_bits : max(32 - seg_bits, 0));
    const int key_bits = exact ? 32 - seg_bits : code_bits;
    const int passes = max(seg_bits + key_bits + 7, 8) / 8;
    // more than the buffers hold: the scenes are flagged and left empty (the
    // caller without limits checks that positions fit 31 bits). So are scenes with a
    // bad box: what follows is queued already
    const bool bad = hdr->flags != 0;
    const bool fits = !bad && R < 0xffffffffull &&
                      (rep_cap < 0 || ((long long)R <= rep_cap && (long long)lists <= seg_cap && passes <= max_passes));
    if (!fits && !bad) atomicOr(&hdr->flags, kFlagReplicaOverflow);
    hdr->replicas = fits ? unsigned(R) : 0u;
    hdr->cells = fits ? carry : 0u;
    hdr->lists = fits ? unsigned(lists) : 0u;
    // each of the 3 lists of a cell is followed by its empty position; the last
    // of these is not a start position
    hdr->length = fits && carry > 0 && R > 0 ? unsigned(R + lists - 1) : 0u;
    hdr->max_list = 0u;
    hdr->key_bits = key_bits;
    hdr->exact = exact ? 1 : 0;
    hdr->passes = unsigned(passes);
    front->replicas = R;
    front->cells = carry;
    front->passes = unsigned(passes);
    front->flags = hdr->flags;
  }
}

// ---- 3. per box: the level-0 cell range and type, the sweep-axis codes of its
// minimum and maximum, and the replicas of every grid level, per scene
__device__ __forceinline__ uint32_t axis_code(float v, const float *split, const float *inv) {
  int i = 0;
#pragma unroll
  for (int step = kSplits / 2; step > 0; step >>= 1)
    if (v >= split[i + step]) i += step;
  // monotone: the segment is, and so is the step inside it (round-to-nearest
  // operations, clamped; NaN, which only infinite ends give, counts as 0)
  const float t = __fmul_rn(__fsub_rn(v, split[i]), inv[i]);
  return uint32_t(i * kSplitSteps) + uint32_t(fminf(fmaxf(t, 0.f), float(kSplitSteps - 1)));
}

__global__ void __launch_bounds__(kBlock)
batch_box_keys_kernel(const stq_aabb *__restrict__ boxes, const TileRec *__restrict__ tiles,
                      const long long *__restrict__ box_off, const SceneInput *__restrict__ inputs, SceneSums *sums,
                      SceneRecord *scenes, unsigned int *cell_base, unsigned long long *tile_reps, uint32_t *tile_off,
                      BatchHeader *hdr, FrontInfo *front, long long rep_cap, long long seg_cap, int max_passes,
                      uint2 *__restrict__ box_cells, uint32_t *__restrict__ box_q) {
  after_previous();
  if (int(blockIdx.x) >= hdr->n_tiles) return;
  const TileRec t = tiles[blockIdx.x];
  if (threadIdx.x == 0) want_l2(&sums[t.scene].level_reps), want_l2(&hdr->keys_done);
  const SceneRecord &r = scenes[t.scene];
  const GridParams g = r.grid;
  __shared__ float split[kSplits], inv[kSplits];
  if (threadIdx.x < kSplits) {
    split[threadIdx.x] = r.split[threadIdx.x];
    inv[threadIdx.x] = r.split_inv[threadIdx.x];
  }
  __syncthreads();
  // a thread sees at most kTileBoxes / kBlock = 16 boxes of at most 2048^2
  // cells each: 32-bit sums per thread, 64-bit per block
  static_assert(uint64_t(kTileBoxes / kBlock) * kMaxGridSide * kMaxGridSide < (uint64_t(1) << 32),
                "per-thread level sums");
  unsigned reps[kGridLevels] = {};
#pragma unroll 2
  for (int i = threadIdx.x; i < t.count; i += kBlock) {
    const long long bi = t.begin + i;
    const stq_aabb &x = boxes[bi];
    box_q[bi] = axis_code(x.min[g.axis], split, inv) | axis_code(x.max[g.axis], split, inv) << 16;
    // level-0 coordinates fit kCoordBits = 11 bits
    const Range q = cell_range(x, g.axis, g.ob, g.ib, g.nb0, g.oc, g.ic, g.nc0);
    const unsigned type = unsigned(box_type(x.vertex_ids[1], x.vertex_ids[2]));
    box_cells[bi] = make_uint2(unsigned(q.b0) | unsigned(q.b1) << 11 | type << 22,
                               unsigned(q.c0) | unsigned(q.c1) << 11);
#pragma unroll
    for (int l = 0; l < kGridLevels; ++l)
      reps[l] += unsigned((q.b1 >> l) - (q.b0 >> l) + 1) * unsigned((q.c1 >> l) - (q.c0 >> l) + 1);
  }
  __shared__ unsigned long long red[kBlock / 32][kGridLevels];
  unsigned long long wide[kGridLevels], tot[kGridLevels];
#pragma unroll
  for (int l = 0; l < kGridLevels; ++l) wide[l] = reps[l];
  block_sums(wide, tot, red);
  __shared__ bool last;
  __shared__ OneScene one;
  if (threadIdx.x == 0) {
    const SceneInput &in = inputs[t.scene];
    SceneSums &sum = sums[t.scene];
    const unsigned tiles_all = unsigned(hdr->n_tiles);
#pragma unroll
    for (int l = 0; l < kGridLevels; ++l) {
      tile_reps[size_t(blockIdx.x) * kGridLevels + l] = tot[l];
      if (in.tiles > 1 && tot[l]) atomicAdd(&sum.level_reps[l], tot[l]);
    }
    // the block whose tile is the scene's last chooses its level (in a batch of one
    // scene, the one that goes on)
    bool scene_last = in.tiles == 1;
    if (!scene_last) {
      __threadfence();
      if (unsigned(in.tiles) != tiles_all) {
        scene_last = atomicAdd(&sum.keys_done, 1u) + 1u == unsigned(in.tiles);
      } else {
        scene_last = last = atomicAdd(&hdr->keys_done, 1u) + 1u == tiles_all;
      }
      if (scene_last) {  // the other blocks' sums, cleared for the next prepare
        __threadfence();
#pragma unroll
        for (int l = 0; l < kGridLevels; ++l) tot[l] = __ldcg(&sum.level_reps[l]), sum.level_reps[l] = 0ull;
        sum.keys_done = 0u;
      }
    }
    if (scene_last) {
      GridParams &sg = scenes[t.scene].grid;
      const unsigned long long used = choose_level(in, tot, sg, box_off[t.scene + 1] - box_off[t.scene], hdr->budget);
      if (unsigned(in.tiles) == tiles_all) one = OneScene{used, uint32_t(sg.ncells), sg.shift};
      else if (used) atomicAdd(&hdr->used, used);
    }
    // the block whose tile is the batch's last goes on to the layout
    __threadfence();
    if (unsigned(in.tiles) != tiles_all || in.tiles == 1) last = atomicAdd(&hdr->keys_done, 1u) + 1u == tiles_all;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  lay_out(tiles, scenes, one, cell_base, tile_reps, tile_off, hdr, front, rep_cap, seg_cap, max_passes);
}

// ---- 5. replica keys in box order: (list id << key_bits) | sweep-axis code, where
// the list is (global cell, box type). One tile (one scene) per block, from the
// tile's first replica on.
__device__ __forceinline__ uint32_t cells_count(uint2 r, int shift) {
  return (((r.x >> 11 & 2047u) >> shift) - ((r.x & 2047u) >> shift) + 1u) *
         (((r.y >> 11 & 2047u) >> shift) - ((r.y & 2047u) >> shift) + 1u);
}

// Sweep-axis bits of a bound's key where the batch's keys are exact: monotone, the
// bounds of inverted boxes clamped to the scene's.
__device__ __forceinline__ uint32_t exact_code(float v, const GridParams &g, int key_bits) {
  const uint32_t above = min(max(float_key(v), g.key_lo) - g.key_lo, g.key_span);
  return above >> max(32 - __clz(g.key_span) - key_bits, 0);
}

__global__ void __launch_bounds__(kBlock)
batch_emit_kernel(const stq_aabb *__restrict__ boxes, const uint2 *__restrict__ box_cells, uint32_t *box_q,
                  const TileRec *__restrict__ tiles, const uint32_t *__restrict__ tile_off,
                  const SceneRecord *__restrict__ scenes, const unsigned int *__restrict__ cell_base,
                  const BatchHeader *hdr, uint32_t *k0, uint32_t *k1, uint32_t *v0, uint32_t *v1) {
  after_previous();
  if (hdr->replicas == 0u || int(blockIdx.x) >= hdr->n_tiles) return;
  const int key_bits = hdr->key_bits;
  const bool exact = hdr->exact != 0;
  const bool second = hdr->passes & 1u;
  uint32_t *__restrict__ keys = second ? k1 : k0;
  uint32_t *__restrict__ vals = second ? v1 : v0;
  constexpr int kWarps = kBlock / 32;
  __shared__ uint32_t warp_count[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const TileRec t = tiles[blockIdx.x];
  const GridParams &g = scenes[t.scene].grid;
  const int sh = g.shift, nc = g.nc;
  const unsigned cb0 = cell_base[t.scene];
  uint32_t o = tile_off[blockIdx.x];
  // a warp takes consecutive boxes of the tile, 32 at a time
  const int share = (t.count + kWarps * 32 - 1) / (kWarps * 32) * 32;
  const int w0 = min(warp * share, t.count), w1 = min(w0 + share, t.count);
  uint32_t mine = 0;
#pragma unroll 4
  for (int i = w0 + lane; i < w1; i += 32) mine += cells_count(box_cells[t.begin + i], sh);
  mine = __reduce_add_sync(kFullMask, mine);
  if (lane == 0) warp_count[warp] = mine;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kWarps; ++w) o += w < warp ? warp_count[w] : 0u;
#pragma unroll 2
  for (int i = w0 + lane; i - lane < w1; i += 32) {
    uint2 r = make_uint2(0u, 0u);
    uint32_t n = 0, q = 0;
    if (i < w1) {
      r = box_cells[t.begin + i];
      if (exact) {  // (the gather takes the maximum's code from the same bits)
        const stq_aabb &x = boxes[t.begin + i];
        q = exact_code(x.min[g.axis], g, key_bits);
        box_q[t.begin + i] = exact_code(x.max[g.axis], g, key_bits) << (32 - key_bits);
      } else {
        q = (box_q[t.begin + i] & 0xffffu) >> (kAxisCodeBits - key_bits);
      }
      n = cells_count(r, sh);
    }
    uint32_t x = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(kFullMask, x, d);
      if (lane >= d) x += y;
    }
    uint32_t at = o + x - n;
    o += __shfl_sync(kFullMask, x, 31);
    if (i < w1) {
      const unsigned b0 = (r.x & 2047u) >> sh, b1 = (r.x >> 11 & 2047u) >> sh;
      const unsigned c0 = (r.y & 2047u) >> sh, c1 = (r.y >> 11 & 2047u) >> sh;
      const unsigned type = r.x >> 22;
      for (unsigned cb = b0; cb <= b1; ++cb)
        for (unsigned cc = c0; cc <= c1; ++cc) {
          const unsigned seg = (cb0 + cb * unsigned(nc) + cc) * 3u + type;
          keys[at] = seg << key_bits | q;
          vals[at] = uint32_t(t.begin + i);
          ++at;
        }
    }
  }
}

// First position of every (cell, type) list in the sorted replicas, and one
// entry past the last (the replica count): the keys are sorted by list id, so
// each offset is the lower bound of its id. Sorted replica p of list s sits at
// position p + s, so list s ends at position offset[s + 1] + s: the slot after
// it is an empty position (its run starts and ends at itself), and so are
// kSortedPad slots of padding after the last list. The gather writes every
// other position. Also the longest list, a statistic of the prepared scene.
__global__ void __launch_bounds__(kBlock)
list_offsets_kernel(const uint32_t *__restrict__ keys, BatchHeader *__restrict__ hdr,
                    uint32_t *__restrict__ seg_scan, long long seg_cap, SortedScene scene, int64_t slots_cap) {
  after_previous();
  // (cells past the capacity are flagged and counted as none; the loads together)
  const uint32_t nseg = uint32_t(min(3ll * hdr->cells, seg_cap));
  const uint32_t R = hdr->replicas;
  const int key_bits = hdr->key_bits;
  if (hdr->fault) return;  // the replicas are not sorted
  auto empty = [&](int64_t k) {
    if (k < slots_cap) {
      scene.partner[k] = int(k);
      scene.run_end[k] = int(k);
    }
  };
  // A search goes through a sample of the list ids in shared memory first (ten of
  // its steps) and then through the part of the keys that is left: a small scene
  // has too few lists to hide the chain of loads of a whole search.
  constexpr int kSample = 1024;
  __shared__ uint32_t sample[kSample];
  __shared__ uint32_t lows[kBlock];
  const uint32_t every = R / kSample + 1;  // sample[i] is the list id at i * every
  for (uint32_t i = threadIdx.x; i < uint32_t(kSample); i += kBlock)
    sample[i] = uint64_t(i) * every < R ? keys[i * every] >> key_bits : 0xffffffffu;
  __syncthreads();
  auto lower = [&](uint32_t s) {
    uint32_t a = 0, e = kSample;
    while (a < e) {
      const uint32_t mid = (a + e) >> 1;
      if (sample[mid] < s) a = mid + 1;
      else e = mid;
    }
    // sample[a - 1] < s <= sample[a]
    uint32_t lo = a > 0 ? (a - 1) * every + 1 : 0u, hi = min(uint64_t(a) * every, uint64_t(R));
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (keys[mid] >> key_bits < s) lo = mid + 1;
      else hi = mid;
    }
    return lo;
  };
  uint32_t mx = 0;
  // kBlock - 1 lists per block and step: a list's end is the next thread's start
  constexpr uint32_t kLists = kBlock - 1;
  for (uint32_t b = blockIdx.x * kLists; b <= nseg; b += gridDim.x * kLists) {
    const uint32_t s = b + threadIdx.x;
    const uint32_t lo = s < nseg ? lower(s) : R;
    lows[threadIdx.x] = lo;
    __syncthreads();
    if (threadIdx.x < kLists && s <= nseg) {
      seg_scan[s] = lo;
      if (s < nseg) {
        const uint32_t hi = lows[threadIdx.x + 1];
        mx = max(mx, hi - lo);
        empty(int64_t(hi) + s);
      }
    }
    __syncthreads();
  }
  const uint32_t stride = gridDim.x * kBlock;
  for (uint32_t t = blockIdx.x * kBlock + threadIdx.x; t < uint32_t(kSortedPad); t += stride)
    empty(int64_t(R) + nseg + t);
  mx = __reduce_max_sync(kFullMask, mx);
  if ((threadIdx.x & 31) == 0 && mx) atomicMax(&hdr->max_list, mx);
}

// Sorted replica p of segment s (cell c, type t; s = 3c + t) goes to
// position p + s.
// First-cell bits of a position: bit 0 set if the cell is the box's first cell
// along b, bit 1 if it is its first cell along c. Since the cell coordinate is
// monotone, the cell of a pair's reference point (max of the two minima on b,
// on c) is the max of the two boxes' first cells; both boxes lie in this cell,
// so the reference point is here exactly when, on each of b and c, one of the
// two replicas is its box's first cell.
// scode of a position: its box's y/z interval in the cell and the inverted
// first-cell bits (stq_device.cuh): one integer that the sweep tests against
// the start box's before it loads any bound.
// partner of a position: its first candidate. An edge's candidates are the
// edges after it in its list; a vertex's are the cell's faces whose code is
// >= its code (lower bound), a face's the cell's vertices whose code is > its
// code (upper bound): every V-F pair that can overlap on the sweep axis is found
// once, and vertex-vertex, edge-face and face-face candidates are never tested.
// run_end: one past the last candidate whose code is at most that of the box's
// maximum (or its own, if that is larger: an inverted box still meets the boxes
// of its code). Codes are monotone, so every candidate with a minimum at or
// below the maximum is in the run; those of an equal code that are not are left
// to the exact test.
__global__ void __launch_bounds__(kBlock)
gather_cells_kernel(const stq_aabb *__restrict__ boxes, const uint32_t *__restrict__ keys,
                    const uint32_t *__restrict__ order, const uint32_t *__restrict__ box_q, const BatchHeader *hdr,
                    const unsigned int *__restrict__ cell_base,
                    const SceneRecord *__restrict__ scenes, const uint32_t *__restrict__ seg_scan,
                    SortedScene scene) {
  after_previous();
  const int64_t R = hdr->fault ? 0 : hdr->replicas;  // (none where they are not sorted)
  const int S = hdr->n_scenes;
  const int key_bits = hdr->key_bits;
  for (int64_t p = blockIdx.x * int64_t(kBlock) + threadIdx.x; p < R;
       p += int64_t(gridDim.x) * kBlock) {
    const uint32_t key = keys[p];
    const uint32_t bi = order[p];
    const stq_aabb &x = boxes[bi];
    const uint32_t qmax = (box_q[bi] >> 1) >> (31 - key_bits);  // its leading bits (none where key_bits is 0)
    const unsigned int seg = key >> key_bits;
    const unsigned int cell = seg / 3u, type = seg - 3u * cell;
    int lo = 0, hi = S - 1;  // scene of the cell
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (cell_base[mid] <= cell) lo = mid;
      else hi = mid - 1;
    }
    const GridParams g = scenes[lo].grid;
    int b, c;
    axes_bc(g.axis, b, c);
    const int local = int(cell - cell_base[lo]);
    const int cb = local / g.nc, cc = local - cb * g.nc;
    const int fb = (cell_coord(x.min[b], g.ob, g.ib, g.nb0) >> g.shift) == cb;
    const int fc = (cell_coord(x.min[c], g.oc, g.ic, g.nc0) >> g.shift) == cc;
    const int64_t k = p + seg;
    int64_t first = k + 1;
    // the candidate list: the edge's own list after it, or the other type's
    // list of the cell from the bound search below
    unsigned int cand = seg;
    uint32_t run_a = uint32_t(p) + 1u, run_e = seg_scan[seg + 1];
    const uint32_t q = key - (seg << key_bits);
    if (type != 1u) {
      cand = 3u * cell + (type == 0u ? 2u : 0u);
      const uint32_t want = cand << key_bits | q;
      uint32_t a = seg_scan[cand], e = seg_scan[cand + 1];
      run_e = e;
      while (a < e) {
        const uint32_t mid = (a + e) >> 1;
        const uint32_t mk = keys[mid];
        if (type == 0u ? mk < want : mk <= want) a = mid + 1;
        else e = mid;
      }
      first = int64_t(a) + cand;
      run_a = a;
    }
    // galloping from the run's start, then a bisection
    const uint32_t last = cand << key_bits | max(qmax, q);
    uint32_t a = run_a, step = 8;
    while (a + step <= run_e && keys[a + step - 1] <= last) {
      a += step;
      step <<= 1;
    }
    uint32_t e = min(a + step, run_e);
    while (a < e) {
      const uint32_t mid = (a + e) >> 1;
      if (keys[mid] <= last) a = mid + 1;
      else e = mid;
    }
    scene.yz[k] = make_float4(x.min[b], x.min[c], x.max[b], x.max[c]);
    scene.x[k] = make_float2(x.min[g.axis], x.max[g.axis]);
    scene.v[k] = make_int4(x.vertex_ids[0], x.vertex_ids[1], x.vertex_ids[2], x.id);
    scene.flag[k] = (lo << 2) | (fc << 1) | fb;
    scene.scode[k] = code_pack(code_step(x.min[b], g.ob, g.sb, cb), code_step(x.min[c], g.oc, g.sc, cc),
                               code_step(x.max[b], g.ob, g.sb, cb), code_step(x.max[c], g.oc, g.sc, cc), !fb, !fc);
    scene.partner[k] = int(first);
    scene.run_end[k] = int(int64_t(a) + cand);
  }
}

int blocks_for(int64_t n, int cap = 152 * 16) {
  int64_t g = (n + kBlock - 1) / kBlock;
  return int(g < 1 ? 1 : (g > cap ? cap : g));
}

// Blocks of kBlock threads of a grid-stride kernel over n items: one per
// kBlock items, at most one wave of resident blocks. Every block of a grid-
// stride loop takes the same share, so a grid of 2.7 waves would run its last
// wave on two thirds of the block slots.
int wave_blocks(const void *kernel, int64_t n) {
  static std::mutex m;
  static std::vector<std::pair<const void *, int>> per_sm;  // kernel -> resident blocks per SM
  int resident = 0;
  {
    std::lock_guard<std::mutex> g(m);
    for (const auto &e : per_sm)
      if (e.first == kernel) resident = e.second;
    if (!resident) {
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kernel, kBlock, 0) != cudaSuccess ||
          resident < 1) {
        (void)cudaGetLastError();
        resident = 1;
      }
      per_sm.emplace_back(kernel, resident);
    }
  }
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      sms < 1) {
    (void)cudaGetLastError();
    sms = 152;
  }
  return blocks_for(n, sms * resident);
}

__global__ void __launch_bounds__(kBlock)
reset_sweep_kernel(BatchHeader *hdr, unsigned long long *scene_pairs, const DevScalars *sel, long long capacity) {
  after_previous();
  if (sel && sel->count <= (unsigned long long)capacity) return;
  const int S = hdr->n_scenes;
  for (int s = blockIdx.x * kBlock + threadIdx.x; s < S; s += gridDim.x * kBlock)
    scene_pairs[s] = 0ull;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    hdr->pairs = 0ull;
    hdr->work = 0;
    hdr->long_items = 0u;
    hdr->long_work = 0ull;
    hdr->candidates = 0ull;
  }
}

// After a window of a host-buffer sweep: stores the slot's running pair count
// in page-locked host memory (a kernel store, so that no copy-engine work sits
// between two windows of a stream while the engines move pair lists) and
// restarts the slot's cursors for its next window.
__global__ void window_step_kernel(WindowCounters *wc, unsigned long long *host_count) {
  after_previous();
  if (threadIdx.x != 0) return;
  *reinterpret_cast<volatile unsigned long long *>(host_count) = wc->pairs;
  wc->work = 0;
  wc->long_items = 0u;
  wc->long_work = 0ull;
  __threadfence_system();
}

}  // namespace

cudaError_t launch_window_step(cudaStream_t s, WindowCounters *wc, unsigned long long *host_count) {
  launch_after(window_step_kernel, 1, 32, 0, s, wc, host_count);
  return cudaGetLastError();
}

cudaError_t launch_reset_sweep(cudaStream_t s, BatchHeader *hdr, unsigned long long *scene_pairs,
                               int scene_cap, const DevScalars *sel, long long capacity) {
  launch_after(reset_sweep_kernel, blocks_for(scene_cap, 64), kBlock, 0, s, hdr, scene_pairs, sel, capacity);
  return cudaGetLastError();
}

cudaError_t launch_batch_stats(cudaStream_t s, const BatchBuffers &b) {
  launch_after(batch_stats_kernel, unsigned(b.tile_cap), kBlock, 0, s, b.boxes, b.tiles, b.box_off, b.inputs,
               b.sums, b.scenes, b.hdr);
  return cudaGetLastError();
}

cudaError_t launch_batch_box_keys(cudaStream_t s, const BatchBuffers &b, int64_t rep_cap, int64_t seg_cap, int passes) {
  launch_after(batch_box_keys_kernel, unsigned(b.tile_cap), kBlock, 0, s, b.boxes, b.tiles, b.box_off, b.inputs,
               b.sums, b.scenes, b.cell_base, b.tile_reps, b.tile_off, b.hdr, b.front, rep_cap, seg_cap, passes, b.box_cells,
               b.box_q);
  return cudaGetLastError();
}

cudaError_t launch_batch_emit(cudaStream_t s, const BatchBuffers &b) {
  launch_after(batch_emit_kernel, unsigned(b.tile_cap), kBlock, 0, s, b.boxes, b.box_cells, b.box_q, b.tiles, b.tile_off,
               b.scenes, b.cell_base, b.hdr, b.keys[0], b.keys[1], b.vals[0], b.vals[1]);
  return cudaGetLastError();
}

cudaError_t launch_list_offsets(cudaStream_t s, const uint32_t *keys, BatchHeader *hdr, uint32_t *seg_scan,
                                int64_t seg_cap, const SortedScene &scene, int64_t slots_cap, int64_t lists) {
  launch_after(list_offsets_kernel, blocks_for((lists + 1) / (kBlock - 1) * kBlock + kBlock), kBlock, 0, s, keys,
               hdr, seg_scan, seg_cap, scene, slots_cap);
  return cudaGetLastError();
}

cudaError_t launch_gather_cells(cudaStream_t s, const BatchBuffers &b, int64_t replicas, const SortedScene &scene) {
  launch_after(gather_cells_kernel, wave_blocks((const void *)gather_cells_kernel, replicas), kBlock, 0, s, b.boxes,
               b.keys[0], b.vals[0], b.box_q, b.hdr, b.cell_base, b.scenes, b.seg_scan, scene);
  return cudaGetLastError();
}

}  // namespace stq
