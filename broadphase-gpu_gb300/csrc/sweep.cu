// sweep.cu - the sweep-and-tiniest-queue pass, pair compaction, the
// overflow prefix selection and the all-pairs checker.
//
// Reference: twostage_queue (src/sweep.cu:226-279) with its shared Queue
// (src/queue.cuh:9-38, src/queue.cu:75-115), does_collide / covertex /
// is_valid_pair (src/collision.cu:38-48, src/aabb.cu:33-40) and add_overlap
// (src/collision.cu:50-74).
//
// GB300 design. A start box k's candidates are its run [partner[k], run_end[k])
// of one list, found by the gather: the edges after it for an edge, the faces (for
// a vertex) or vertices (for a face) of the same cell. A run holds every
// candidate that can overlap on the sweep axis, and a few that do not (those of
// an equal sweep-axis code); a candidate's position code is tested first, then
// the pair exactly. Two shapes walk the runs:
//   - queue (stq_sweep_lane_kernel, stq_sweep_kernel): each warp owns a
//     shared-memory ring of pending start boxes (the "tiniest queue"); a lane,
//     or a group of G lanes, takes one start box from the ring and walks its
//     run, and takes the next pending box when the run ends, so a long run
//     never stalls the others;
//   - flat (stq_sweep_flat_kernel, the default): a warp takes the runs of 32
//     consecutive start positions together.
// Runs longer than a cap go to a warp pass (the flat kernel over a list). Refill,
// hand-out and pair output use __ballot_sync/__popc compaction: no
// shared-memory atomics, and one global atomic per 32 or more pairs.
#include <algorithm>
#include <map>
#include <mutex>
#include <type_traits>
#include <utility>

#include "stq_device.cuh"
#include "stq_internal.h"

namespace stq {

namespace {

__device__ __forceinline__ PosRec load_pos(const SweepParams &p, int j) { return PosRec{p.yz[j], p.x[j], p.v[j]}; }

// The exact test of a pair that passed the filter: overlap on the non-sweep
// axes and on the sweep axis (the box with the smaller minimum reaches the other's
// minimum; on ties the start box a goes first), is_valid_pair where the lists
// mix types, and covertex.
__device__ __forceinline__ bool pair_hit(const PosRec &a, const PosRec &b, int typed) {
  const bool x = b.x.x >= a.x.x ? b.x.x <= a.x.y : a.x.x <= b.x.y;
  return x && overlap_bc(a.yz, b.yz) && (typed || valid_pair(a.v, b.v)) && !covertex(a.v, b.v);
}

// One past the last start position of a sweep, from the sizes on the device (none
// if a wait of the sort ran out: there is no sorted scene then).
__device__ __forceinline__ int sweep_end(const SweepParams &p) {
  const int end = p.hdr->fault ? p.begin : min(p.end, int(p.hdr->length));
  if (!p.sel) return end;
  return p.sel->count <= (unsigned long long)p.capacity ? p.begin : int(min((long long)end, p.begin + p.sel->prefix));
}

// Start positions per grab of a sweep over `span` of them.
__device__ __forceinline__ int sweep_chunk(const SweepParams &p, int span) {
  return p.grabs ? max(32, min(p.chunk, (span / p.grabs + 31) / 32 * 32)) : p.chunk;
}

// Appends the warp's n staged pairs with one atomic; pairs past the capacity
// are counted but not written.
__device__ __forceinline__ void flush_staged(const int2 *st, int n, int lane, const SweepParams &p) {
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(p.count, (unsigned long long)n);
  base = __shfl_sync(kFullMask, base, 0);
  int2 *out = reinterpret_cast<int2 *>(p.pairs);
  for (int i = lane; i < n; i += 32)
    if (base + i < (unsigned long long)p.capacity) out[base + i] = st[i];
  __syncwarp();
}

template <int G, int Q, int BLOCK>
__global__ void __launch_bounds__(BLOCK)
stq_sweep_kernel(const SweepParams p) {
  after_previous();
  static_assert(32 % G == 0, "lane group must divide the warp");
  // the refill tops the ring up to one entry per group: Q >= 32 / G
  static_assert((Q & (Q - 1)) == 0 && Q >= 16 && Q >= 32 / G, "queue depth: power of two >= 16 and >= groups");
  constexpr int E = 32 / G;  // lane groups per warp
  constexpr int STAGE = 64;  // pairs staged per warp before one global append
  __shared__ int ring[BLOCK / 32][Q];
  __shared__ int2 stage[BLOCK / 32][STAGE];

  const int lane = threadIdx.x & 31;
  const int gl = lane % G;              // lane within group
  const int grp = lane / G;             // group within warp
  const unsigned grp_mask = G == 32 ? kFullMask : (((1u << G) - 1u) << (grp * G));
  const unsigned leaders_below = (grp * G) == 0 ? 0u : ((1u << (grp * G)) - 1u);
  int *q = ring[threadIdx.x >> 5];

  // warp-uniform queue and work state
  int qhead = 0, qsize = 0;
  int next_k = 0, chunk_end = 0;
  bool more = true;
  // lane-group state (identical in the G lanes of a group)
  int k = -1, j0 = 0, taken = 0;
  int jend = 0;       // one past the run of the current start box
  PosRec kr = {};     // the current start box
  uint32_t code = 0;  // and its code
  int kf = 0;         // its scene, above the first-cell bits
  const int end = sweep_end(p);
  const int span = end - p.begin, chunk = sweep_chunk(p, span);
  unsigned tested = 0;  // candidates this lane tested (statistics)
  // warp-uniform: staged pairs, and pairs of the current scene not yet added
  // to its counter
  int staged = 0;
  int wscene = 0;
  unsigned long long wpairs = 0;
  const bool multi = p.hdr->n_scenes > 1;  // per-scene counts need the scene of each hit
  int2 *st = stage[threadIdx.x >> 5];

  while (true) {
    // 1. Refill the ring with start boxes that have at least one candidate.
    while (qsize < E && more) {
      if (next_k >= chunk_end) {
        int c = 0;
        if (lane == 0) c = atomicAdd(p.work, chunk);
        c = __shfl_sync(kFullMask, c, 0);
        if (c >= span) {
          more = false;
          break;
        }
        next_k = p.begin + c;
        chunk_end = min(next_k + chunk, end);
      }
      const int take = min(32, min(Q - qsize, chunk_end - next_k));
      const int kk = next_k + lane;
      bool push = false;
      if (lane < take) push = p.partner[kk] < p.run_end[kk];
      const unsigned m = __ballot_sync(kFullMask, push);
      if (push) q[(qhead + qsize + __popc(m & lanemask_lt())) & (Q - 1)] = kk;
      qsize += __popc(m);
      next_k += take;
    }
    __syncwarp();
    // 2. Idle groups take pending start boxes, in ring order.
    const bool idle = k < 0;
    const unsigned needm = __ballot_sync(kFullMask, idle && gl == 0);
    const int ntake = min(__popc(needm), qsize);
    if (idle) {
      const int r = __popc(needm & leaders_below);
      if (r < ntake) {
        k = q[(qhead + r) & (Q - 1)];
        j0 = p.partner[k];
        jend = p.run_end[k];
        kr = load_pos(p, k);
        code = code_start(p.scode[k]);
        kf = multi ? p.flag[k] : 0;
        taken = 0;
      }
    }
    qhead = (qhead + ntake) & (Q - 1);
    qsize -= ntake;
    __syncwarp();
    const bool active = k >= 0;
    if (__ballot_sync(kFullMask, active) == 0) {
      if (!more && qsize == 0) break;
      continue;
    }
    // 3. Test G consecutive candidates per group: those before the run's end,
    //    by their codes, then exactly.
    const int j = j0 + gl;
    const bool valid = active && j < jend;
    bool hit = false;
    int lo_id = 0, hi_id = 0;
    if (valid) {
      ++tested;
      if (code_pass(code, p.scode[j])) {
        const PosRec c = load_pos(p, j);
        hit = pair_hit(kr, c, p.typed);
        lo_id = min(kr.v.w, c.v.w);
        hi_id = max(kr.v.w, c.v.w);
      }
    }
    // 4. Emit: compact the step's hits into the warp's staging buffer; append
    //    it to the pair list with one global atomic per 32 or more pairs.
    const unsigned hm = __ballot_sync(kFullMask, hit);
    const int ghits = __popc(hm & grp_mask);
    if (hm) {
      if (hit) st[staged + __popc(hm & lanemask_lt())] = make_int2(lo_id, hi_id);
      staged += __popc(hm);
      // per-scene counts: one register while the warp stays in one scene
      if (!multi) {
        wpairs += __popc(hm);
      } else {
        const int lead = __shfl_sync(kFullMask, kf >> 2, __ffs(hm) - 1);
        if (__all_sync(kFullMask, !hit || (kf >> 2) == lead)) {
          if (lead != wscene) {
            if (lane == 0 && wpairs) atomicAdd(&p.scene_pairs[wscene], wpairs);
            wscene = lead;
            wpairs = 0;
          }
          wpairs += __popc(hm);
        } else if (gl == 0 && ghits) {
          atomicAdd(&p.scene_pairs[kf >> 2], (unsigned long long)ghits);
        }
      }
      if (staged >= 32) {
        __syncwarp();
        flush_staged(st, staged, lane, p);
        staged = 0;
      }
    }
    // 5. A group whose G lanes all passed continues; otherwise its run ended.
    const unsigned vm = __ballot_sync(kFullMask, valid);
    if (active) {
      if ((vm & grp_mask) == grp_mask) {
        j0 += G;
        taken += G;
        if (p.run_cap && taken >= p.run_cap) {  // a long run: the warp pass takes the rest
          if (gl == 0) {
            p.long_list[atomicAdd(p.long_items, 1u)] = make_int2(k, j0);
          }
          k = -1;
        }
      } else {
        k = -1;
      }
    }
  }
  __syncwarp();
  if (staged) flush_staged(st, staged, lane, p);
  if (lane == 0 && wpairs) atomicAdd(&p.scene_pairs[wscene], wpairs);
  const unsigned t = __reduce_add_sync(kFullMask, tested);
  if (lane == 0 && p.stats) atomicAdd(p.stats, (unsigned long long)t);
}

// One start box per lane. A lane walks its own run, U consecutive candidates
// per step: the U codes are loaded together (U independent loads in flight per
// lane), and a lane whose run ended takes the next pending box from the warp's
// ring. Otherwise as stq_sweep_kernel: ring refill by ballot compaction, per-warp
// staging of pairs.
template <int U, int Q, int BLOCK>
__global__ void __launch_bounds__(BLOCK)
stq_sweep_lane_kernel(const SweepParams p) {
  after_previous();
  static_assert(U == 1 || U == 2 || U == 4 || U == 8, "candidates per lane step: 1, 2, 4 or 8");
  static_assert((Q & (Q - 1)) == 0 && Q >= 32, "queue depth: power of two >= 32");
  constexpr int STAGE = 32 * (U + 1);  // < 32 left over + at most 32 * U new pairs
  // A ring entry carries the partner the refill read for its start box, so a
  // take starts the candidate loads without a dependent global load; where
  // that would pass 48 KB of shared memory the entry is the start box alone.
  constexpr bool kWide = (BLOCK / 32) * (Q * 8 + STAGE * 8) <= 48 * 1024;
  using Entry = typename std::conditional<kWide, int2, int>::type;
  __shared__ Entry ring[BLOCK / 32][Q];
  __shared__ int2 stage[BLOCK / 32][STAGE];

  const int lane = threadIdx.x & 31;
  const unsigned below = lanemask_lt();
  Entry *q = ring[threadIdx.x >> 5];
  int2 *st = stage[threadIdx.x >> 5];

  int qhead = 0, qsize = 0;
  int next_k = 0, chunk_end = 0;
  bool more = true;
  int k = -1, j = 0, jend = 0, taken = 0;
  PosRec kr = {};     // the start box
  uint32_t code = 0;  // and its code
  int kf = 0;         // its scene, above the first-cell bits
  const int end = sweep_end(p);
  const int span = end - p.begin, chunk = sweep_chunk(p, span);
  unsigned tested = 0;
  int staged = 0;
  int wscene = 0;
  unsigned long long wpairs = 0;
  const bool multi = p.hdr->n_scenes > 1;

  while (true) {
    // 1. Refill the ring with start boxes that have at least one candidate.
    while (qsize < 32 && more) {
      if (next_k >= chunk_end) {
        int c = 0;
        if (lane == 0) c = atomicAdd(p.work, chunk);
        c = __shfl_sync(kFullMask, c, 0);
        if (c >= span) {
          more = false;
          break;
        }
        next_k = p.begin + c;
        chunk_end = min(next_k + chunk, end);
      }
      const int take = min(32, min(Q - qsize, chunk_end - next_k));
      const int kk = next_k + lane;
      bool push = false;
      int pk = 0;
      if (lane < take) {
        pk = p.partner[kk];
        push = pk < p.run_end[kk];
      }
      const unsigned m = __ballot_sync(kFullMask, push);
      if (push) {
        Entry &slot = q[(qhead + qsize + __popc(m & below)) & (Q - 1)];
        if constexpr (kWide) slot = make_int2(kk, pk);
        else slot = kk;
      }
      qsize += __popc(m);
      next_k += take;
    }
    __syncwarp();
    // 2. Idle lanes take pending start boxes, in ring order.
    const unsigned needm = __ballot_sync(kFullMask, k < 0);
    const int ntake = min(__popc(needm), qsize);
    if (k < 0) {
      const int r = __popc(needm & below);
      if (r < ntake) {
        const Entry e = q[(qhead + r) & (Q - 1)];
        if constexpr (kWide) {
          k = e.x;
          j = e.y;
        } else {
          k = e;
          j = p.partner[k];
        }
        jend = p.run_end[k];
        kr = load_pos(p, k);
        code = code_start(p.scode[k]);
        kf = multi ? p.flag[k] : 0;
        taken = 0;
      }
    }
    qhead = (qhead + ntake) & (Q - 1);
    qsize -= ntake;
    __syncwarp();
    const bool active = k >= 0;
    if (__ballot_sync(kFullMask, active) == 0) {
      if (!more && qsize == 0) break;
      continue;
    }
    // 3. U candidates of the lane's run (their codes are loaded together), by
    //    their codes, then exactly. Hits as bits; a hit's id is loaded again on
    //    output (an L1 hit) rather than kept in registers for the whole step.
    const int nvalid = active ? min(U, jend - j) : 0;
    uint32_t cc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) cc[u] = u < nvalid ? p.scode[j + u] : 0u;
    tested += unsigned(nvalid);
    unsigned hits = 0;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u < nvalid && code_pass(code, cc[u]) && pair_hit(kr, load_pos(p, j + u), p.typed)) hits |= 1u << u;
    // 4. Emit the step's hits through the warp's staging buffer.
    const int nh = __popc(hits);
    const unsigned anym = __ballot_sync(kFullMask, nh > 0);
    if (anym) {
      int total = 0;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool hit = (hits >> u) & 1u;
        const unsigned hm = __ballot_sync(kFullMask, hit);
        if (hit) {
          const int id = p.v[j + u].w;
          st[staged + __popc(hm & below)] = make_int2(min(kr.v.w, id), max(kr.v.w, id));
        }
        staged += __popc(hm);
        total += __popc(hm);
      }
      // per-scene counts: one register while the warp stays in one scene
      if (!multi) {
        wpairs += unsigned(total);
      } else {
        const int lead = __shfl_sync(kFullMask, kf >> 2, __ffs(anym) - 1);
        if (__all_sync(kFullMask, nh == 0 || (kf >> 2) == lead)) {
          if (lead != wscene) {
            if (lane == 0 && wpairs) atomicAdd(&p.scene_pairs[wscene], wpairs);
            wscene = lead;
            wpairs = 0;
          }
          wpairs += unsigned(total);
        } else if (nh) {
          atomicAdd(&p.scene_pairs[kf >> 2], (unsigned long long)nh);
        }
      }
      if (staged >= 32) {
        __syncwarp();
        flush_staged(st, staged, lane, p);
        staged = 0;
      }
    }
    // 5. A lane whose U candidates all passed continues; otherwise its run ended.
    if (active) {
      if (nvalid == U) {
        j += U;
        taken += U;
        if (p.run_cap && taken >= p.run_cap) {  // a long run: the warp pass takes the rest
          p.long_list[atomicAdd(p.long_items, 1u)] = make_int2(k, j);
          k = -1;
        }
      } else {
        k = -1;
      }
    }
  }
  __syncwarp();
  if (staged) flush_staged(st, staged, lane, p);
  if (lane == 0 && wpairs) atomicAdd(&p.scene_pairs[wscene], wpairs);
  const unsigned t = __reduce_add_sync(kFullMask, tested);
  if (lane == 0 && p.stats) atomicAdd(p.stats, (unsigned long long)t);
}

// Flat shape. A warp takes 32 consecutive start positions; each one's run on
// the sweep axis is [partner, run_end), both found by the gather (runs longer
// than run_cap are cut there and the rest goes to the warp pass).
//
// The filter compares position codes (stq_device.cuh): one integer per
// candidate and one per start box, a subtraction and a test for the y/z
// overlap and the first-cell rule. It has two forms, chosen for each 32 starts:
//   - band: the starts' runs lie in one window of positions. One start per
//     lane, the window's codes 32 at a time through shared memory, every lane
//     tests all 32 (three integer instructions each) and keeps the bits inside
//     its own run. The cost goes with the window, whatever the runs cover of it.
//   - flat: the runs are laid end to end and the warp takes 32 candidates per
//     step, one per lane: lane l of the step at `base` takes flat candidate
//     base + l, whose start is the last one whose run begins at or before it (a
//     bit mask of the run beginnings inside the step, one OR-reduction, and a
//     population count). The cost goes with the candidates.
// Candidates that pass are queued in shared memory (start slot and offset in
// its run), and taken 32 at a time, one per lane, for the exact y/z test, the
// vertex ids, is_valid_pair and covertex. The hits go through the staging
// buffer. The starts' records sit in shared memory, so the queue is drained
// before the next 32 starts replace them.
//
// LONG: the warp pass over the runs that were handed over (longer than run_cap,
// which would keep one lane, group or warp busy long after the others finished).
// The warp's starts are entries of that list, and when there are fewer of them
// than warps each run is cut into as many equal parts as give every warp one; at
// least into as many as keep a part within kLongPart candidates, so that the warp's
// 32 together are within 31 bits, and an offset in a part within the queue's 27.
struct FlatStart {
  float4 yz;      // the start box (PosRec)
  int4 v;
  float2 x;
  int kf;         // first-cell bits and scene
  int j;          // first position of its run
};
static_assert(sizeof(FlatStart) == 48, "FlatStart: three 16-byte words");

// Band or flat: a band step takes some 500 instructions for 32 positions, 130 of
// them the filter, and a flat step some 30 for its 32 candidates. The time is
// level between 3 and 8 candidates per position of the window (within 2% on the
// 6 M-box scene, where 98% of the candidates are in bands); without bands that
// sweep takes 18% longer.
constexpr int kBandRatio = 6;
// Pairs staged per warp, appended with one atomic on the pair counter once
// fewer than 32 places are left. All warps share that counter: on the 6 M-box
// scene (92 M pairs) 64 places took 1.61 ms, 128 1.16, 192 1.12; larger stages
// take resident blocks away (384: 1.20, 768: 1.38 ms).
constexpr int kFlatStage = 192;
constexpr int kFlatRound = 256;  // candidates queued at once by a band step (or 32 V by a flat one)
constexpr int kFlatQueue = 32 + kFlatRound;
constexpr unsigned kLongPart = 1u << 25;
struct FlatWarp {
  FlatStart rec[32];
  int2 lookup[32];             // flat form: code_start of a start's code, and joff: its
                               // run's flat candidate f is at position joff + f
  int2 stage[kFlatStage];
  uint32_t queue[kFlatQueue];  // slot | offset in the run << 5 (run_cap < 2^27)
  uint4 code[8];               // a band step's 32 candidate codes
  int hits[32];                // count mode: pairs per slot
};

template <int BLOCK, int V, SweepMode MODE, bool LONG>
__global__ void __launch_bounds__(BLOCK)
stq_sweep_flat_kernel(const SweepParams p) {
  after_previous();
  static_assert(32 * V <= kFlatRound, "queue holds a flat round");
  constexpr bool COUNT = MODE != kSweepEmit, EMIT = MODE != kSweepCount;
  extern __shared__ __align__(16) unsigned char flat_smem[];
  FlatWarp &sw = reinterpret_cast<FlatWarp *>(flat_smem)[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const unsigned below = lanemask_lt();
  const unsigned upto = below | (1u << lane);
  FlatStart *rec = sw.rec;
  int2 *st = sw.stage;
  uint32_t *qu = sw.queue;

  using Index = typename std::conditional<LONG, long long, int>::type;  // a part of a run, or a start position
  Index end, span;
  int chunk;
  unsigned parts = 1;  // LONG: parts of a run
  if (LONG) {
    if (p.sel && p.sel->count <= (unsigned long long)p.capacity) return;  // the list is of an earlier sweep
    const unsigned items = *p.long_items, warps = gridDim.x * (BLOCK / 32);
    if (items == 0) return;
    parts = max(max(1u, min(64u, warps / items)), (p.hdr->length + kLongPart - 1u) / kLongPart);
    end = span = Index(items) * parts;
    chunk = int(max(Index(1), min(Index(32), span / Index(4 * warps))));
  } else {
    end = sweep_end(p);
    span = end - p.begin;
    chunk = sweep_chunk(p, span);
  }
  const Index first = LONG ? 0 : p.begin;
  const bool multi = p.hdr->n_scenes > 1;
  Index next_k = 0, chunk_end = 0;
  unsigned long long tested = 0;  // warp-uniform
  int staged = 0, queued = 0;
  int wscene = 0;
  unsigned long long wpairs = 0;

  while (true) {
    if (next_k >= chunk_end) {
      Index c = 0;
      if constexpr (LONG) {
        if (lane == 0) c = Index(atomicAdd(p.long_work, (unsigned long long)chunk));
      } else {
        if (lane == 0) c = atomicAdd(p.work, chunk);
      }
      c = __shfl_sync(kFullMask, c, 0);
      if (c >= span) break;
      next_k = first + c;
      chunk_end = min(next_k + chunk, end);
    }
    const int take = int(min(Index(32), chunk_end - next_k));
    const Index at_k = next_k + lane;
    next_k += take;
    // 1. Runs (that of the position after a list is empty).
    int k = int(at_k), len = 0, j = 0;
    if constexpr (LONG) {
      if (lane < take) {
        const unsigned item = span >> 32 ? unsigned(at_k / parts) : unsigned(at_k) / parts;
        const int part = int(at_k - Index(item) * parts);
        const int2 it = p.long_list[item];
        const int run_end = p.run_end[it.x];
        const int each = int((unsigned(run_end - it.y) + parts - 1u) / parts);
        k = it.x;
        j = it.y + part * each;
        len = max(min(each, run_end - j), 0);
      }
    } else if (lane < take) {
      j = p.partner[k];
      len = max(p.run_end[k] - j, 0);
      if (p.run_cap && len > p.run_cap) {  // a long run: the warp pass takes the rest
        p.long_list[atomicAdd(p.long_items, 1u)] = make_int2(k, j + p.run_cap);
        len = p.run_cap;
      }
    }
    const unsigned nz = __ballot_sync(kFullMask, len > 0);
    if (nz == 0) continue;
    // 2. Exclusive prefix of the lengths; the starts with candidates keep their
    //    records in shared memory, in lane order.
    int incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(kFullMask, incl, o);
      if (lane >= o) incl += v;
    }
    const int excl = incl - len;
    const int total = __shfl_sync(kFullMask, incl, 31);
    const int slot = __popc(nz & below);
    uint32_t code = 0;
    if (len > 0) {
      FlatStart r;
      r.yz = p.yz[k];
      r.x = p.x[k];
      r.v = p.v[k];
      r.kf = multi ? p.flag[k] : 0;
      code = code_start(p.scode[k]);
      r.j = j;
      rec[slot] = r;
      sw.lookup[slot] = make_int2(int(code), j - excl);
    }
    if (COUNT) sw.hits[lane] = 0;
    tested += unsigned(total);
    const int jlo = __reduce_min_sync(kFullMask, len > 0 ? j : 0x7fffffff);
    const int jhi = __reduce_max_sync(kFullMask, len > 0 ? j + len : 0);
    __syncwarp();
    const bool band = jhi - jlo <= total / kBandRatio;
    const unsigned my_begin = len > 0 ? unsigned(excl) : 0xffffffffu;
    int at = band ? jlo : 0;  // next position (band) or flat candidate
    const int stop = band ? jhi : total;
    int begun = 0;      // flat: starts whose run began before the current step
    int lo = 0;         // band: the lane's run begins lo positions into the step
    uint32_t ahead = band ? p.scode[at + lane] : 0u;  // band: the next step's codes
    uint32_t hits = 0;  // band: candidates of the step that are not queued yet,
    uint32_t part = 0;  // and those of them that go next
    bool more;
    do {
      if (band) {
        // 3a. The band: 32 positions of the window per step.
        if (part == 0u) {
          lo = j - at;
          const int hi = lo + len;
          uint32_t mine = 0;  // positions of this step inside the lane's run
          if (len > 0 && lo < 32 && hi > 0)
            mine = (kFullMask << max(lo, 0)) & (hi >= 32 ? kFullMask : ~(kFullMask << hi));
          reinterpret_cast<uint32_t *>(sw.code)[lane] = ahead;
          __syncwarp();
          at += 32;
          // the next step's, loaded while this one is taken (6 M boxes: sweep 1.27 ms
          // without, 1.25 with)
          if (at < stop) ahead = p.scode[at + lane];
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const uint4 c = sw.code[q];
            if (code_pass(code, c.x)) hits |= 1u << (4 * q);
            if (code_pass(code, c.y)) hits |= 2u << (4 * q);
            if (code_pass(code, c.z)) hits |= 4u << (4 * q);
            if (code_pass(code, c.w)) hits |= 8u << (4 * q);
          }
          hits &= mine;
          // more than the queue holds go 8 positions (at most 256) at a time
          part = __reduce_add_sync(kFullMask, __popc(hits)) <= unsigned(kFlatRound) ? kFullMask : 0xffu;
        }
        uint32_t h = hits & part;
        hits ^= h;
        part <<= 8;
        if (part == kFullMask << 8) part = 0u;  // all of them went
        // places by a prefix sum of the lanes' counts
        const int count = __popc(h);
        int to = count;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(kFullMask, to, o);
          if (lane >= o) to += v;
        }
        const int all = __shfl_sync(kFullMask, to, 31);
        to += queued - count;
        while (h) {
          const int c = __ffs(h) - 1;
          h &= h - 1u;
          qu[to++] = unsigned(slot) | unsigned(c - lo) << 5;
        }
        queued += all;
      } else {
        // 3b. Flat: V steps of 32 candidates at a time. A run that begins inside
        //     the step at `at` marks bit (excl - at).
        int si[V], rel[V];
        uint32_t sc[V], cc[V];
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const unsigned d = my_begin - unsigned(at + 32 * v);
          const unsigned heads = __reduce_or_sync(kFullMask, d < 32u ? (1u << d) : 0u);
          si[v] = begun + __popc(heads & upto) - 1;
          begun += __popc(heads);
          const int f = at + 32 * v + lane;
          const int2 r = sw.lookup[si[v]];
          const int jj = r.y + f;
          sc[v] = uint32_t(r.x);
          rel[v] = f < total ? jj - rec[si[v]].j : -1;
          cc[v] = f < total ? p.scode[jj] : 0u;
        }
        at += 32 * V;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const bool pass = rel[v] >= 0 && code_pass(sc[v], cc[v]);
          const unsigned pm = __ballot_sync(kFullMask, pass);
          if (pass) qu[queued + __popc(pm & below)] = unsigned(si[v]) | unsigned(rel[v]) << 5;
          queued += __popc(pm);
        }
      }
      __syncwarp();
      more = at < stop || part != 0u;
      // 4. The check of the last queued candidates, one per lane (idle lanes
      //    take a queued one again).
      while (queued >= 32 || (!more && queued > 0)) {
        const int n = min(queued, 32);
        const uint32_t e = qu[queued - 1 - (lane < n ? lane : 0)];
        queued -= n;
        const FlatStart &r = rec[e & 31u];
        const int c = r.j + int(e >> 5);
        const float4 b = p.yz[c];
        const int4 bv = p.v[c];
        const int4 kv = r.v;
        const bool hit = lane < n && pair_hit(PosRec{r.yz, r.x, kv}, PosRec{b, p.x[c], bv}, p.typed);
        if (COUNT && hit) atomicAdd(&sw.hits[e & 31u], 1);
        if (EMIT) {
          const unsigned hm = __ballot_sync(kFullMask, hit);
          if (hit) st[staged + __popc(hm & below)] = make_int2(min(kv.w, bv.w), max(kv.w, bv.w));
          staged += __popc(hm);
          if (!multi) {
            wpairs += __popc(hm);
          } else if (hm) {
            const int kf = r.kf;
            const int lead = __shfl_sync(kFullMask, kf >> 2, __ffs(hm) - 1);
            if (__all_sync(kFullMask, !hit || (kf >> 2) == lead)) {
              if (lead != wscene) {
                if (lane == 0 && wpairs) atomicAdd(&p.scene_pairs[wscene], wpairs);
                wscene = lead;
                wpairs = 0;
              }
              wpairs += __popc(hm);
            } else if (hit) {
              atomicAdd(&p.scene_pairs[kf >> 2], 1ull);
            }
          }
          if (staged > kFlatStage - 32) {
            __syncwarp();
            flush_staged(st, staged, lane, p);
            staged = 0;
          }
        }
        __syncwarp();
      }
    } while (more);
    if (COUNT) {
      if (len > 0) {
        if (LONG) atomicAdd(&p.box_counts[k - p.begin], sw.hits[slot]);
        else p.box_counts[k - p.begin] = sw.hits[slot];
      }
      __syncwarp();
    }
  }
  if (!EMIT) return;
  __syncwarp();
  if (staged) flush_staged(st, staged, lane, p);
  if (lane == 0 && wpairs) atomicAdd(&p.scene_pairs[wscene], wpairs);
  if (lane == 0 && p.stats) atomicAdd(p.stats, tested);
}

// Resident blocks per SM of a sweep kernel, queried once per kernel and
// device: the query costs host time on every launch otherwise, and the host
// calls launch one sweep per window back to back.
template <typename Kern>
cudaError_t resident_blocks(Kern kern, int block, size_t smem, int *per_sm) {
  static std::mutex mu;
  static std::map<std::pair<const void *, int>, int> known;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const auto key = std::make_pair(reinterpret_cast<const void *>(kern), dev);
  std::lock_guard<std::mutex> lock(mu);
  auto it = known.find(key);
  if (it == known.end()) {
    int v = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, kern, block, smem);
    if (e != cudaSuccess) return e;
    it = known.emplace(key, v).first;
  }
  *per_sm = it->second;
  return cudaSuccess;
}

template <typename Kern>
cudaError_t launch_persistent(Kern kern, int block, cudaStream_t s, const SweepParams &p, int num_sms,
                              size_t smem = 0) {
  int per_sm = 0;
  cudaError_t e = resident_blocks(kern, block, smem, &per_sm);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) per_sm = 1;
  // persistent grid: all resident blocks, capped by the available work
  const int64_t chunk = p.grabs ? std::min(p.chunk, 32) : p.chunk;
  const int64_t warps_needed = (int64_t(p.end) - p.begin + chunk - 1) / chunk;
  int64_t blocks = int64_t(num_sms) * per_sm;
  const int64_t max_useful = (warps_needed + block / 32 - 1) / (block / 32);
  if (blocks > max_useful) blocks = max_useful;
  if (blocks < 1) blocks = 1;
  launch_after(kern, unsigned(blocks), block, smem, s, p);
  return cudaGetLastError();
}

template <int G, int Q, int BLOCK>
cudaError_t launch_variant(cudaStream_t s, const SweepParams &p, int num_sms) {
  return launch_persistent(stq_sweep_kernel<G, Q, BLOCK>, BLOCK, s, p, num_sms);
}

template <int G, int Q>
cudaError_t launch_gq(cudaStream_t s, const SweepParams &p, int block, int sms) {
  switch (block) {
    case 128: return launch_variant<G, Q, 128>(s, p, sms);
    case 512: return launch_variant<G, Q, 512>(s, p, sms);
    default: return launch_variant<G, Q, 256>(s, p, sms);
  }
}

template <int G>
cudaError_t launch_g(cudaStream_t s, const SweepParams &p, const SweepTuning &t, int sms) {
  switch (t.queue) {
    case 16:  // at least one entry per lane group
      if constexpr (G >= 2) return launch_gq<G, 16>(s, p, t.block, sms);
      else return launch_gq<G, 32>(s, p, t.block, sms);
    case 32: return launch_gq<G, 32>(s, p, t.block, sms);
    case 128: return launch_gq<G, 128>(s, p, t.block, sms);
    default: return launch_gq<G, 64>(s, p, t.block, sms);
  }
}

template <int U, int Q>
cudaError_t launch_uq(cudaStream_t s, const SweepParams &p, int block, int sms) {
  switch (block) {
    case 128: return launch_persistent(stq_sweep_lane_kernel<U, Q, 128>, 128, s, p, sms);
    case 512: return launch_persistent(stq_sweep_lane_kernel<U, Q, 512>, 512, s, p, sms);
    default: return launch_persistent(stq_sweep_lane_kernel<U, Q, 256>, 256, s, p, sms);
  }
}

template <int U>
cudaError_t launch_u(cudaStream_t s, const SweepParams &p, const SweepTuning &t, int sms) {
  switch (t.queue) {
    case 16:  // one start box per lane refills to 32 entries: the ring holds at least 32
    case 32: return launch_uq<U, 32>(s, p, t.block, sms);
    case 128: return launch_uq<U, 128>(s, p, t.block, sms);
    default: return launch_uq<U, 64>(s, p, t.block, sms);
  }
}

// The flat shape's blocks are 128 or 256 threads.
template <int BLOCK, int V, SweepMode MODE>
cudaError_t launch_flat_block(cudaStream_t s, const SweepParams &p, int sms) {
  constexpr auto kern = stq_sweep_flat_kernel<BLOCK, V, MODE, false>;
  constexpr size_t smem = sizeof(FlatWarp) * (BLOCK / 32);
  cudaError_t e = allow_smem<kern>(smem);
  if (e != cudaSuccess) return e;
  return launch_persistent(kern, BLOCK, s, p, sms, smem);
}

// The warp pass: four blocks per SM (most sweeps hand nothing over, and the
// blocks leave at once).
template <SweepMode MODE>
cudaError_t launch_long_runs(cudaStream_t s, const SweepParams &p, int sms) {
  constexpr auto kern = stq_sweep_flat_kernel<256, 4, MODE, true>;
  constexpr size_t smem = sizeof(FlatWarp) * 8;
  cudaError_t e = allow_smem<kern>(smem);
  if (e != cudaSuccess) return e;
  launch_after(kern, unsigned(sms * 4), 256, smem, s, p);
  return cudaGetLastError();
}

template <int V>
cudaError_t launch_flat(cudaStream_t s, const SweepParams &p, int block, int sms) {
  if (block == 128) return launch_flat_block<128, V, kSweepEmit>(s, p, sms);
  return launch_flat_block<256, V, kSweepEmit>(s, p, sms);
}

// ---- overflow: longest prefix of start boxes whose pairs fit ------------------
constexpr int kScanBlock = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanBlock * kScanItems;

// Tile sums, then, in the last block to finish, the last tile whose pairs before
// it are within the capacity and, in that tile, the longest prefix whose pairs
// are. Both searches are scans by the whole block: with one thread each they took
// 180 us for the 1.4 M start positions of a 684,000-box scene, as long as the
// sweeps around them.
struct PrefixDone {
  unsigned int blocks;  // zero before the launch
};

// Inclusive scan of one value per thread of the block.
__device__ __forceinline__ long long block_inclusive(long long v, long long *scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(kFullMask, v, o);
    if (lane >= o) v += y;
  }
  __syncthreads();  // scratch may be in use
  if (lane == 31) scratch[warp] = v;
  __syncthreads();
  for (int w = 0; w < warp; ++w) v += scratch[w];
  return v;
}

__global__ void __launch_bounds__(kScanBlock)
prefix_select_kernel(const int32_t *__restrict__ c, int64_t m, long long capacity, long long *__restrict__ sums,
                     int64_t ntiles, PrefixDone *done, DevScalars *scalars, const unsigned long long *found) {
  after_previous();
  __shared__ long long scratch[kScanBlock / 32];
  __shared__ long long at[2];  // the selected tile and the pairs before it
  __shared__ bool last;
  const int64_t base = int64_t(blockIdx.x) * kScanTile;
  long long s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    const int64_t idx = base + int64_t(i) * kScanBlock + threadIdx.x;
    if (idx < m) s += c[idx];
  }
  const long long total = block_inclusive(s, scratch);
  if (threadIdx.x == kScanBlock - 1) {
    sums[blockIdx.x] = total;
    __threadfence();
    last = atomicAdd(&done->blocks, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x == 0) at[0] = 0, at[1] = 0;
  long long carry = 0;
  for (int64_t b = 0; b < ntiles; b += kScanBlock) {
    const int64_t t = b + threadIdx.x;
    const long long v = t < ntiles ? __ldcg(&sums[t]) : 0;
    const long long incl = carry + block_inclusive(v, scratch), excl = incl - v;
    // sums are not negative: the tiles within the capacity come first
    const int within = __syncthreads_count(t < ntiles && excl <= capacity);
    if (t < ntiles && int(threadIdx.x) == within - 1) at[0] = t, at[1] = excl;
    __syncthreads();
    if (threadIdx.x == kScanBlock - 1) scratch[0] = incl;
    __syncthreads();
    carry = scratch[0];
    if (carry > capacity || within < kScanBlock) break;
  }
  const int64_t t0 = at[0] * kScanTile;
  long long run = at[1], prefix = t0;
  for (int i = 0; i < kScanItems; ++i) {
    const int64_t idx = t0 + int64_t(i) * kScanBlock + threadIdx.x;
    const long long incl = run + block_inclusive(idx < m ? c[idx] : 0, scratch);
    const int within = __syncthreads_count(idx < m && incl <= capacity);
    prefix += within;
    if (threadIdx.x == kScanBlock - 1) scratch[0] = incl;
    __syncthreads();
    run = scratch[0];
    if (within < kScanBlock) break;
  }
  if (threadIdx.x == 0) {
    scalars->prefix = prefix;
    scalars->count = found ? *found : ~0ull;
  }
}

// ---- all-pairs checker (get_collision_pairs, src/collision.cu:91-154) ---------
constexpr int kBruteTile = 128;

__global__ void __launch_bounds__(kBruteTile)
brute_force_kernel(const stq_aabb *__restrict__ boxes, int64_t n,
                   stq_pair *__restrict__ pairs, long long capacity,
                   unsigned long long *count) {
  __shared__ stq_aabb tile[kBruteTile];
  const int64_t i = int64_t(blockIdx.x) * kBruteTile + threadIdx.x;
  stq_aabb a;
  if (i < n) a = boxes[i];
  for (int64_t t0 = int64_t(blockIdx.y) * kBruteTile; t0 < n; t0 += int64_t(gridDim.y) * kBruteTile) {
    __syncthreads();
    if (t0 + threadIdx.x < n) tile[threadIdx.x] = boxes[t0 + threadIdx.x];
    __syncthreads();
    if (i >= n) continue;
    for (int q = 0; q < kBruteTile && t0 + q < n; ++q) {
      const int64_t jj = t0 + q;
      if (jj <= i) continue;
      const stq_aabb &b = tile[q];
      bool ov = true;
      for (int k = 0; k < 3; ++k) ov = ov && a.max[k] >= b.min[k] && a.min[k] <= b.max[k];
      const int4 av = make_int4(a.vertex_ids[0], a.vertex_ids[1], a.vertex_ids[2], a.id);
      const int4 bv = make_int4(b.vertex_ids[0], b.vertex_ids[1], b.vertex_ids[2], b.id);
      if (ov && valid_pair(av, bv) && !covertex(av, bv)) {
        const unsigned long long idx = atomicAdd(count, 1ull);
        if (idx < (unsigned long long)capacity)
          reinterpret_cast<int2 *>(pairs)[idx] = make_int2(min(a.id, b.id), max(a.id, b.id));
      }
    }
  }
}

}  // namespace

static cudaError_t launch_sweep_lanes(cudaStream_t s, const SweepParams &p, const SweepTuning &t,
                                      SweepMode mode, int num_sms);

cudaError_t launch_sweep(cudaStream_t s, const SweepParams &p, const SweepTuning &t,
                         SweepMode mode, int num_sms) {
  if (p.end <= p.begin) return cudaSuccess;
  cudaError_t e = launch_sweep_lanes(s, p, t, mode, num_sms);
  if (e != cudaSuccess) return e;
  if (!p.run_cap) return cudaSuccess;
  switch (mode) {
    case kSweepCount: return launch_long_runs<kSweepCount>(s, p, num_sms);
    case kSweepBoth: return launch_long_runs<kSweepBoth>(s, p, num_sms);
    default: return launch_long_runs<kSweepEmit>(s, p, num_sms);
  }
}

static cudaError_t launch_sweep_lanes(cudaStream_t s, const SweepParams &p, const SweepTuning &t,
                                      SweepMode mode, int num_sms) {
  // per-start-box counts do not depend on the tuning
  if (mode == kSweepCount) return launch_flat_block<256, 4, kSweepCount>(s, p, num_sms);
  if (mode == kSweepBoth) return launch_flat_block<256, 4, kSweepBoth>(s, p, num_sms);
  if (t.shape == kShapeFlat) {
    switch (t.per_lane) {  // filter steps per round
      case 2: return launch_flat<2>(s, p, t.block, num_sms);
      default: return launch_flat<4>(s, p, t.block, num_sms);
    }
  }
  if (t.lanes == 1) {  // one start box per lane
    switch (t.per_lane) {
      case 1: return launch_u<1>(s, p, t, num_sms);
      case 2: return launch_u<2>(s, p, t, num_sms);
      case 8: return launch_u<8>(s, p, t, num_sms);
      default: return launch_u<4>(s, p, t, num_sms);
    }
  }
  switch (t.lanes) {
    case 2: return launch_g<2>(s, p, t, num_sms);
    case 4: return launch_g<4>(s, p, t, num_sms);
    case 16: return launch_g<16>(s, p, t, num_sms);
    case 32: return launch_g<32>(s, p, t, num_sms);
    default: return launch_g<8>(s, p, t, num_sms);
  }
}

size_t prefix_workspace_bytes(int64_t m) {
  const int64_t ntiles = (m + kScanTile - 1) / kScanTile;
  return sizeof(long long) * (ntiles + 2);
}

cudaError_t launch_prefix_select(cudaStream_t s, const int32_t *box_counts, int64_t m,
                                 long long capacity, void *workspace, DevScalars *scalars,
                                 int64_t *launches, const unsigned long long *found) {
  const int64_t ntiles = (m + kScanTile - 1) / kScanTile;
  long long *sums = static_cast<long long *>(workspace);
  PrefixDone *done = reinterpret_cast<PrefixDone *>(sums + ntiles + 1);
  const cudaError_t e = cudaMemsetAsync(done, 0, sizeof(PrefixDone), s);
  if (e != cudaSuccess) return e;
  launch_after(prefix_select_kernel, unsigned(ntiles), kScanBlock, 0, s, box_counts, m, capacity, sums, ntiles, done,
               scalars, found);
  if (launches) *launches += 1;
  return cudaGetLastError();
}

cudaError_t launch_brute_force(cudaStream_t s, const stq_aabb *boxes, int64_t n,
                               stq_pair *pairs, long long capacity,
                               unsigned long long *count) {
  if (n < 2) return cudaSuccess;
  const int64_t tiles = (n + kBruteTile - 1) / kBruteTile;
  dim3 grid(unsigned(tiles), unsigned(tiles < 64 ? tiles : 64));
  brute_force_kernel<<<grid, kBruteTile, 0, s>>>(boxes, n, pairs, capacity, count);
  return cudaGetLastError();
}

}  // namespace stq
