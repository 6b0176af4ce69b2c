// pair_sort.cu - lexicographic sort of pairs by buckets of their first id.
//
// The pairs are cut into buckets of about 2,560 by the first id and each bucket
// is sorted by one block. A histogram of 8,192 bins of the first ids gives
// every bin its place; bins whose places begin in the same 2,560 make a bucket.
// A partition kernel moves the pairs to their buckets, in no order (its ranks are
// shared-memory atomics, a third of the instructions of a radix pass's stable
// ranks). In a bucket, pairs are grouped by first id and the leading bits of the
// second the same way, and each pair counts the smaller ones of its group. Above
// 4 M pairs the same histogram and partition first cut them into segments of about
// half a million. Up to 8,192 pairs are one bucket.
//
// Bins hold whole ids, so ids with many pairs make large buckets. Those above
// 4,096 pairs are left to a second launch, once the host sees that there are any
// (in meshes of millions of boxes: a few); where one passes 8,192 the later
// kernels do nothing, and the radix sort takes over (radix_sort.cu). A bucket of
// large groups (one id with many pairs, close to each other) is sorted by digits in
// its block.
//
// What bounds it: instruction issue (83% of cycles in the bucket kernel, half of
// the time; shared memory 71%, DRAM 13%, 21 of 32 lanes active in the loops over
// groups). Five light passes over the pairs take the place of one heavy pass per
// digit of both ids: against the radix sort, call to return, uniform ids: 92 M
// pairs 3.13 -> 1.87 ms, 36 M 1.26 -> 0.81, 2.1 M 138 -> 76 us, 346,000 70 -> 40 us.
// A crumpled mesh's 92 M pairs, where ids have up to 540: 3.04 -> 2.40 ms.
#include <algorithm>

#include "radix_device.cuh"
#include "stq_internal.h"

namespace stq {

namespace {

constexpr int kBlock = 512;
constexpr int kWarps = kBlock / 32;
constexpr int kPairBinBits = 13;
constexpr int kPairBins = 1 << kPairBinBits;  // at most
// Pairs between the places of two buckets. 92 M pairs take 2.39 ms at 2,048, 2.31 at
// 2,560 and 2.29 at 3,072; the rest up to kBucketCap is what a bin may hold.
constexpr uint32_t kBucket = 2560;
constexpr int kBucketCap = 4096;          // most pairs of a bucket that a block of 512 sorts
constexpr int kBigCap = 8192;             // and a block of 1024
constexpr int kGroupBits = 11;
constexpr int kGroups = 1 << kGroupBits;  // groups of a bucket
// Pairs of a pair's group, in the mean, up to which a bucket is sorted by counting. 5 M
// pairs in groups of 64, 96, 128 and 192: 233, 254, 274 and 325 us by counting, 281, 279,
// 276 and 277 by digits.
constexpr int kMaxGroup = 96;
constexpr uint32_t kSegment = 1u << 19;   // the same for segments (2^20: equal times, bins twice as large)
constexpr int kMaxSegments = 2048;
// Pairs that need no segments. The tables of one level are sized by it. One level, two
// levels: 1.25 M pairs 51, 107 us; 4 M 101, 152; 5 M, with tables for 8 M, 124, 170.
constexpr int64_t kOneLevel = 4 << 20;
constexpr int64_t kTwoLevels = int64_t(kSegment) * (kMaxSegments / 2);
constexpr int kHistTile = 65536;          // pairs per histogram block of a segment
constexpr int kPairPartTile = kBlock * 16;  // pairs per partition block of a segment
// buckets of a partition tile's segment: one level has up to kOneLevel / kBucket
// windows, a segment 2 * kSegment / kBucket, each with one bucket more at most
constexpr int kMaxTileBuckets = std::max(int(kOneLevel / kBucket), kMaxSegments) + 2;
static_assert(kMaxTileBuckets >= int(2 * kSegment / kBucket) + 2, "partition counters");

struct PairSeg {
  uint32_t begin, end;   // positions
  uint32_t base, span;   // first ids base .. base + span - 1 (0: 2^32)
  uint32_t shift;        // bin of id f: (f - base) >> shift
  uint32_t tile0;        // first of its tiles of the histogram
  uint32_t ptile0;       // and of the partition
  uint32_t bucket0, buckets;
};

struct PairBucket {
  uint32_t begin, end;  // positions
  uint32_t base, span;  // first ids base .. base + span - 1
};

// Counters of one level, cleared before it.
struct PairHead {
  uint32_t max_first;   // largest first id
  uint32_t max_bucket;  // longest bucket
  uint32_t buckets;     // buckets of all segments
  uint32_t segs_done;
  uint32_t fits;        // set once all segments are planned, if no bucket is too long
  uint32_t big;         // buckets above kBucketCap
  uint32_t segs, tiles, part_tiles;  // next level's segments and tiles
  uint32_t tiles_done[kMaxSegments];
};

constexpr int64_t div_up(int64_t a, int64_t b) { return (a + b - 1) / b; }
constexpr size_t up256(size_t v) { return (v + 255) & ~size_t(255); }

int bits_of(uint32_t v) {
  int b = 0;
  while (b < 32 && v >> b) ++b;
  return b;
}

// Workspace: the first level's and the last level's tables.
struct PairLayout {
  int64_t segs = 0, buckets = 0;  // most of them
  size_t head[2], bins[2], table[2], bucket[2], cursor[2], big, seg, total;
  static PairLayout make(int64_t n) {
    PairLayout l;
    const bool two = n > kOneLevel;
    l.segs = two ? n / kSegment + 2 : 1;
    l.buckets = n / kBucket + 2 * l.segs + 2;
    size_t o = 0;
    auto take = [&](size_t bytes) {
      const size_t at = o;
      o += up256(bytes);
      return at;
    };
    for (int k = 0; k < 2; ++k) {
      const int64_t s = k == 0 ? 1 : l.segs, b = k == 0 ? l.segs : l.buckets;
      l.head[k] = take(sizeof(PairHead));
      l.bins[k] = take(sizeof(uint32_t) * kPairBins * size_t(s));  // cleared with the head
      l.table[k] = take(sizeof(uint16_t) * kPairBins * size_t(s));
      l.bucket[k] = take(sizeof(PairBucket) * size_t(b));
      l.cursor[k] = take(sizeof(uint32_t) * size_t(b));
    }
    l.big = take(sizeof(uint32_t) * size_t(l.buckets));
    l.seg = take(sizeof(PairSeg) * size_t(l.segs));
    l.total = o;
    return l;
  }
};

struct PairLevel {
  PairHead *head;
  uint32_t *bins;     // per segment
  uint16_t *table;    // bucket of each bin, in the segment
  PairBucket *bucket;
  uint32_t *cursor;   // next place of each bucket
  uint32_t *big;      // the buckets above kBucketCap (last level), or null
  uint32_t window;    // pairs between the places of two buckets
  uint32_t cap;       // most pairs of a bucket
  int nbins;          // bins of a segment: a power of two, kBlock to kPairBins
  const PairHead *before;  // of the level before, which gives segs; or null
  PairSeg *next;      // segments made of the buckets (first of two levels), or null
  PairPlan *plan;     // page-locked
};

// Exclusive scan of one value per thread; *total in every thread.
template <int THREADS = kBlock>
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t *total, uint32_t *scratch) {
  constexpr int kN = THREADS / 32;
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
  uint32_t w = lane < kN ? scratch[lane] : 0u;  // every warp scans the warps' sums
#pragma unroll
  for (int o = 1; o < kN; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFullMask, w, o);
    if (lane >= o) w += y;
  }
  *total = __shfl_sync(kFullMask, w, kN - 1);
  const uint32_t before = __shfl_sync(kFullMask, w, warp > 0 ? warp - 1 : 0);
  return (warp > 0 ? before : 0u) + x - v;
}

// The segment of this block's tile; false if there is none.
__device__ __forceinline__ bool segment_of(const PairSeg *segs, const PairLevel &lv, bool partition, PairSeg *sg,
                                           int *which) {
  *which = 0;
  if (!segs) return true;
  if (!lv.before->fits || blockIdx.x >= (partition ? lv.before->part_tiles : lv.before->tiles)) return false;
  int lo = 0, hi = int(lv.before->segs) - 1;  // the last segment whose first tile is at or before this block's
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((partition ? segs[mid].ptile0 : segs[mid].tile0) <= blockIdx.x) lo = mid;
    else hi = mid - 1;
  }
  *which = lo;
  *sg = segs[lo];
  return true;
}

__device__ __forceinline__ uint32_t bin_of(unsigned long long pair, const PairSeg &sg, int nbins) {
  return min((uint32_t(pair) - sg.base) >> sg.shift, uint32_t(nbins - 1));
}

// Bins of a segment -> buckets, by the block that finished its histogram. pre:
// kPairBins + 256 words of shared memory.
__device__ void plan_segment(const PairLevel &lv, const PairSeg &sg, int which, int nsegs, PairSeg *segs, uint32_t *pre,
                             uint32_t *scratch) {
  const int kPer = lv.nbins / kBlock;
  auto at = [](int x) { return x + (x >> 5); };
  const uint32_t *bins = lv.bins + size_t(which) * kPairBins;
  __shared__ uint32_t bucket0;
  for (int i = threadIdx.x; i < lv.nbins; i += kBlock) pre[at(i)] = __ldcg(&bins[i]);
  __syncthreads();
  uint32_t sum = 0, total;
  for (int i = 0; i < kPer; ++i) sum += pre[at(threadIdx.x * kPer + i)];
  uint32_t run = block_scan(sum, &total, scratch);
  for (int i = 0; i < kPer; ++i) {
    const uint32_t c = pre[at(threadIdx.x * kPer + i)];
    pre[at(threadIdx.x * kPer + i)] = run;
    run += c;
  }
  __syncthreads();
  // a bucket begins at the first bin of each window
  auto begins = [&](int f) { return f == 0 || pre[at(f)] / lv.window != pre[at(f - 1)] / lv.window; };
  uint32_t mine = 0, nb;
  for (int i = 0; i < kPer; ++i) mine += begins(threadIdx.x * kPer + i) ? 1u : 0u;
  uint32_t id = block_scan(mine, &nb, scratch);
  if (threadIdx.x == 0) bucket0 = atomicAdd(&lv.head->buckets, nb);
  __syncthreads();
  PairBucket *bk = lv.bucket + bucket0;
  for (int i = 0; i < kPer; ++i) {
    const int f = threadIdx.x * kPer + i;
    if (begins(f)) {
      bk[id].begin = sg.begin + pre[at(f)];
      bk[id].base = sg.base + (uint32_t(f) << sg.shift);
      ++id;
    }
    lv.table[size_t(which) * kPairBins + f] = uint16_t(id - 1);
  }
  __syncthreads();
  const uint32_t past = sg.base + (segs ? sg.span : __ldcg(&lv.head->max_first) + 1u);  // (2^32 reads 0: spans wrap)
  uint32_t longest = 0;
  for (uint32_t d = threadIdx.x; d < nb; d += kBlock) {
    const uint32_t begin = bk[d].begin, end = d + 1 < nb ? bk[d + 1].begin : sg.end;
    bk[d].end = end;
    bk[d].span = (d + 1 < nb ? bk[d + 1].base : past) - bk[d].base;
    lv.cursor[bucket0 + d] = begin;
    if (lv.big && end - begin > unsigned(kBucketCap)) lv.big[atomicAdd(&lv.head->big, 1u)] = bucket0 + d;
    longest = max(longest, end - begin);
  }
  longest = __reduce_max_sync(kFullMask, longest);
  if ((threadIdx.x & 31) == 0 && longest) atomicMax(&lv.head->max_bucket, longest);
  if (segs && threadIdx.x == 0) {
    segs[which].bucket0 = bucket0;
    segs[which].buckets = nb;
  }
  __syncthreads();
  if (lv.next) {  // the buckets as the next level's segments, but for an empty one
    //               after the last pair
    const uint32_t nb_all = nb;
    if (bk[nb_all - 1].begin == sg.end) --nb;
    uint32_t tiles = 0, ptiles = 0;
    for (uint32_t b = 0; b < nb; b += kBlock) {
      const uint32_t d = b + threadIdx.x;
      const uint32_t size = d < nb ? bk[d].end - bk[d].begin : 0u;
      const uint32_t t = (size + kHistTile - 1) / kHistTile, pt = (size + kPairPartTile - 1) / kPairPartTile;
      uint32_t all, pall;
      const uint32_t t0 = tiles + block_scan(t, &all, scratch), pt0 = ptiles + block_scan(pt, &pall, scratch);
      if (d < nb) {
        const int bits = 32 - __clz(bk[d].span - 1u);
        lv.next[d] = PairSeg{bk[d].begin, bk[d].end, bk[d].base, bk[d].span, uint32_t(max(bits - kPairBinBits, 0)),
                             t0, pt0, 0u, 0u};
      }
      tiles += all;
      ptiles += pall;
    }
    if (threadIdx.x == 0) lv.head->tiles = tiles, lv.head->part_tiles = ptiles, lv.head->segs = nb;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(&lv.head->segs_done, 1u) + 1u == unsigned(nsegs)) {
    __threadfence();
    const uint32_t longest_all = __ldcg(&lv.head->max_bucket), most = __ldcg(&lv.head->max_first);
    const bool fits = longest_all <= lv.cap && (segs || most >> sg.shift < unsigned(lv.nbins));
    lv.head->fits = fits ? 1u : 0u;
    if (!segs) lv.plan->max_first = most;
    lv.plan->fits = fits ? 1u : 0u;
    lv.plan->big = __ldcg(&lv.head->big);
  }
}

// Histogram of the first ids of one tile of a segment (of `tile` pairs).
__global__ void __launch_bounds__(kBlock)
pair_hist_kernel(const unsigned long long *__restrict__ pairs, PairSeg one, PairSeg *segs, uint32_t tile, PairLevel lv) {
  after_previous();
  __shared__ uint32_t h[kPairBins + kPairBins / 32];
  __shared__ uint32_t scratch[kWarps];
  __shared__ bool last;
  int which;
  PairSeg sg = one;
  if (!segment_of(segs, lv, false, &sg, &which)) return;
  const int nsegs = segs ? int(lv.before->segs) : 1;
  const uint32_t begin = sg.begin + (blockIdx.x - sg.tile0) * tile, end = min(begin + tile, sg.end);
  for (int i = threadIdx.x; i < lv.nbins; i += kBlock) h[i] = 0;
  __syncthreads();
  uint32_t most = 0;
  constexpr int U = 4;
  for (uint32_t b = begin; b < end; b += kBlock * U) {
    unsigned long long k[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t i = b + u * kBlock + threadIdx.x;
      k[u] = i < end ? pairs[i] : 0ull;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (b + u * kBlock + threadIdx.x < end) {
        most = max(most, uint32_t(k[u]));
        atomicAdd(&h[bin_of(k[u], sg, lv.nbins)], 1u);
      }
  }
  most = __reduce_max_sync(kFullMask, most);
  if ((threadIdx.x & 31) == 0) atomicMax(&lv.head->max_first, most);
  __syncthreads();
  uint32_t *bins = lv.bins + size_t(which) * kPairBins;
  for (int i = threadIdx.x; i < lv.nbins; i += kBlock)
    if (h[i]) atomicAdd(&bins[i], h[i]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0)
    last = atomicAdd(&lv.head->tiles_done[which], 1u) + 1u == (sg.end - sg.begin + tile - 1) / tile;
  __syncthreads();
  if (!last) return;
  __threadfence();
  plan_segment(lv, sg, which, nsegs, segs, h, scratch);
}

// Moves a tile's pairs to their buckets, through shared memory so that each
// bucket's pairs of the tile are written together.
template <int ITEMS>
struct PartShared {
  unsigned long long stage[kBlock * ITEMS];
  uint32_t cnt[kMaxTileBuckets];    // pairs of the tile per bucket, then their first places in it
  uint32_t gbase[kMaxTileBuckets];  // output position of the tile's staged pair p: gbase + p
  uint32_t scratch[kWarps];
};

template <int ITEMS>
__global__ void __launch_bounds__(kBlock, 2)
pair_partition_kernel(const unsigned long long *__restrict__ in, unsigned long long *__restrict__ out, PairSeg one,
                      const PairSeg *segs, PairLevel lv) {
  after_previous();
  constexpr uint32_t TILE = kBlock * ITEMS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PartShared<ITEMS> &sm = *reinterpret_cast<PartShared<ITEMS> *>(smem_raw);
  int which;
  PairSeg sg = one;
  if (!lv.head->fits || !segment_of(segs, lv, true, &sg, &which)) return;
  const uint32_t begin = sg.begin + (blockIdx.x - sg.ptile0) * TILE;
  const uint32_t count = min(TILE, sg.end - begin);
  const uint16_t *__restrict__ table = lv.table + size_t(which) * kPairBins;
  uint32_t *cursor = lv.cursor + sg.bucket0;
  const int nb = int(segs ? sg.buckets : lv.head->buckets), nbins = lv.nbins;
  unsigned long long key[ITEMS];
  uint32_t place[ITEMS];  // bucket << 16 | rank in the tile's pairs of it
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const uint32_t p = i * kBlock + threadIdx.x;
    key[i] = p < count ? in[begin + p] : 0ull;
  }
  for (int i = threadIdx.x; i < nb; i += kBlock) sm.cnt[i] = 0;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ITEMS; ++i)
    if (i * kBlock + threadIdx.x < count) place[i] = uint32_t(table[bin_of(key[i], sg, nbins)]) << 16;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i)
    if (i * kBlock + threadIdx.x < count) place[i] |= atomicAdd(&sm.cnt[place[i] >> 16], 1u);
  __syncthreads();
  uint32_t carry = 0;
  for (int b = 0; b < nb; b += kBlock) {
    const int d = b + threadIdx.x;
    const uint32_t c = d < nb ? sm.cnt[d] : 0u;
    uint32_t all;
    const uint32_t at = carry + block_scan(c, &all, sm.scratch);
    if (d < nb) {
      sm.cnt[d] = at;
      if (c) sm.gbase[d] = atomicAdd(&cursor[d], c) - at;
    }
    carry += all;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ITEMS; ++i)
    if (i * kBlock + threadIdx.x < count) sm.stage[sm.cnt[place[i] >> 16] + (place[i] & 0xffffu)] = key[i];
  __syncthreads();
#pragma unroll 4
  for (uint32_t p = threadIdx.x; p < count; p += kBlock) {
    const unsigned long long k = sm.stage[p];
    out[sm.gbase[table[bin_of(k, sg, nbins)]] + p] = k;
  }
}

// Sorts one bucket; one of more than CAP pairs is left. AUTO: the only bucket, of
// n pairs, whose first ids are not known beforehand. Else with a list: the bucket
// that the list has for the block.
// Where the bucket has no more first ids than groups (narrow), an id's pairs are
// cut into several groups by the leading bits of their second ids, so that the
// groups number 2,048 whatever the pairs per id; a group's number stands for the
// id, and the comparisons are of second ids alone: 3.5 instructions each, against
// 10 of whole pairs with the place as a tie-break.
template <int THREADS, int CAP>
struct BucketShared {
  union {
    unsigned long long key[CAP];  // first id << 32 | second id, by group
    struct {
      uint32_t second[CAP];       // narrow: second id
      uint16_t group[CAP];        // and group
    };
  };
  union {
    uint32_t off[kGroups + 1];  // counts, then first places of the groups
    uint32_t cnt[THREADS / 32][kRadixBins];  // by digits: counts per warp
  };
  uint32_t scratch[THREADS / 32];
  uint32_t least, most;    // first ids (of the only bucket)
  uint32_t least2, most2;  // second ids
  uint32_t squares;        // of the groups' sizes, summed
};

template <int THREADS, int CAP, bool AUTO>
__global__ void __launch_bounds__(THREADS, THREADS == 512 && !AUTO ? 4 : 1)
pair_bucket_kernel(const unsigned long long *in, unsigned long long *out, const PairBucket *__restrict__ buckets,
                   const PairHead *head, const uint32_t *__restrict__ list, int n) {
  after_previous();
  constexpr int ITEMS = CAP / THREADS;
  static_assert(kGroups % THREADS == 0, "groups per thread");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using S = BucketShared<THREADS, CAP>;
  S &sm = *reinterpret_cast<S *>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t start = 0, base = 0, span = 0;
  if (!AUTO) {
    if (!head->fits || blockIdx.x >= head->buckets) return;
    const PairBucket b = buckets[list ? list[blockIdx.x] : blockIdx.x];
    start = b.begin;
    n = int(b.end - b.begin);
    if (n > CAP) return;
    base = b.base;
    span = b.span;
  }
  if (n == 0) return;
  // pairs as sort keys: first id above second
  unsigned long long key[ITEMS];
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int p = i * THREADS + tid;
    if (i * THREADS >= n) break;  // the same for all threads: a bucket may be half full
    const unsigned long long r = p < n ? in[start + p] : 0ull;
    key[i] = r << 32 | r >> 32;
  }
  for (int i = tid; i <= kGroups; i += THREADS) sm.off[i] = 0;
  if (tid == 0) sm.least = sm.least2 = 0xffffffffu, sm.most = sm.most2 = 0u, sm.squares = 0u;
  __syncthreads();
  uint32_t lo2 = 0xffffffffu, hi2 = 0u;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i)
    if (i * THREADS + tid < n) lo2 = min(lo2, uint32_t(key[i])), hi2 = max(hi2, uint32_t(key[i]));
  lo2 = __reduce_min_sync(kFullMask, lo2);
  hi2 = __reduce_max_sync(kFullMask, hi2);
  if (lane == 0) atomicMin(&sm.least2, lo2), atomicMax(&sm.most2, hi2);
  if (AUTO) {
    uint32_t lo = 0xffffffffu, hi = 0u;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
      if (i * THREADS + tid < n) lo = min(lo, uint32_t(key[i] >> 32)), hi = max(hi, uint32_t(key[i] >> 32));
    lo = __reduce_min_sync(kFullMask, lo);
    hi = __reduce_max_sync(kFullMask, hi);
    if (lane == 0) atomicMin(&sm.least, lo), atomicMax(&sm.most, hi);
  }
  __syncthreads();
  if (AUTO) {
    base = sm.least;
    span = sm.most - base + 1u;
  }
  // a group: the pairs of 2^shift first ids (span 0 stands for 2^32), or one first
  // id's pairs of 2^shift2 second ids
  const int bits = 32 - __clz(span - 1u);
  const int shift = max(bits - kGroupBits, 0), sub = max(kGroupBits - bits, 0);
  lo2 = sm.least2;
  const int shift2 = max(32 - __clz(sm.most2 - lo2) - sub, 0);
  const uint32_t mask2 = sub ? 0xffffffffu : 0u;
  auto group_of = [&](unsigned long long k) {
    return (((uint32_t(k >> 32) - base) >> shift) << sub) + (((uint32_t(k) - lo2) & mask2) >> shift2);
  };
  uint32_t rank[ITEMS];
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    if (i * THREADS >= n) break;
    if (i * THREADS + tid < n) rank[i] = atomicAdd(&sm.off[group_of(key[i])], 1u);
  }
  __syncthreads();
  {
    constexpr int kPer = kGroups / THREADS;
    uint32_t c[kPer], sum = 0, squares = 0, all;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      c[i] = sm.off[tid * kPer + i];
      sum += c[i];
      squares += c[i] * c[i];
    }
    squares = __reduce_add_sync(kFullMask, squares);
    if (lane == 0) atomicAdd(&sm.squares, squares);
    uint32_t run = block_scan<THREADS>(sum, &all, sm.scratch);
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      sm.off[tid * kPer + i] = run;
      run += c[i];
    }
    if (tid == 0) sm.off[kGroups] = uint32_t(n);
  }
  __syncthreads();
  const bool counting = sm.squares <= uint32_t(n) * kMaxGroup;
  if (counting && shift == 0) {
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      if (i * THREADS >= n) break;
      if (i * THREADS + tid < n) {
        const uint32_t g = group_of(key[i]), at = sm.off[g] + rank[i];
        sm.second[at] = uint32_t(key[i]);
        sm.group[at] = uint16_t(g);
      }
    }
    __syncthreads();
    for (int p = tid; p < n; p += THREADS) {
      const uint32_t k = sm.second[p], g = sm.group[p];
      const int lo = int(sm.off[g]), hi = int(sm.off[g + 1]);
      int at = lo;  // equal pairs keep their order
#pragma unroll 4
      for (int j = lo; j < p; ++j) at += sm.second[j] <= k ? 1 : 0;
#pragma unroll 4
      for (int j = p + 1; j < hi; ++j) at += sm.second[j] < k ? 1 : 0;
      out[start + at] = (unsigned long long)k << 32 | (base + (g >> sub));
    }
    return;
  }
  if (counting) {
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
      if (i * THREADS + tid < n) sm.key[sm.off[group_of(key[i])] + rank[i]] = key[i];
    __syncthreads();
    for (int p = tid; p < n; p += THREADS) {
      const unsigned long long k = sm.key[p];
      const uint32_t g = group_of(k);
      const int lo = int(sm.off[g]), hi = int(sm.off[g + 1]);
      int at = lo;
      for (int j = lo; j < p; ++j) at += sm.key[j] <= k ? 1 : 0;
      for (int j = p + 1; j < hi; ++j) at += sm.key[j] < k ? 1 : 0;
      out[start + at] = k << 32 | k >> 32;
    }
    return;
  }
  // large groups: by digits, the ones that vary (stable ranks as in radix_sort.cu;
  // here a warp holds ITEMS x 32 consecutive places). The counts take the groups'
  // place, which nobody reads any more.
  const int first = warp * 32 * ITEMS + lane;
  const unsigned below = lanemask_lt();
#pragma unroll
  for (int i = 0; i < ITEMS; ++i)
    if (i * THREADS + tid < n) sm.key[i * THREADS + tid] = key[i];
  for (int s = 0; s < 64; s += 8) {
    for (int i = lane; i < kRadixBins; i += 32) sm.cnt[warp][i] = 0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) key[i] = first + i * 32 < n ? sm.key[first + i * 32] : ~0ull;
    const unsigned d0 = digit_of(sm.key[0], s);
    bool same = true;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
      if (first + i * 32 < n) {
        const unsigned d = digit_of(key[i], s);
        same &= d == d0;
        atomicAdd(&sm.cnt[warp][d], 1u);
      }
    if (__syncthreads_and(same)) continue;
    uint32_t total = 0;
    if (tid < kRadixBins)
      for (int w = 0; w < THREADS / 32; ++w) total += sm.cnt[w][tid];
    uint32_t all;
    uint32_t run = block_scan<THREADS>(total, &all, sm.scratch);
    if (tid < kRadixBins)
      for (int w = 0; w < THREADS / 32; ++w) {
        const uint32_t c = sm.cnt[w][tid];
        sm.cnt[w][tid] = run;
        run += c;
      }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      // places past the end hold all bits: they stay last
      const unsigned d = digit_of(key[i], s);
      const unsigned peers = same_digit(d);
      const uint32_t at = sm.cnt[warp][d];
      __syncwarp();
      if ((peers & below) == 0) sm.cnt[warp][d] = at + __popc(peers);
      __syncwarp();
      if (first + i * 32 < n) sm.key[at + __popc(peers & below)] = key[i];
    }
    __syncthreads();
  }
  __syncthreads();
  for (int p = tid; p < n; p += THREADS) out[start + p] = sm.key[p] << 32 | sm.key[p] >> 32;
}

template <int ITEMS>
cudaError_t launch_partition(cudaStream_t s, int64_t blocks, const unsigned long long *in, unsigned long long *out,
                             const PairSeg &one, const PairSeg *segs, const PairLevel &lv) {
  constexpr auto kern = pair_partition_kernel<ITEMS>;
  constexpr size_t smem = sizeof(PartShared<ITEMS>);
  const cudaError_t e = allow_smem<kern>(smem);
  if (e != cudaSuccess) return e;
  launch_after(kern, unsigned(blocks), kBlock, smem, s, in, out, one, segs, lv);
  return cudaGetLastError();
}

template <int THREADS, int CAP, bool AUTO>
cudaError_t launch_buckets(cudaStream_t s, int64_t blocks, const unsigned long long *in, unsigned long long *out,
                           const PairBucket *buckets, const PairHead *head, const uint32_t *list, int n) {
  constexpr auto kern = pair_bucket_kernel<THREADS, CAP, AUTO>;
  constexpr size_t smem = sizeof(BucketShared<THREADS, CAP>);
  const cudaError_t e = allow_smem<kern>(smem);
  if (e != cudaSuccess) return e;
  launch_after(kern, unsigned(blocks), THREADS, smem, s, in, out, buckets, head, list, n);
  return cudaGetLastError();
}

}  // namespace

size_t pair_workspace_bytes(int64_t n) {
  return std::max(radix_workspace_bytes(n), n <= kTwoLevels ? PairLayout::make(n).total : size_t(0));
}

cudaError_t sort_pairs(cudaStream_t s, stq_pair *d_pairs, stq_pair *tmp, int64_t n, void *ws, PairPlan *plan,
                       int *id_bits, int *fault, int64_t *launches) {
  if (n < 2) return cudaSuccess;
  unsigned long long *a = reinterpret_cast<unsigned long long *>(d_pairs);
  unsigned long long *b = reinterpret_cast<unsigned long long *>(tmp);
  if (n <= kBigCap) {  // one bucket
    *launches += 1;
    return n <= kBucketCap ? launch_buckets<512, kBucketCap, true>(s, 1, a, a, nullptr, nullptr, nullptr, int(n))
                           : launch_buckets<1024, kBigCap, true>(s, 1, a, a, nullptr, nullptr, nullptr, int(n));
  }
  if (n > kTwoLevels) return radix_sort_pairs(s, d_pairs, tmp, n, ws, fault, launches);
  const PairLayout l = PairLayout::make(n);
  const bool two = n > kOneLevel;
  char *w = static_cast<char *>(ws);
  PairSeg *segs = reinterpret_cast<PairSeg *>(w + l.seg);
  auto level = [&](int k) {
    PairLevel lv{};
    lv.head = reinterpret_cast<PairHead *>(w + l.head[k]);
    lv.bins = reinterpret_cast<uint32_t *>(w + l.bins[k]);
    lv.table = reinterpret_cast<uint16_t *>(w + l.table[k]);
    lv.bucket = reinterpret_cast<PairBucket *>(w + l.bucket[k]);
    lv.cursor = reinterpret_cast<uint32_t *>(w + l.cursor[k]);
    lv.window = kBucket;
    lv.cap = kBigCap;
    lv.nbins = kPairBins;
    lv.plan = plan;
    return lv;
  };
  auto clear = [&](const PairLevel &lv, int k, int64_t nsegs) {
    return cudaMemsetAsync(lv.head, 0, l.bins[k] - l.head[k] + sizeof(uint32_t) * kPairBins * size_t(nsegs), s);
  };
  const PairLevel last = [&] {
    PairLevel lv = level(1);
    lv.big = reinterpret_cast<uint32_t *>(w + l.big);
    if (two) lv.before = reinterpret_cast<const PairHead *>(w + l.head[0]);
    // some eight bins per bucket: every block adds its bins to the segment's
    else while (lv.nbins > kBlock && lv.nbins / 2 >= 8 * (n / int64_t(kBucket))) lv.nbins /= 2;
    return lv;
  }();
  PairLevel first = last;
  if (two) {
    first = level(0);
    first.window = kSegment;
    first.cap = 2 * kSegment;
    first.next = segs;
    first.big = nullptr;
  }
  int bin_bits = 0;
  while ((1 << bin_bits) < first.nbins) ++bin_bits;
  // one histogram block per SM and 4,096 pairs at least
  const int64_t tile = div_up(std::max<int64_t>(div_up(n, sm_count() * (two ? 2 : 1)), 4096), kBlock) * kBlock;
  PairSeg one{0, uint32_t(n), 0, 0, 0, 0, 0, 0, 0};
  for (int tries = 0;; ++tries) {
    one.shift = uint32_t(std::max(*id_bits - bin_bits, 0));
    plan->fits = 0;
    cudaError_t e = clear(first, two ? 0 : 1, 1);
    if (e == cudaSuccess && two) e = clear(last, 1, l.segs);
    if (e != cudaSuccess) return e;
    launch_after(pair_hist_kernel, unsigned(div_up(n, tile)), kBlock, 0, s, a, one, nullptr, uint32_t(tile), first);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    // every later kernel looks whether the buckets fit, and does nothing if not. Tiles
    // of 16 pairs per thread where they give every SM one; 16, 4: 0.3 M pairs 35, 33 us,
    // 1.25 M 51, 52, 2 M 66, 72, 4 M 101, 117
    e = n >= int64_t(sm_count()) * 8192 ? launch_partition<16>(s, div_up(n, kBlock * 16), a, b, one, nullptr, first)
                                        : launch_partition<4>(s, div_up(n, kBlock * 4), a, b, one, nullptr, first);
    if (e != cudaSuccess) return e;
    *launches += 2;
    if (two) {
      launch_after(pair_hist_kernel, unsigned(n / kHistTile + l.segs), kBlock, 0, s, b, one, segs, kHistTile, last);
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
      e = launch_partition<16>(s, n / kPairPartTile + l.segs, b, a, one, segs, last);
      if (e != cudaSuccess) return e;
      *launches += 2;
    }
    e = launch_buckets<512, kBucketCap, false>(s, l.buckets, two ? a : b, a, last.bucket, last.head, nullptr, 0);
    *launches += 1;
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return e;
    if (plan->fits) {
      if (plan->big == 0) return cudaSuccess;
      *launches += 1;
      return launch_buckets<1024, kBigCap, false>(s, plan->big, two ? a : b, a, last.bucket, last.head, last.big, 0);
    }
    // the ids' true width, once; then ids have very many pairs
    const int bits = bits_of(plan->max_first);
    if (bits == *id_bits || tries > 0) return radix_sort_pairs(s, d_pairs, tmp, n, ws, fault, launches);
    *id_bits = bits;
  }
}

}  // namespace stq
