// radix_sort.cu - stable LSD radix sort on the device, one launch per digit.
//
// Replaces the comparison sort of the reference (thrust::sort_by_key with
// sort_aabb_x, src/simulation.cu:645-649, 277-293).
//
// A histogram kernel reads the keys once and counts every digit; its last
// block turns the counts into first positions. Each digit is then one launch
// that reads the keys once and writes them once: a block takes tiles from a
// ticket counter, publishes a tile's digit counts, ranks the tile's keys in
// shared memory, and gets its tile's first positions by looking back over the
// tiles before it (a tile's predecessors have their tickets already, so they
// are running: the wait always ends; it is bounded all the same). A digit
// that is the same in every key is skipped.
//
// It sorts the replicas of a prepare, and those pairs that the bucket sort
// (pair_sort.cu) cannot take.
//
// What bounds it: the integer pipe (70% busy in a pass, shared-memory
// wavefronts 50%, DRAM 31%), that is the stable ranks. Measured against a
// histogram, two scans and a scatter per digit, with no digit skipped
// (CUDA events): 92 M pairs 5.58 -> 3.13 ms (six digits of 46 used bits are
// run, two skipped; 9.6 GB at 3.1 TB/s).
#include <algorithm>

#include "radix_device.cuh"
#include "stq_internal.h"

namespace stq {

namespace {

constexpr int kBins = kRadixBins;
constexpr int kMaxPasses = 8;
constexpr int kPassBlock = 512;
constexpr int kPassWarps = kPassBlock / 32;
constexpr int kMinTile = kRadixMinTile;  // smallest tile of a pass
static_assert(kMinTile == kPassBlock * 4, "smallest tile: four keys per thread");
constexpr int kHistBlock = 512;
// polls of one status word before a block gives up (each is a load from L2,
// some 0.5 us; a predecessor's counts take a few microseconds). A test builds the
// sort with 0: every tile but the first gives up.
#ifndef STQ_SORT_POLL_LIMIT
#define STQ_SORT_POLL_LIMIT (1 << 20)
#endif
constexpr int kPollLimit = STQ_SORT_POLL_LIMIT;

// Head of the workspace, cleared before every sort; the tiles' status words
// follow it.
struct SortHead {
  uint32_t hist[kMaxPasses][kBins];  // digit counts, then first positions
  uint32_t ticket[kMaxPasses];       // next tile of each pass; kNoTile and more: a wait gave up
  uint32_t done;                     // blocks of the histogram kernel that are done
  uint32_t run[kMaxPasses];          // the pass is run (not skipped)
  uint32_t src[kMaxPasses];          // buffer that the pass reads
};

static_assert(sizeof(SortHead) <= kRadixHeadBytes, "workspace sizing");

// Added to the tickets of a pass, and no later pass run, once a wait gave up: the words
// that blocks read anyway (a word of its own cost each tile of a pass 0.7 us).
constexpr uint32_t kNoTile = 1u << 30;

__device__ __forceinline__ void give_up(SortHead *head, int pass) {
  atomicMax(&head->ticket[pass], kNoTile);
  for (int q = pass + 1; q < kMaxPasses; ++q) head->run[q] = 0u;
}

// Bits of each digit of a sort, lowest first.
struct Digits {
  int passes;
  uint8_t shift[kMaxPasses];
  // on the device, the passes to run (null: those whose digit is not the same
  // in every key); the input is in buffer *d_passes & 1, the result in buffer 0
  const unsigned int *d_passes;
};

__device__ __forceinline__ unsigned long long load_status(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void store_status(unsigned long long *p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Exclusive scan of v over the first 256 threads of the block (every thread
// calls it; scratch: 8 words).
__device__ __forceinline__ uint32_t scan_bins(uint32_t v, uint32_t *scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
  if (threadIdx.x < kBins) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFullMask, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) scratch[warp] = x;
  }
  __syncthreads();
  uint32_t base = 0;
  if (threadIdx.x < kBins)
    for (int w = 0; w < warp; ++w) base += scratch[w];
  return base + x - v;
}

// Digit counts of every pass (one read of the keys) and, in the last block to
// finish, the first position of every digit, the passes to run and the buffer
// each reads. Also clears the tiles' status words. A digit that all keys share
// is skipped, unless that would leave the result in the second buffer: then one
// such pass is run as a copy (the number of passes is even).
template <typename K>
__global__ void __launch_bounds__(kHistBlock)
radix_hist_kernel(const K *__restrict__ k0, const K *__restrict__ k1, int64_t n, const unsigned int *d_n, Digits dg,
                  SortHead *head, unsigned long long *status, int tile) {
  after_previous();
  if (d_n && int64_t(*d_n) < n) n = *d_n;
  const K *__restrict__ keys = dg.d_passes && (*dg.d_passes & 1u) ? k1 : k0;
  __shared__ uint32_t h[kMaxPasses][kBins];
  __shared__ unsigned same;  // passes whose digit all keys share
  __shared__ uint32_t last;
  if (threadIdx.x == 0) same = 0;
  for (int i = threadIdx.x; i < kMaxPasses * kBins; i += kHistBlock) (&h[0][0])[i] = 0;
  const int64_t words = (n + tile - 1) / tile * kBins;
  for (int64_t i = blockIdx.x * int64_t(kHistBlock) + threadIdx.x; i < words; i += int64_t(gridDim.x) * kHistBlock)
    status[i] = 0ull;
  __syncthreads();
  constexpr int U = 4;
  const int64_t step = int64_t(gridDim.x) * kHistBlock * U;
  for (int64_t b = blockIdx.x * int64_t(kHistBlock) * U + threadIdx.x; b < n; b += step) {
    K k[U];
#pragma unroll
    for (int u = 0; u < U; ++u) k[u] = b + u * kHistBlock < n ? keys[b + u * kHistBlock] : K(0);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (b + u * kHistBlock < n)
#pragma unroll
        for (int p = 0; p < kMaxPasses; ++p)
          if (p < dg.passes) atomicAdd(&h[p][(k[u] >> dg.shift[p]) & (kBins - 1)], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < dg.passes * kBins; i += kHistBlock) {
    const uint32_t c = (&h[0][0])[i];
    if (c) atomicAdd(&(&head->hist[0][0])[i], c);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&head->done, 1u) == gridDim.x - 1 ? 1u : 0u;
  __syncthreads();
  if (!last) return;
  __threadfence();
  // one warp per pass, 8 digits per lane
  static_assert(kHistBlock / 32 >= kMaxPasses && kBins == 8 * 32, "a warp per pass");
  const int lane = threadIdx.x & 31, p = threadIdx.x >> 5;
  if (p < dg.passes) {
    uint32_t c[8], sum = 0;
    bool one = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      c[i] = __ldcg(&head->hist[p][lane * 8 + i]);
      sum += c[i];
      one |= int64_t(c[i]) == n;
    }
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFullMask, x, o);
      if (lane >= o) x += y;
    }
    x -= sum;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      head->hist[p][lane * 8 + i] = x;
      x += c[i];
    }
    one = __any_sync(kFullMask, one);
    if (lane == 0 && one) atomicOr(&same, 1u << p);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned skip = same;
    if (__popc(skip) & 1) skip &= skip - 1;  // run one of them: the result ends in the first buffer
    uint32_t src = 0;
    if (dg.d_passes) {
      const unsigned run = min(*dg.d_passes, unsigned(dg.passes));
      skip = ~((1u << run) - 1u);
      src = *dg.d_passes & 1u;
    }
    for (int q = 0; q < dg.passes; ++q) {
      const uint32_t run = (skip >> q & 1u) ? 0u : 1u;
      head->run[q] = run;
      head->src[q] = src;
      src ^= run;
    }
  }
}

// Sum of digit d's counts over the tiles before `tile`: reads the status words
// of the tiles before it, eight at a time, back to one that holds its own sum.
// Status word: (2 * pass + 1) << 32 | count of the tile, or (2 * pass + 2) << 32
// | sum up to and with the tile; smaller tags are from earlier passes.
// *timeout: a word did not come, here or in another block of the pass.
__device__ __forceinline__ uint32_t look_back(const uint32_t *ticket, const unsigned long long *status, int64_t tile,
                                              int d, uint32_t tag, bool *timeout) {
  uint32_t sum = 0;
  int polls = 0;
  int64_t t = tile - 1;
  while (t >= 0) {
    if (polls == kPollLimit ||
        (polls % 1024 == 1023 && *reinterpret_cast<const volatile uint32_t *>(ticket) >= kNoTile)) {
      *timeout = true;
      break;
    }
    ++polls;
    unsigned long long w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      w[i] = t - i >= 0 ? load_status(status + (t - i) * kBins + d) : (unsigned long long)(tag + 1) << 32;
    bool wait = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (wait || t < 0) continue;
      const uint32_t g = uint32_t(w[i] >> 32);
      if (g < tag) {
        wait = true;
        t -= i;
        if (i > 0) polls = 0;
      } else {
        sum += uint32_t(w[i]);
        if (g == tag + 1) t = -1;
      }
    }
    if (t < 0) break;
    if (!wait) {
      t -= 8;
      polls = 0;
    }
  }
  return sum;
}

template <typename K, bool VALS, int ITEMS>
struct PassShared {
  static constexpr int kTile = kPassBlock * ITEMS;
  K stage[kTile];
  uint32_t vstage[VALS ? kTile : 1];
  uint32_t cnt[kPassWarps][kBins];
  uint32_t out_base[kBins];  // output position of the tile's staged element p of digit d: out_base[d] + p
  uint32_t scratch[8];
  int64_t tile;
};

// One digit. Ranks are stable: a warp holds ITEMS x 32 consecutive keys, and
// takes them 32 at a time in order.
template <typename K, bool VALS, int ITEMS>
__global__ void __launch_bounds__(kPassBlock, 2)
radix_pass_kernel(K *k0, K *k1, uint32_t *v0, uint32_t *v1, int64_t n, const unsigned int *d_n, int pass, int shift,
                  SortHead *head, unsigned long long *status, int *fault) {
  after_previous();
  if (!head->run[pass]) return;
  if (d_n && int64_t(*d_n) < n) n = *d_n;
  const bool flip = head->src[pass] != 0;
  const K *__restrict__ kin = flip ? k1 : k0;
  K *__restrict__ kout = flip ? k0 : k1;
  const uint32_t *__restrict__ vin = flip ? v1 : v0;
  uint32_t *__restrict__ vout = flip ? v0 : v1;
  using S = PassShared<K, VALS, ITEMS>;
  constexpr int TILE = S::kTile;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  S &sm = *reinterpret_cast<S *>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t tag = 2u * unsigned(pass) + 1u;
  const int64_t tiles = (n + TILE - 1) / TILE;
  uint32_t *cnt = sm.cnt[warp];
  const unsigned below = lanemask_lt();
  while (true) {
    if (tid == 0) sm.tile = int64_t(atomicAdd(&head->ticket[pass], 1u));
    for (int i = lane; i < kBins; i += 32) cnt[i] = 0;
    __syncthreads();  // also: the tile before has been written out
    const int64_t tile = sm.tile;
    if (tile >= tiles) return;
    const int64_t start = tile * TILE;
    const int64_t wstart = start + int64_t(warp) * 32 * ITEMS + lane;
    const int count = int(n - start < TILE ? n - start : TILE);
    K key[ITEMS];
    uint32_t val[VALS ? ITEMS : 1];
    const bool full = count == TILE;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
      key[i] = full || wstart + i * 32 < n ? kin[wstart + i * 32] : ~K(0);
    if (VALS)
#pragma unroll
      for (int i = 0; i < ITEMS; ++i) val[i] = full || wstart + i * 32 < n ? vin[wstart + i * 32] : 0u;
    // 1. the tile's digit counts, per warp; published before the ranking, so
    //    that the tiles after this one need not wait for it
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
      if (full || wstart + i * 32 < n) atomicAdd(&cnt[digit_of(key[i], shift)], 1u);
    __syncthreads();
    uint32_t total = 0;
    if (tid < kBins) {
#pragma unroll
      for (int w = 0; w < kPassWarps; ++w) total += sm.cnt[w][tid];
      store_status(status + tile * kBins + tid, (unsigned long long)(tag + (tile == 0 ? 1u : 0u)) << 32 | total);
    }
    const uint32_t base = scan_bins(total, sm.scratch);  // the digit's first place in the tile
    if (tid < kBins) {
      uint32_t run = base;
#pragma unroll
      for (int w = 0; w < kPassWarps; ++w) {
        const uint32_t c = sm.cnt[w][tid];
        sm.cnt[w][tid] = run;
        run += c;
      }
    }
    __syncthreads();
    // 2. stable ranks; keys and values go to their places in the tile
    //    (keys past the end have all bits set: they come last)
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const unsigned d = digit_of(key[i], shift);
      const unsigned peers = same_digit(d);
      const uint32_t at = cnt[d];
      __syncwarp();
      if ((peers & below) == 0) cnt[d] = at + __popc(peers);
      __syncwarp();
      const uint32_t r = at + __popc(peers & below);
      sm.stage[r] = key[i];
      if (VALS) sm.vstage[r] = val[i];
    }
    // 3. the digits' first output positions
    bool timeout = false;
    if (tid < kBins) {
      const uint32_t before = look_back(&head->ticket[pass], status, tile, tid, tag, &timeout);
      if (tile > 0 && !timeout) store_status(status + tile * kBins + tid, (unsigned long long)(tag + 1u) << 32 | (before + total));
      sm.out_base[tid] = head->hist[pass][tid] + before - base;
    }
    // a wait that gave up leaves wrong positions: nothing is written then, here, by
    // the tiles that wait for this one, or in a later pass
    if (__syncthreads_or(timeout)) {
      if (tid == 0) {
        give_up(head, pass);
        *reinterpret_cast<volatile int *>(fault) = 1;
      }
      return;
    }
    // 4. out, digit by digit
#pragma unroll 4
    for (int p = tid; p < count; p += kPassBlock) {
      const K k = sm.stage[p];
      const uint32_t o = sm.out_base[digit_of(k, shift)] + unsigned(p);
      kout[o] = k;
      if (VALS) vout[o] = sm.vstage[p];
    }
  }
}

// A whole sort of at most kPassBlock * ITEMS keys by one block: keys (and
// values) stay in registers and shared memory between the digits. A small sort
// is all latency: 6,600 replicas take 16 us in this one launch; in the launches
// above each digit run costs 8 us and each skipped one 2.4.
template <int ITEMS>
struct BlockShared {
  uint32_t stage[kPassBlock * ITEMS];
  uint32_t vstage[kPassBlock * ITEMS];
  uint32_t cnt[kPassWarps][kBins];
  uint32_t scratch[8];
  uint32_t any, all;  // OR and AND of the keys
};

template <int ITEMS>
__global__ void __launch_bounds__(kPassBlock)
radix_block_kernel(const uint32_t *k0, const uint32_t *k1, uint32_t *kout, const uint32_t *v0, const uint32_t *v1,
                   uint32_t *vout, int n, const unsigned int *d_n, Digits dg) {
  after_previous();
  if (d_n && int(*d_n) < n) n = int(*d_n);
  const bool second = dg.d_passes && (*dg.d_passes & 1u);
  const uint32_t *kin = second ? k1 : k0;
  const uint32_t *vin = second ? v1 : v0;
  using S = BlockShared<ITEMS>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  S &sm = *reinterpret_cast<S *>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int first = warp * 32 * ITEMS + lane;
  const unsigned below = lanemask_lt();
  uint32_t *cnt = sm.cnt[warp];
  uint32_t key[ITEMS], val[ITEMS], o = 0u, a = ~0u;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const bool in = first + i * 32 < n;
    key[i] = in ? kin[first + i * 32] : ~0u;
    val[i] = in ? vin[first + i * 32] : 0u;
    if (in) o |= key[i], a &= key[i];
  }
  if (tid == 0) sm.any = 0u, sm.all = ~0u;
  __syncthreads();
  o = __reduce_or_sync(kFullMask, o);
  a = __reduce_and_sync(kFullMask, a);
  if (lane == 0) atomicOr(&sm.any, o), atomicAnd(&sm.all, a);
  __syncthreads();
  const uint32_t varies = sm.any & ~sm.all;  // bits that are not the same in every key
  for (int p = 0; p < dg.passes; ++p) {
    const int shift = dg.shift[p];
    if (((varies >> shift) & (kBins - 1)) == 0) continue;
    for (int i = lane; i < kBins; i += 32) cnt[i] = 0;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
      if (first + i * 32 < n) atomicAdd(&cnt[digit_of(key[i], shift)], 1u);
    __syncthreads();
    uint32_t total = 0;
    if (tid < kBins)
#pragma unroll
      for (int w = 0; w < kPassWarps; ++w) total += sm.cnt[w][tid];
    uint32_t run = scan_bins(total, sm.scratch);
    if (tid < kBins)
#pragma unroll
      for (int w = 0; w < kPassWarps; ++w) {
        const uint32_t c = sm.cnt[w][tid];
        sm.cnt[w][tid] = run;
        run += c;
      }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      // keys past the end have all bits set: they stay last
      const unsigned d = digit_of(key[i], shift);
      const unsigned peers = same_digit(d);
      const uint32_t at = cnt[d];
      __syncwarp();
      if ((peers & below) == 0) cnt[d] = at + __popc(peers);
      __syncwarp();
      if (first + i * 32 < n) {
        const uint32_t r = at + __popc(peers & below);
        sm.stage[r] = key[i];
        sm.vstage[r] = val[i];
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
      if (first + i * 32 < n) {
        key[i] = sm.stage[first + i * 32];
        val[i] = sm.vstage[first + i * 32];
      }
    // the next digit writes the stage after two more barriers
  }
#pragma unroll
  for (int i = 0; i < ITEMS; ++i)
    if (first + i * 32 < n) {
      kout[first + i * 32] = key[i];
      vout[first + i * 32] = val[i];
    }
}

template <typename K, bool VALS, int ITEMS>
cudaError_t launch_passes(cudaStream_t s, K *const kbuf[2], uint32_t *const vbuf[2], int64_t n, const unsigned int *d_n,
                          const Digits &dg, SortHead *head, unsigned long long *status, int *fault) {
  constexpr auto kern = radix_pass_kernel<K, VALS, ITEMS>;
  constexpr size_t smem = sizeof(PassShared<K, VALS, ITEMS>);
  cudaError_t e = allow_smem<kern>(smem);
  if (e != cudaSuccess) return e;
  const int64_t tiles = (n + kPassBlock * ITEMS - 1) / (kPassBlock * ITEMS);
  const unsigned grid = unsigned(std::min<int64_t>(tiles, int64_t(sm_count()) * 2));
  for (int p = 0; p < dg.passes; ++p) {
    launch_after(kern, grid, kPassBlock, smem, s, kbuf[0], kbuf[1], VALS ? vbuf[0] : nullptr,
                 VALS ? vbuf[1] : nullptr, n, d_n, p, dg.shift[p], head, status, fault);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <int ITEMS>
cudaError_t launch_block(cudaStream_t s, uint32_t *const kbuf[2], uint32_t *const vbuf[2], int64_t n, const Digits &dg,
                         const unsigned int *d_n, int64_t *launches) {
  constexpr auto kern = radix_block_kernel<ITEMS>;
  constexpr size_t smem = sizeof(BlockShared<ITEMS>);
  cudaError_t e = allow_smem<kern>(smem);
  if (e != cudaSuccess) return e;
  launch_after(kern, 1, kPassBlock, smem, s, kbuf[0], kbuf[1], kbuf[0], vbuf[0], vbuf[1], vbuf[0], int(n), d_n, dg);
  if (launches) *launches += 1;
  return cudaGetLastError();
}

template <typename K, bool VALS>
cudaError_t sort_impl(cudaStream_t s, K *const kbuf[2], uint32_t *const vbuf[2], int64_t n, const unsigned int *d_n,
                      const Digits &dg, void *workspace, int *fault, int64_t *launches, int64_t likely) {
  if (dg.passes == 0 || (n <= 1 && !dg.d_passes)) return cudaSuccess;
  SortHead *head = static_cast<SortHead *>(workspace);
  unsigned long long *status = reinterpret_cast<unsigned long long *>(static_cast<char *>(workspace) +
                                                                      kRadixHeadBytes);
  cudaError_t e = cudaMemsetAsync(head, 0, sizeof(SortHead), s);
  if (e != cudaSuccess) return e;
  // large tiles write longer digit runs and look back over fewer tiles; small
  // inputs take small ones, so that every SM gets a tile. The line is at half a
  // large tile per SM: 1.0 M u32 keys take 74 us in large tiles and 91 in small
  // ones, 346,000 64-bit keys 78 us in large and 70 in small ones.
  constexpr int kLarge = 16;
  static_assert(kPassBlock * kLarge >= 2 * kMinTile, "workspace sizing: status words of large tiles");
  const bool large = likely >= int64_t(sm_count()) * 4096 || n > kRadixMinTiles * kMinTile;
  const int tile = large ? kPassBlock * kLarge : kMinTile;
  const int64_t hist_blocks = (n + kHistBlock * 4 - 1) / (kHistBlock * 4);
  launch_after(radix_hist_kernel<K>, unsigned(std::min<int64_t>(hist_blocks, int64_t(sm_count()) * 4)), kHistBlock, 0,
               s, kbuf[0], kbuf[1], n, d_n, dg, head, status, tile);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  e = large ? launch_passes<K, VALS, kLarge>(s, kbuf, vbuf, n, d_n, dg, head, status, fault)
            : launch_passes<K, VALS, 4>(s, kbuf, vbuf, n, d_n, dg, head, status, fault);
  if (launches) *launches += 1 + dg.passes;
  return e;
}

}  // namespace

int sm_count() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) {
    (void)cudaGetLastError();
    sms = 152;
  }
  return sms;
}

cudaError_t radix_sort_u32(cudaStream_t s, uint32_t *const kbuf[2], uint32_t *const vbuf[2], int64_t n, void *workspace,
                           int *fault, int64_t *launches, const unsigned int *d_n, const unsigned int *d_passes,
                           int passes, int64_t likely) {
  const Digits dg{passes, {0, 8, 16, 24}, d_passes};
  // one block up to its 16 keys per thread. 1,000, 4,000 and 8,000 keys with 2, 8 and 16
  // per thread: 7.5, 13.2 and 18.0 us (with 16: 17.5, 17.8); in launches per digit 20, 23, 26
  if (passes > 0 && (n > 1 || d_passes)) {
    if (n <= kPassBlock * 2) return launch_block<2>(s, kbuf, vbuf, n, dg, d_n, launches);
    if (n <= kPassBlock * 8) return launch_block<8>(s, kbuf, vbuf, n, dg, d_n, launches);
    if (n <= kPassBlock * 16) return launch_block<16>(s, kbuf, vbuf, n, dg, d_n, launches);
  }
  return sort_impl<uint32_t, true>(s, kbuf, vbuf, n, d_n, dg, workspace, fault, launches, likely < 0 ? n : likely);
}

cudaError_t radix_sort_pairs(cudaStream_t s, stq_pair *pairs, stq_pair *tmp, int64_t n, void *workspace, int *fault,
                             int64_t *launches) {
  // a pair read as one little-endian word is second << 32 | first: the
  // second ids' digits, then the first ids'
  unsigned long long *kb[2] = {reinterpret_cast<unsigned long long *>(pairs),
                               reinterpret_cast<unsigned long long *>(tmp)};
  return sort_impl<unsigned long long, false>(s, kb, nullptr, n, nullptr,
                                              Digits{8, {32, 40, 48, 56, 0, 8, 16, 24}, nullptr},
                                              workspace, fault, launches, n);
}

}  // namespace stq
