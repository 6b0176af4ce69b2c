// static_sweep.cu - the one entry point that allocates nothing.
//
// Some callers cannot allocate device memory at the moment they need a broad
// phase: simulation steps that run under a memory budget reserved up front
// (an out-of-memory error in the middle of a step is not recoverable for
// them), hosts whose own pooling allocator owns the device memory and forbids
// the CUDA runtime's, and real-time loops that cannot take the device-wide
// synchronisation cudaFree may cause. stq_sweep_static serves them: it sorts
// and sweeps one scene of at most STQ_STATIC_MAX_BOXES boxes using only the
// file-scope scratch array below, which every GPU that loads this library
// holds until the process exits. The caller passes the boxes and the pair
// buffer.
#include <mutex>

#include "stq_device.cuh"
#include "stq_internal.h"

namespace stq {
namespace {

constexpr int64_t kMax = STQ_STATIC_MAX_BOXES;
constexpr int64_t kSlots = kMax + 1 + kSortedPad;

// Byte layout of the scratch array (offsets are multiples of 256).
constexpr size_t up256(size_t v) { return (v + 255) & ~size_t(255); }
constexpr size_t kOffKeys0 = 0;
constexpr size_t kOffVals0 = kOffKeys0 + up256(sizeof(uint32_t) * kMax);
// the sort's second buffers; the sweep's list of long runs takes their place
constexpr size_t kOffKeys1 = kOffVals0 + up256(sizeof(uint32_t) * kMax);
constexpr size_t kOffVals1 = kOffKeys1 + up256(sizeof(uint32_t) * kMax);
constexpr size_t kOffLong = kOffKeys1;
static_assert(sizeof(int2) * kMax <= 2 * up256(sizeof(uint32_t) * kMax), "long runs fit the sort's second buffers");
constexpr size_t kOffSortWs = kOffVals1 + up256(sizeof(uint32_t) * kMax);
constexpr size_t kSortWsBytes = radix_workspace_bytes(kMax);
constexpr size_t kOffYz = kOffSortWs + up256(kSortWsBytes);
constexpr size_t kOffX = kOffYz + up256(sizeof(float4) * kSlots);
constexpr size_t kOffV = kOffX + up256(sizeof(float2) * kSlots);
constexpr size_t kOffFlag = kOffV + up256(sizeof(int4) * kSlots);
constexpr size_t kOffCode = kOffFlag + up256(sizeof(int) * kSlots);
constexpr size_t kOffPartner = kOffCode + up256(sizeof(uint32_t) * kSlots);
constexpr size_t kOffRunEnd = kOffPartner + up256(sizeof(int) * kSlots);
constexpr size_t kOffHdr = kOffRunEnd + up256(sizeof(int) * kSlots);
constexpr size_t kOffExtent = kOffHdr + up256(sizeof(BatchHeader));  // see static_keys_kernel
constexpr size_t kOffScenePairs = kOffExtent + 256;
constexpr size_t kScratchBytes = kOffScenePairs + up256(sizeof(unsigned long long));

// The scratch of every stq_sweep_static call on this device (about 4.5 MB).
static __device__ __align__(256) unsigned char g_static_scratch[kScratchBytes];

// Writes the scene's sizes into the header (zeroed by the host before this
// launch, so the NaN flag that any block may set is never cleared after it),
// the sort keys and the box indices, and the scene's extent on the two other
// axes: the largest ~key(min) and key(max) of each (zero before this launch).
__global__ void static_keys_kernel(const stq_aabb *__restrict__ boxes, int n, int axis,
                                   unsigned char *scratch) {
  after_previous();
  BatchHeader *hdr = reinterpret_cast<BatchHeader *>(scratch + kOffHdr);
  uint32_t *keys = reinterpret_cast<uint32_t *>(scratch + kOffKeys0);
  uint32_t *vals = reinterpret_cast<uint32_t *>(scratch + kOffVals0);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    hdr->n_boxes = n;
    hdr->n_scenes = 1;
    hdr->replicas = unsigned(n);
    hdr->cells = 1;
    hdr->length = unsigned(n);
  }
  bool nan = false;
  uint32_t ext[4] = {0u, 0u, 0u, 0u};
  if (i < n) {
    const stq_aabb &b = boxes[i];
    for (int k = 0; k < 3; ++k) nan |= (b.min[k] != b.min[k]) | (b.max[k] != b.max[k]);
    keys[i] = float_key(b.min[axis]);
    vals[i] = uint32_t(i);
    const int bb = axis == 0 ? 1 : 0, cc = axis == 2 ? 1 : 2;
    ext[0] = ~float_key(b.min[bb]);
    ext[1] = ~float_key(b.min[cc]);
    ext[2] = float_key(b.max[bb]);
    ext[3] = float_key(b.max[cc]);
  }
  if (__any_sync(kFullMask, nan) && (threadIdx.x & 31) == 0) atomicOr(&hdr->flags, kFlagNaN);
  uint32_t *extent = reinterpret_cast<uint32_t *>(scratch + kOffExtent);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const uint32_t m = __reduce_max_sync(kFullMask, ext[e]);
    if ((threadIdx.x & 31) == 0) atomicMax(&extent[e], m);
  }
}

// Sorted positions 0..n-1 (one cell), then the NaN sentinel and the padding.
__global__ void static_gather_kernel(const stq_aabb *__restrict__ boxes, int n, int axis,
                                     const uint32_t *__restrict__ keys, const uint32_t *__restrict__ order,
                                     unsigned char *scratch) {
  after_previous();
  if (reinterpret_cast<const BatchHeader *>(scratch + kOffHdr)->fault) return;  // the boxes are not sorted
  float4 *yz = reinterpret_cast<float4 *>(scratch + kOffYz);
  float2 *xx = reinterpret_cast<float2 *>(scratch + kOffX);
  int4 *v = reinterpret_cast<int4 *>(scratch + kOffV);
  int *flag = reinterpret_cast<int *>(scratch + kOffFlag);
  uint32_t *scode = reinterpret_cast<uint32_t *>(scratch + kOffCode);
  int *partner = reinterpret_cast<int *>(scratch + kOffPartner);
  int *run_end = reinterpret_cast<int *>(scratch + kOffRunEnd);
  const uint32_t *extent = reinterpret_cast<const uint32_t *>(scratch + kOffExtent);
  const int b = axis == 0 ? 1 : 0, c = axis == 2 ? 1 : 2;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) {
    const stq_aabb &x = boxes[order[k]];
    yz[k] = make_float4(x.min[b], x.min[c], x.max[b], x.max[c]);
    xx[k] = make_float2(x.min[axis], x.max[axis]);
    v[k] = make_int4(x.vertex_ids[0], x.vertex_ids[1], x.vertex_ids[2], x.id);
    flag[k] = 3;  // one cell, one scene: every box is in its first cell
    const float ob = key_float(~extent[0]), oc = key_float(~extent[1]);
    const float lb = key_float(extent[2]) - ob, lc = key_float(extent[3]) - oc;
    const float sb = lb > 0.f && isfinite(lb) ? 64.f / lb : 0.f, sc = lc > 0.f && isfinite(lc) ? 64.f / lc : 0.f;
    scode[k] = code_pack(code_step(x.min[b], ob, sb, 0), code_step(x.min[c], oc, sc, 0), code_step(x.max[b], ob, sb, 0),
                         code_step(x.max[c], oc, sc, 0), false, false);
    partner[k] = k + 1;  // one list: candidates follow in sort order
    // one past the last minimum that is not above this maximum
    const uint32_t xk = float_key(x.max[axis]);
    int lo = k + 1, hi = n;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (keys[mid] <= xk) lo = mid + 1;
      else hi = mid;
    }
    run_end[k] = lo;
  } else if (k < n + 1 + kSortedPad) {
    partner[k] = k;
    run_end[k] = k;
  }
}

std::mutex g_mutex;
void *g_scratch_ptr[256] = {};  // per device, set at the first call on it

}  // namespace
}  // namespace stq

extern "C" int stq_sweep_static(const stq_aabb *d_boxes, int64_t n, int axis, stq_pair *d_pairs,
                                int64_t capacity, int64_t *count, int64_t *total, void *stream) {
  using namespace stq;
  if (!count || n < 0) return STQ_ERR_INVALID_ARG;
  if (n > kMax) return STQ_ERR_CAPACITY;  // larger scenes need stq_sweep
  if (axis < 0 || axis > 2 || capacity < 0 || (n > 0 && !d_boxes) || (capacity > 0 && !d_pairs))
    return STQ_ERR_INVALID_ARG;
  *count = 0;
  if (total) *total = 0;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 256) return STQ_ERR_CUDA;
  unsigned char *scratch = nullptr;
  {
    // host code must not use g_static_scratch's address directly: look it up
    // once per device, with that device current
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_scratch_ptr[dev] &&
        cudaGetSymbolAddress(&g_scratch_ptr[dev], g_static_scratch) != cudaSuccess) {
      g_scratch_ptr[dev] = nullptr;
      return STQ_ERR_CUDA;
    }
    scratch = static_cast<unsigned char *>(g_scratch_ptr[dev]);
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int ni = int(n);
  const int blocks = (ni + 1 + int(kSortedPad) + 255) / 256;
  // the header and the scene's pair counter start at zero (the array keeps
  // the last call's contents); a memset on the stream, not an allocation
  if (cudaMemsetAsync(scratch + kOffHdr, 0, kScratchBytes - kOffHdr, s) != cudaSuccess) return STQ_ERR_CUDA;
  launch_after(static_keys_kernel, (ni + 255) / 256 > 0 ? (ni + 255) / 256 : 1, 256, 0, s, d_boxes, ni, axis, scratch);
  uint32_t *kb[2] = {reinterpret_cast<uint32_t *>(scratch + kOffKeys0),
                     reinterpret_cast<uint32_t *>(scratch + kOffKeys1)};
  uint32_t *vb[2] = {reinterpret_cast<uint32_t *>(scratch + kOffVals0),
                     reinterpret_cast<uint32_t *>(scratch + kOffVals1)};
  BatchHeader *hdr = reinterpret_cast<BatchHeader *>(scratch + kOffHdr);
  if (radix_sort_u32(s, kb, vb, n, scratch + kOffSortWs, &hdr->fault, nullptr) != cudaSuccess)
    return STQ_ERR_CUDA;
  launch_after(static_gather_kernel, blocks, 256, 0, s, d_boxes, ni, axis, kb[0], vb[0], scratch);
  int num_sms = 152;
  cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
  SweepParams p;
  p.yz = reinterpret_cast<const float4 *>(scratch + kOffYz);
  p.x = reinterpret_cast<const float2 *>(scratch + kOffX);
  p.v = reinterpret_cast<const int4 *>(scratch + kOffV);
  p.flag = reinterpret_cast<const int *>(scratch + kOffFlag);
  p.scode = reinterpret_cast<const uint32_t *>(scratch + kOffCode);
  p.partner = reinterpret_cast<const int *>(scratch + kOffPartner);
  p.run_end = reinterpret_cast<const int *>(scratch + kOffRunEnd);
  p.begin = 0;
  p.end = ni;
  // start boxes per warp: 32 would leave warps without any (65,536 boxes are 2,048
  // warps of 32)
  p.chunk = 8;
  p.grabs = 0;
  p.pairs = d_pairs;
  p.capacity = capacity;
  p.count = &hdr->pairs;
  p.work = &hdr->work;
  p.box_counts = nullptr;
  p.scene_pairs = reinterpret_cast<unsigned long long *>(scratch + kOffScenePairs);
  p.hdr = hdr;
  p.stats = nullptr;
  p.typed = 0;  // one list of all box types
  p.run_cap = 512;
  p.sel = nullptr;
  p.long_list = reinterpret_cast<int2 *>(scratch + kOffLong);
  p.long_items = &hdr->long_items;
  p.long_work = &hdr->long_work;
  if (launch_sweep(s, p, SweepTuning(), kSweepEmit, num_sms) != cudaSuccess) return STQ_ERR_CUDA;
  BatchHeader h;
  if (cudaMemcpyAsync(&h, hdr, sizeof(BatchHeader), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return STQ_ERR_CUDA;
  if (h.flags & kFlagNaN) return STQ_ERR_INVALID_INPUT;
  if (h.fault) return STQ_ERR_TIMEOUT;
  const int64_t found = int64_t(h.pairs);
  if (total) *total = found;
  *count = found < capacity ? found : capacity;
  return found <= capacity ? STQ_OK : STQ_OVERFLOW;
}
