// stq_device.cuh - device-side primitives shared by the STQ kernels.
//
// Box layout, the exact outward rounding of the box builder, the order-
// preserving sort key, and the pair predicates of the reference
// (Ahdhn/broadphase-gpu src/aabb.cu:12-40, src/collision.cu:24-48).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

#include "../../include/stq_abi.h"

namespace stq {

static_assert(sizeof(stq_aabb) == 44, "stq_aabb must match stq::gpu::Aabb (44 B)");
static_assert(offsetof(stq_aabb, min) == 4 && offsetof(stq_aabb, max) == 16 &&
                  offsetof(stq_aabb, vertex_ids) == 28 && offsetof(stq_aabb, ref_id) == 40,
              "stq_aabb field offsets must match stq::gpu::Aabb");

constexpr unsigned kFullMask = 0xffffffffu;

// First statement of a kernel launched by launch_after: waits until the kernels
// before it have ended and their writes are seen. Also in blocks that return at
// once: a kernel that ended without the wait could end before those before it.
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Asks for the line of p in L2: for words that are first met by an atomic at a kernel's
// end, and may be in device memory.
__device__ __forceinline__ void want_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Padding after the last sentinel of a sorted scene, so that a lane group of
// up to 32 lanes may read past a run end without leaving the allocation.
constexpr int kSortedPad = 256;

// ---- IEEE next float, as the reference calls it -----------------------------
// nextafter_up(x) = nextafterf(x, x + FLT_MAX) and nextafter_down(x) =
// nextafterf(x, x - FLT_MAX) (src/aabb.cu:56-61, src/cpu/aabb.cpp:16-21).
// For finite x that is the adjacent float toward +inf / -inf; for infinite x
// the direction argument equals x and x is returned. Written on the bit
// pattern from the IEEE 754 definition of adjacent floats.
__host__ __device__ inline float ref_next_up(float x) {
  if (x != x) return x;                            // NaN
  if (x == INFINITY || x == -INFINITY) return x;   // y == x
  uint32_t b;
  memcpy(&b, &x, 4);
  if ((b & 0x7fffffffu) == 0) b = 1u;              // +-0 -> +min denormal
  else if (b & 0x80000000u) b -= 1u;               // negative: toward zero
  else b += 1u;                                    // positive: away from zero
  float r;
  memcpy(&r, &b, 4);
  return r;
}

__host__ __device__ inline float ref_next_down(float x) {
  if (x != x) return x;
  if (x == INFINITY || x == -INFINITY) return x;
  uint32_t b;
  memcpy(&b, &x, 4);
  if ((b & 0x7fffffffu) == 0) b = 0x80000001u;     // +-0 -> -min denormal
  else if (b & 0x80000000u) b += 1u;               // negative: away from zero
  else b -= 1u;                                    // positive: toward zero
  float r;
  memcpy(&r, &b, 4);
  return r;
}

// ---- order-preserving float -> uint32 key -----------------------------------
// Key order is float '<' order with -0 and +0 equal (both map to the key of
// +0), so key equality is float equality and bound searches on keys agree
// with the float tests of the sweep; NaN is rejected before sorting.
__device__ __forceinline__ uint32_t float_key(float f) {
  uint32_t b = __float_as_uint(f);
  if (b == 0x80000000u) b = 0u;
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// The float of a key (-0 comes back as +0).
__device__ __forceinline__ float key_float(uint32_t k) {
  const uint32_t b = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  return __uint_as_float(b);
}

// Cell coordinate of a bound: clamp(floor((v - origin) * inv), 0, n - 1),
// with round-to-nearest float steps. Each step is monotone non-decreasing in
// v, so a <= b implies cell(a) <= cell(b): a point inside a box's range has
// its cell inside the box's cell range.
__device__ __forceinline__ int cell_coord(float v, float origin, float inv, int n) {
  float t = __fmul_rn(__fsub_rn(v, origin), inv);
  t = fminf(fmaxf(t, 0.f), float(n - 1));
  return int(t);
}

// ---- position codes -----------------------------------------------------------
// A sorted position's code holds its box's y/z interval in its cell, in 64
// steps per axis, and whether the cell is not the box's first along b and c:
//   bits 0-5 lo_b | 7-12 lo_c | 14-19 63 - hi_b | 21-26 63 - hi_c | 28 nf_b | 30 nf_c
// Every field has a zero guard bit above it. For a start box with code A and a
// candidate with code B, every guard bit of code_start(A) - B is set exactly
// when hi_a >= lo_b and hi_b >= lo_a on both axes (in steps) and neither axis
// has the flag set in both: the fields of code_start(A) are 64 + hi_a, 64 + 63 -
// lo_a and 2 + 1 - nf_a, so that no field borrows. Steps are a monotone function
// of the bound, clamped to the cell, so boxes that overlap always pass: one
// subtraction and one test stand for six float comparisons, and the exact test
// is left to the pairs that pass.
constexpr uint32_t kCodeGuard = 0xa8102040u;
constexpr uint32_t kCodeNotFirst = 0x50000000u;

__host__ __device__ __forceinline__ uint32_t code_pack(uint32_t lo_b, uint32_t lo_c, uint32_t hi_b, uint32_t hi_c,
                                                       bool nf_b, bool nf_c) {
  return lo_b | lo_c << 7 | (63u - hi_b) << 14 | (63u - hi_c) << 21 | (nf_b ? 1u << 28 : 0u) | (nf_c ? 1u << 30 : 0u);
}
__host__ __device__ __forceinline__ uint32_t code_start(uint32_t c) {
  return ~((c >> 14 & 0x3fffu) | (c & 0x3fffu) << 14 | (c & 0xf0000000u));
}
__host__ __device__ __forceinline__ bool code_pass(uint32_t start, uint32_t cand) {
  return (~(start - cand) & kCodeGuard) == 0u;
}

// Step of a bound in cell `cell`: scale is steps (64 per cell) per unit length.
// Monotone in v (round-to-nearest steps, clamped; NaN, which only an infinite
// origin gives, counts as 0).
__device__ __forceinline__ uint32_t code_step(float v, float origin, float scale, int cell) {
  const float t = __fsub_rn(__fmul_rn(__fsub_rn(v, origin), scale), 64.f * float(cell));
  return uint32_t(fminf(fmaxf(t, 0.f), 63.f));
}

// ---- box type and pair filter ------------------------------------------------
// Type from the signs of vertexIds (src/aabb.cu:12-31): vertex {v,-v-1,-v-1}
// -> 0, edge {e0,e1,-e0-1} -> 1, face {f0,f1,f2} -> 2.
__device__ __forceinline__ int box_type(int v1, int v2) {
  return v2 >= 0 ? 2 : (v1 >= 0 ? 1 : 0);
}

// is_valid_pair (src/aabb.cu:33-40): V-F, F-V or E-E, i.e. types sum to 2.
__device__ __forceinline__ bool valid_pair(const int4 &a, const int4 &b) {
  return box_type(a.y, a.z) + box_type(b.y, b.z) == 2;
}

// covertex (src/collision.cu:44-48): any of the 9 id pairs equal.
__device__ __forceinline__ bool covertex(const int4 &a, const int4 &b) {
  return a.x == b.x || a.x == b.y || a.x == b.z || a.y == b.x || a.y == b.y ||
         a.y == b.z || a.z == b.x || a.z == b.y || a.z == b.z;
}

// does_collide(MiniBox) (src/collision.cu:38-42): inclusive overlap on the two
// non-sweep axes. Layout (min_b, min_c, max_b, max_c).
__device__ __forceinline__ bool overlap_bc(const float4 &a, const float4 &b) {
  return a.z >= b.x && a.x <= b.z && a.w >= b.y && a.y <= b.w;
}

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

}  // namespace stq
