// Neighbour lists of both equation sets: how a pass walks a particle's listed
// neighbours and how a build scans a row of candidates.  Lists hold sorted
// slots, four per 16-byte word, word g of particle k at nbr4[g * n + k].
// nvcc only.
#pragma once

#include "pbf_device.cuh"

namespace pbf {
namespace {

// List words are read once per pass: load them without keeping them in L1
// and first in line for eviction from L2 (policy from l2_evict_first), so
// the caches keep the neighbour data that is re-read.
__device__ __forceinline__ uint64_t l2_evict_first() {
  uint64_t policy;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  return policy;
}
__device__ __forceinline__ uint4 load_list_word(const uint4 *p, uint64_t policy) {
  uint4 v;
  asm volatile(
      "ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p), "l"(policy));
  return v;
}

// A value only its own thread reads (once per pass): loaded without
// allocating in L1, so L1 keeps the neighbour data the CTA re-reads.
__device__ __forceinline__ float4 load_own(const float4 *p) {
  float4 v;
  asm volatile("ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t load_own(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.global.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float load_own(const float *p) {
  float v;
  asm volatile("ld.global.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}

// For the `cnt` listed neighbours of particle k, kBatch (4 or 8) at a time:
// the batch's list words, then load(slot) for every entry of the batch, then
// f(data) for each in list order -- the loads of a batch are in flight
// together, and the next batch's list words are loaded into registers while
// the current batch's neighbour data loads and computes.  The list build
// pads the last word with k's own slot and words past the count read as k:
// those entries are the particle itself, which every pass drops through the
// pair test (r^2 = 0), so no entry needs a bound or a count test.
template <int kBatch, typename Load, typename F>
__device__ __forceinline__ void for_each_listed(const uint4 *__restrict__ nbr4, uint32_t n,
                                                uint32_t k, uint32_t cnt, Load &&load, F &&f) {
  static_assert(kBatch % 4 == 0, "whole list words per batch");
  constexpr int kWords = kBatch / 4;
  const uint64_t pol = l2_evict_first();
  uint4 cur[kWords];
#pragma unroll
  for (int w = 0; w < kWords; ++w)
    cur[w] = (w == 0 || 4u * (uint32_t)w < cnt) ? load_list_word(&nbr4[(size_t)w * n + k], pol)
                                                : make_uint4(k, k, k, k);
  for (uint32_t e0 = 0; e0 < cnt; e0 += kBatch) {
    uint4 nxt[kWords];
#pragma unroll
    for (int w = 0; w < kWords; ++w) {
      const uint32_t g = (e0 >> 2) + (uint32_t)(kWords + w);
      nxt[w] = 4u * g < cnt ? load_list_word(&nbr4[(size_t)g * n + k], pol)
                            : make_uint4(k, k, k, k);
    }
    uint32_t slot[kBatch];
#pragma unroll
    for (int w = 0; w < kWords; ++w) {
      slot[4 * w + 0] = cur[w].x;
      slot[4 * w + 1] = cur[w].y;
      slot[4 * w + 2] = cur[w].z;
      slot[4 * w + 3] = cur[w].w;
    }
    decltype(load(0u)) data[kBatch];
#pragma unroll
    for (int e = 0; e < kBatch; ++e) data[e] = load(slot[e]);
#pragma unroll
    for (int e = 0; e < kBatch; ++e) f(data[e]);
#pragma unroll
    for (int w = 0; w < kWords; ++w) cur[w] = nxt[w];
  }
}

// Calls member(j) for every slot j of [a, b) with test(P[j]), ascending: the
// candidates are tested 32 at a time into a membership mask, then member runs
// for the mask's set bits.  Lanes of a warp test candidates of different
// cells, so member work inside the candidate loop would run for nearly every
// candidate (some lane of the warp has a member); here the candidate loop is
// the load, the test and one bit in every lane.
template <typename Test, typename Member>
__device__ __forceinline__ void scan_row_masked(const float4 *__restrict__ P, uint32_t a,
                                                uint32_t b, Test &&test, Member &&member) {
  for (uint32_t c0 = a; c0 < b; c0 += 32u) {
    const uint32_t c1 = min(c0 + 32u, b);
    uint32_t m = 0, bit = 1u;
    uint32_t j = c0;
    for (; j + 4u <= c1; j += 4, bit <<= 4) {
      const float4 *__restrict__ q = P + j;
      float4 d[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) d[e] = __ldg(q + e);
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (test(d[e])) m |= bit << e;
    }
    if (j < c1) {
      float4 d[3];
#pragma unroll
      for (int e = 0; e < 3; ++e) d[e] = __ldg(&P[min(j + e, c1 - 1u)]);
#pragma unroll
      for (int e = 0; e < 3; ++e)
        if (j + e < c1 && test(d[e])) m |= bit << e;
    }
    while (m) {
      const uint32_t e = (uint32_t)__ffs(m) - 1u;
      m &= m - 1u;
      member(c0 + e);
    }
  }
}

// Fills the rest of a listed set's last word with the particle's own slot
// (maxn is a multiple of 8, so the word is inside the list capacity).
__device__ __forceinline__ void pad_list(uint32_t *__restrict__ out, size_t stride,
                                         uint32_t cnt, uint32_t maxn, uint32_t k) {
  if (cnt <= maxn)
    for (uint32_t e = cnt; e & 3u; ++e) out[(size_t)(e >> 2) * stride + (e & 3u)] = k;
}

}  // namespace
}  // namespace pbf
