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

// How a pass loads what it gathers: through the read-only path when an earlier
// kernel wrote it, from L2 when an earlier phase of the same kernel did.
struct EarlierKernel {
  template <typename T>
  __device__ __forceinline__ static T ld(const T *p) {
    return __ldg(p);
  }
};
struct EarlierPhase {
  template <typename T>
  __device__ __forceinline__ static T ld(const T *p) {
    return __ldcg(p);
  }
};

// Positions as three planes (x, y, z), four values per 16-byte word, each plane
// padded to whole words: the list builds test four candidates per three loads
// in 23 instructions (12 of them packed), where the scalar test of one float4
// candidate and its mask bit took about 11 each.  The builds are bound by L1's
// data path (79% busy: 128 bytes to the lanes per clock), so the planes' 12
// bytes per candidate instead of 16 count as much as the instructions.
// Measured at 1,048,576 particles: fused paper build + lambda 260 -> 196 us,
// ref-compat build 226 -> 157 us.
struct Planes {
  const float4 *x, *y, *z;
};
inline Planes make_planes(const float4 *planes, uint32_t n) {
  const size_t words = plane_floats(n) / 4u;
  return Planes{planes, planes + words, planes + 2 * words};
}

// r^2 of two candidates per packed instruction (add/mul/fma.rn.f32x2: each
// half rounded as the scalar instruction rounds it, so these are the squared
// distances separation() gives; (q - p)^2 = (p - q)^2 exactly).
__device__ __forceinline__ float2 packed_r2(float2 x, float2 y, float2 z) {
  return __ffma2_rn(z, z, __ffma2_rn(y, y, __fmul2_rn(x, x)));
}

// Bits 31 - e, e < 4: candidate e of the words has low <= r^2 < h2.
template <bool kLow>
__device__ __forceinline__ uint32_t four_mask(const float4 &x, const float4 &y, const float4 &z,
                                              float2 nx, float2 ny, float2 nz, float low,
                                              float h2) {
  const float2 r01 = packed_r2(__fadd2_rn(make_float2(x.x, x.y), nx),
                               __fadd2_rn(make_float2(y.x, y.y), ny),
                               __fadd2_rn(make_float2(z.x, z.y), nz));
  const float2 r23 = packed_r2(__fadd2_rn(make_float2(x.z, x.w), nx),
                               __fadd2_rn(make_float2(y.z, y.w), ny),
                               __fadd2_rn(make_float2(z.z, z.w), nz));
  const float r[4] = {r01.x, r01.y, r23.x, r23.y};
  uint32_t m = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e)
    if ((!kLow || r[e] >= low) && r[e] < h2) m |= 0x80000000u >> e;
  return m;
}

// Bit 31 - e of the result: candidate c0 + e of [a, b) has low <= r^2 < h2
// (kLow) or r^2 < h2.  c0 is a multiple of 4, less than b, and a - c0 < 32.
template <bool kLow, typename Mem = EarlierKernel>
__device__ __forceinline__ uint32_t row_mask(const Planes &p, uint32_t c0, uint32_t a, uint32_t b,
                                             float2 nx, float2 ny, float2 nz, float low,
                                             float h2) {
  const uint32_t w0 = c0 >> 2;
  uint32_t m = 0;
#pragma unroll
  for (uint32_t g = 0; g < 8; ++g) {
    if (c0 + 4u * g >= b) break;
    const float4 x = Mem::ld(p.x + w0 + g), y = Mem::ld(p.y + w0 + g), z = Mem::ld(p.z + w0 + g);
    m |= four_mask<kLow>(x, y, z, nx, ny, nz, low, h2) >> (4 * g);
  }
  if (a > c0) m &= ~0u >> (a - c0);
  if (b - c0 < 32u) m &= ~(~0u >> (b - c0));
  return m;
}

// A particle's members on their way to its list: the masks found so far
// (nonempty ones, with their first candidate), walked member by member into
// whole list words.  Each lane walks its own masks, so a warp takes as many
// rounds as its longest set, not as the longest of every row in turn; and a
// word leaves as one 16-byte store (stored one by one, a warp's members went
// to L2 as 4-byte writes 16 bytes apart, a sector each).  The queue is indexed
// at run time, so it lives in local memory, in L1; a column of shared memory
// per thread measured the same alone, but its carve-out took L1 away from the
// gather passes of other simulations' streams (three 1,048,576-particle scenes
// at once: 2.02 ms a frame against 1.54).
//
// In crowded scenes the queue has to make room several times.  The lanes of a
// warp (kWarp) do that together, as soon as one of them has to: each alone in its
// turn, the rest of the warp waiting, made the fused build of 64,000 particles
// with 185 members each 320 us instead of 98, and steps of a 262,144-particle
// REF_COMPAT run with 46 particles in a cell 7.7 ms instead of 3.1.  So every lane
// takes part in every row and chunk, with empty ones where it has none.
template <int kCap>
struct MaskQueue {
  uint2 chunk[kCap];     // (mask, first candidate + 31)
  uint32_t chunks = 0;   // masks held
  uint32_t members = 0;  // members in them
  uint32_t words = 0;    // list words handed on

  // The row of candidates [a, b), in chunks of 32: adds the members that mask(c0)
  // finds from c0 on; word(w, slots) takes word w of the list whenever the queue
  // has to make room.  kWarp: all 32 lanes call it alike.
  template <bool kWarp, typename Mask, typename Word>
  __device__ __forceinline__ void add_row(uint32_t a, uint32_t b, Mask &&mask, Word &&word) {
    for (uint32_t c0 = a & ~3u;; c0 += 32u) {
      const uint32_t m = c0 < b ? mask(c0) : 0u;
      if (m != 0u) {
        chunk[chunks++] = make_uint2(m, c0 + 31u);
        members += (uint32_t)__popc(m);
      }
      const bool full = chunks == (uint32_t)kCap;
      if (!any<kWarp>(full || c0 + 32u < b)) break;  // most rows: one vote
      if (any<kWarp>(full)) drain(word);
    }
  }
  template <bool kWarp>
  __device__ __forceinline__ static bool any(bool mine) {
    return kWarp ? __any_sync(0xffffffffu, mine) : mine;
  }
  // Members added so far.
  __device__ __forceinline__ uint32_t count() const { return 4u * words + members; }
  // Hands on every whole word; at most three members stay.
  template <typename Word>
  __device__ __forceinline__ void drain(Word &&word) {
    uint32_t at = 0;
    uint2 c = chunks ? chunk[0] : make_uint2(0u, 0u);
    for (; members >= 4u; members -= 4u) {
      uint32_t j[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) j[e] = next(c, at);
      word(words++, make_uint4(j[0], j[1], j[2], j[3]));
    }
    uint32_t kept = 0;
    if (c.x) chunk[kept++] = c;
    while (++at < chunks) chunk[kept++] = chunk[at];
    chunks = kept;
  }
  // Every member left; the last word is filled up with `self`.
  template <typename Word>
  __device__ __forceinline__ void finish(uint32_t self, Word &&word) {
    uint32_t at = 0;
    uint2 c = members ? chunk[0] : make_uint2(0u, 0u);
    for (int left = (int)members; left > 0; left -= 4) {
      uint32_t j[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) j[e] = left > e ? next(c, at) : self;
      word(words++, make_uint4(j[0], j[1], j[2], j[3]));
    }
  }
  // The next member of the masks from `c`, chunk `at` (there is one).
  __device__ __forceinline__ uint32_t next(uint2 &c, uint32_t &at) const {
    if (c.x == 0u) c = chunk[++at];
    const uint32_t top = 31u - (uint32_t)__clz((int)c.x);
    c.x ^= 1u << top;
    return c.y - top;
  }
};
// Masks a list build holds: nine rows of three cells, some of them over 32
// candidates.
constexpr int kMaskQueue = 14;

// Fills the rest of a listed set's last word with the particle's own slot
// (maxn is a multiple of 8, so the word is inside the list capacity).
__device__ __forceinline__ void pad_list(uint32_t *__restrict__ out, size_t stride,
                                         uint32_t cnt, uint32_t maxn, uint32_t k) {
  if (cnt <= maxn)
    for (uint32_t e = cnt; e & 3u; ++e) out[(size_t)(e >> 2) * stride + (e & 3u)] = k;
}

}  // namespace
}  // namespace pbf
