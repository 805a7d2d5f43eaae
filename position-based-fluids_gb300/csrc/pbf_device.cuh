// Device helpers shared by the CUDA translation units (nvcc only).
#pragma once

#include "pbf_internal.cuh"

namespace pbf {

// Device helpers used by several translation units.
__device__ __forceinline__ int axis_cell(float p, float mn, float cl, int n) {
  // trunc((p - min) / cell_length) as the reference's (int) cast, clamped.
  const int c = __float2int_rz(__fdiv_rn(__fsub_rn(p, mn), cl));
  return c < 0 ? 0 : (c >= n ? n - 1 : c);
}

__device__ __forceinline__ uint32_t scene_cell(float x, float y, float z,
                                               const SceneDesc &s) {
  const int cx = axis_cell(x, s.gmin[0], s.clen[0], s.ncell[0]);
  const int cy = axis_cell(y, s.gmin[1], s.clen[1], s.ncell[1]);
  const int cz = axis_cell(z, s.gmin[2], s.clen[2], s.ncell[2]);
  return (uint32_t)cx +
         (uint32_t)s.ncell[0] * ((uint32_t)cy + (uint32_t)s.ncell[1] * (uint32_t)cz);
}

// One key per lane (whole warp; invalid lanes count nothing) into the per-pass
// digit histograms in shared memory (digit_bits wide, pass p's at
// p << digit_bits): one addition where the warp's keys agree in the digit --
// the upper digits of keys that are nearly in order -- and one per key
// otherwise.  (Grouping equal digits with __match_any_sync instead cost more
// than all the rest of the histogram: 21 us of 1M keys' 82 us sort, now 6.5.)
__device__ __forceinline__ void warp_digit_histogram(uint32_t key, bool valid,
                                                     uint32_t passes, uint32_t digit_bits,
                                                     uint32_t *s_hist) {
  const uint32_t mask = (1u << digit_bits) - 1u;
  const unsigned lanes = __ballot_sync(0xffffffffu, valid);
  if (lanes == 0u) return;
  const uint32_t first = __shfl_sync(0xffffffffu, key, __ffs(lanes) - 1);
  for (uint32_t p = 0; p < passes; ++p) {
    const uint32_t shift = p * digit_bits;
    const uint32_t d = key >> shift & mask, d0 = first >> shift & mask;
    if (__all_sync(0xffffffffu, !valid || d == d0)) {
      if ((threadIdx.x & 31u) == 0u)
        atomicAdd(&s_hist[(p << digit_bits) + d0], (uint32_t)__popc(lanes));
    } else if (valid) {
      atomicAdd(&s_hist[(p << digit_bits) + d], 1u);
    }
  }
}

// Counts a warp's keys (four per lane, key u of the lane's particle i + u * step;
// bit u of `valid`) with one atomic for all lanes of the same key, if more than
// kManyApart lanes see their key again 16, 18 or 20 lanes on; returns whether it
// did, the same in every lane.  The atomics on one word wait for each other, about
// 1 ns each: 1M random keys of 2 cells 181 us by runs and 24 joined, of 8 cells 125
// and 22, 4.2M of which half are the same 878 and 196.  Keys that a warp hardly
// repeats are better left to the runs, as __match_any_sync takes a round per
// distinct one (4.2M nearly in order 28 and 20 us: 3 such lanes on average; keys of
// 64 cells too, which the rule leaves at 253 us for 171); and one test for all four
// keys leaves their atomics together (a test per key: the 4.2M-particle scene's
// hashes 18 us instead of 12).
constexpr uint32_t kManyApart = 8;  // of four keys' lanes
__device__ __forceinline__ bool count_joined(uint4 keys, uint32_t valid, uint32_t i,
                                             uint32_t step, uint32_t *__restrict__ counts,
                                             uint32_t *__restrict__ pos) {
  constexpr unsigned kWarp = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t key[4] = {keys.x, keys.y, keys.z, keys.w};
  uint32_t apart = 0;  // lanes whose key another lane holds
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    bool again = false;
#pragma unroll
    for (const uint32_t o : {16u, 18u, 20u}) {
      const uint32_t other = __shfl_down_sync(kWarp, key[u], o);  // every lane
      again |= other == key[u] && lane + o < 32u;
    }
    apart += (uint32_t)__popc(__ballot_sync(kWarp, again));
  }
  if (apart <= kManyApart) return false;
  unsigned same[4];
  uint32_t base[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const bool counts_here = valid >> u & 1u;
    same[u] = __match_any_sync(kWarp, counts_here ? key[u] : kWarp);
    base[u] = 0;
    if (counts_here && lane == (uint32_t)__ffs((int)same[u]) - 1u)
      base[u] = atomicAdd(&counts[key[u]], (uint32_t)__popc(same[u]));
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const uint32_t first = __shfl_sync(kWarp, base[u], __ffs((int)same[u]) - 1);
    if (valid >> u & 1u)
      pos[i + (uint32_t)u * step] = first + (uint32_t)__popc(same[u] & ((1u << lane) - 1u));
  }
  return true;
}

// Counts kKeys keys per lane (whole warp) into counts[] for the counting sort,
// all their atomics in flight together: one atomic per run of equal keys in
// neighbouring lanes; pos[i] = the particle's place among the increments of
// its cell (a run's lanes in order, runs in atomic order).
// kScattered (four keys, equally far apart): keys in any order, so warps of more
// than kManyRuns runs per key look for lanes to join; the 4.2M-particle scene's
// hashes have 10 runs.  (A step's kernels count by runs alone: with so many
// particles per cell its passes over the pairs take a thousand times as long.)
constexpr uint32_t kManyRuns = 12;  // of a warp's 32 keys
template <bool kScattered, int kKeys>
__device__ __forceinline__ void count_cell_keys(const uint32_t (&key)[kKeys],
                                                const bool (&valid)[kKeys],
                                                const uint32_t (&i)[kKeys],
                                                uint32_t *__restrict__ counts,
                                                uint32_t *__restrict__ pos) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t head[kKeys], end[kKeys], base[kKeys], runs = 0;
#pragma unroll
  for (int u = 0; u < kKeys; ++u) {
    const uint32_t before = __shfl_up_sync(0xffffffffu, key[u], 1);
    const bool valid_before = __shfl_up_sync(0xffffffffu, (int)valid[u], 1);
    const unsigned heads =
        __ballot_sync(0xffffffffu, lane == 0u || key[u] != before || valid[u] != valid_before);
    // the caller's run: from the last head at or below its lane to the next one
    const unsigned below = 0xffffffffu >> (31u - lane);
    head[u] = 31u - (uint32_t)__clz((int)(heads & below));
    const unsigned later = heads & ~below;
    end[u] = later ? (uint32_t)__ffs((int)later) - 1u : 32u;
    runs += (uint32_t)__popc(heads);
  }
  if constexpr (kScattered) {
    static_assert(kKeys == 4, "as count_joined takes them");
    if (runs > kManyRuns * kKeys) {
      const uint32_t bits = (valid[0] ? 1u : 0u) | (valid[1] ? 2u : 0u) | (valid[2] ? 4u : 0u) |
                            (valid[3] ? 8u : 0u);
      if (count_joined(make_uint4(key[0], key[1], key[2], key[3]), bits, i[0], i[1] - i[0], counts,
                       pos))
        return;
    }
  }
#pragma unroll
  for (int u = 0; u < kKeys; ++u) {
    base[u] = 0;
    if (valid[u] && lane == head[u]) base[u] = atomicAdd(&counts[key[u]], end[u] - head[u]);
  }
#pragma unroll
  for (int u = 0; u < kKeys; ++u) {
    const uint32_t first = __shfl_sync(0xffffffffu, base[u], (int)head[u]);
    if (valid[u]) pos[i[u]] = first + (lane - head[u]);
  }
}
// Keys a thread takes at a time in the counting, predicting and scattering
// kernels of large arrays, which wait on their loads and atomics: 4.2M keys
// counted in 12 us instead of 18, scattered in 14 instead of 20.
constexpr int kCountKeys = 4;

// Slot of the particle in unordered slot q once its cell is back in index
// order: cells of up to rank_cell particles are left as the scatter placed
// them, and each particle finds its place by counting the smaller indices
// (larger cells are already in order: k_cell_fix_big).
__device__ __forceinline__ uint32_t ordered_slot(const uint32_t *__restrict__ perm,
                                                 const uint32_t *__restrict__ off, uint32_t key,
                                                 uint32_t q, uint32_t index, uint32_t n,
                                                 uint32_t rank_cell) {
  const uint32_t a = __ldg(&off[key]), b = min(__ldg(&off[key + 1]), n);
  if (b - a > rank_cell || a > q) return q;  // (a <= q < b unless the sort reported an error)
  uint32_t rank = 0;
  for (uint32_t t = a; t < b; ++t) rank += perm[t] < index ? 1u : 0u;
  return min(a + rank, n - 1u);
}

}  // namespace pbf
