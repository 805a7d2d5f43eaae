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

// Counts kKeys keys per lane (whole warp) into counts[] for the counting sort,
// all their atomics in flight together: one atomic per run of equal keys in
// neighbouring lanes; pos[i] = the particle's place among the increments of
// its cell (a group's lanes in order, groups in atomic order).
// kScattered: keys in any order, so a warp in which some lanes 2, 4, 8 or 16 apart
// hold the same key joins all equal ones: the atomics on one word wait for each
// other, about 1 ns each.  1M random keys of 2 cells are counted in 24 us (a run at
// a time 181), of 8 cells 22 (125), 4.2M of which half are the same 192 (288), 4.2M
// nearly in order 23 (31; all warps through __match_any_sync, a round per distinct
// key, 33).  A step's kernels count by runs alone: with so many particles per cell
// its passes over the pairs take a thousand times as long.
template <bool kScattered, int kKeys>
__device__ __forceinline__ void count_cell_keys(const uint32_t (&key)[kKeys],
                                                const bool (&valid)[kKeys],
                                                const uint32_t (&i)[kKeys],
                                                uint32_t *__restrict__ counts,
                                                uint32_t *__restrict__ pos) {
  constexpr unsigned kWarp = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31u;
  unsigned group[kKeys];  // lanes counted by one atomic, the caller among them
  uint32_t base[kKeys];
#pragma unroll
  for (int u = 0; u < kKeys; ++u) {
    const uint32_t before = __shfl_up_sync(kWarp, key[u], 1);
    const bool valid_before = __shfl_up_sync(kWarp, (int)valid[u], 1);
    const unsigned heads =
        __ballot_sync(kWarp, lane == 0u || key[u] != before || valid[u] != valid_before);
    // the caller's run: from the last head at or below its lane to the next one
    const unsigned below = kWarp >> (31u - lane);
    const uint32_t head = 31u - (uint32_t)__clz((int)(heads & below));
    const unsigned later = heads & ~below;
    const uint32_t end = later ? (uint32_t)__ffs((int)later) - 1u : 32u;
    group[u] = kWarp >> (32u - (end - head)) << head;
    if (kScattered && __popc(heads) > 4) {
      bool apart = false;  // the caller's key in another run
#pragma unroll
      for (uint32_t o = 2; o <= 16; o <<= 1) {
        const uint32_t other = __shfl_xor_sync(kWarp, key[u], (int)o);  // every lane
        apart |= other == key[u] && !(group[u] >> (lane ^ o) & 1u);
      }
      if (__any_sync(kWarp, apart)) group[u] = __match_any_sync(kWarp, valid[u] ? key[u] : kWarp);
    }
    base[u] = 0;
    if (valid[u] && lane == (uint32_t)__ffs((int)group[u]) - 1u)
      base[u] = atomicAdd(&counts[key[u]], (uint32_t)__popc(group[u]));
  }
#pragma unroll
  for (int u = 0; u < kKeys; ++u) {
    const uint32_t first = __shfl_sync(kWarp, base[u], __ffs((int)group[u]) - 1);
    if (valid[u]) pos[i[u]] = first + (uint32_t)__popc(group[u] & ((1u << lane) - 1u));
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
