// Gather passes with eight threads per particle: what both equation sets share
// (pbf_group.cu has the reasons and figures).  nvcc only.
#pragma once

#include "pbf_lists.cuh"

namespace pbf {
namespace {

constexpr int kGroup = 8;                       // threads per particle
constexpr int kGroupThreads = 128;              // threads per CTA
constexpr int kCtaParticles = kGroupThreads / kGroup;
constexpr int kTwos = 3;                        // pairs of list entries per thread and round
constexpr int kRoundPairs = 2 * kGroup * kTwos; // list entries per particle and round (48)
constexpr unsigned kAll = 0xffffffffu;

// One particle's terms of a round: kFloats rows, one value of every pair in
// list order per row.  The row length puts the rows that the group's threads
// sum at the same time in different banks (four values each), the stride from
// particle to particle the two particles of a half warp that write together.
template <int kFloats>
struct Terms {
  static constexpr int kRow = kRoundPairs + 4;  // 52: 20 banks on per row
  static constexpr int kStride = (kFloats * kRow + 15) / 32 * 32 + 16;
  static_assert(kStride >= kFloats * kRow && kRow % 4 == 0, "16-byte reads inside the region");
};

// A pair that is none contributes a * b with a = -0 and b = +0 (or the term
// -0) to every sum: x + (-0) is x, also for x = -0.  (Its values are computed
// and selected away, not branched around: a warp's time is the latency of its
// instructions here, and the pairs of a thread then run side by side.)
constexpr float kNothing = -0.0f;

__device__ __forceinline__ uint32_t lane_of_group() { return threadIdx.x & (kGroup - 1); }

// Sums of the pass `Pass` over the listed pairs of particle k, each component
// in list order, in every thread of the group.  two(base, u, e) holds list
// entries e and e + 1 (e even; entries from cnt on are not used), the thread's
// u-th two of the round at `base`.  All 32 threads of the warp call it.
template <typename Pass, typename Own, typename Two>
__device__ __forceinline__ void group_sums(const Pass &pass, const Own &own, uint32_t k,
                                           uint32_t cnt, Two &&two, float *terms,
                                           float (&sum)[Pass::kSums]) {
  constexpr int kFloats = Pass::kFloats, kRow = Terms<kFloats>::kRow;
  constexpr int kMine = (Pass::kSums + kGroup - 1) / kGroup;  // components per thread
  const uint32_t l = lane_of_group();
  float acc[kMine];
  int ia[kMine], ib[kMine];  // rows of the two factors; no row: the factor 1
#pragma unroll
  for (int s = 0; s < kMine; ++s) {
    const int c = min((int)l + s * kGroup, Pass::kSums - 1);
    ia[s] = Pass::factor_a(c);
    ib[s] = Pass::factor_b(c);
    acc[s] = pass.start(c);
  }
  const uint32_t most = __reduce_max_sync(kAll, cnt);
  for (uint32_t base = 0; base < most; base += kRoundPairs) {
    typename Pass::Data data[2 * kTwos];
#pragma unroll
    for (int u = 0; u < kTwos; ++u) {
      const uint32_t e = base + 2u * ((uint32_t)u * kGroup + l);
      const uint2 j = two(base, u, e);
      data[2 * u] = pass.load(e < cnt ? j.x : k);  // k itself: not a pair
      data[2 * u + 1] = pass.load(e + 1u < cnt ? j.y : k);
    }
#pragma unroll
    for (int u = 0; u < kTwos; ++u) {
      float v[2][kFloats];
      pass.pair(own, data[2 * u], v[0]);
      pass.pair(own, data[2 * u + 1], v[1]);
      float *at = terms + 2u * ((uint32_t)u * kGroup + l);
#pragma unroll
      for (int q = 0; q < kFloats; ++q)
        *reinterpret_cast<float2 *>(at + q * kRow) = make_float2(v[0][q], v[1][q]);
    }
    __syncwarp();
    const uint32_t here = cnt > base ? min(cnt - base, (uint32_t)kRoundPairs) : 0u;
#pragma unroll 2
    for (uint32_t e = 0; e < here; e += 4) {  // entries past the last pair hold nothing
#pragma unroll
      for (int s = 0; s < kMine; ++s) {
        const float4 x = Pass::kOnes && ia[s] < 0
                             ? make_float4(1.f, 1.f, 1.f, 1.f)
                             : *reinterpret_cast<const float4 *>(terms + ia[s] * kRow + e);
        const float4 y = *reinterpret_cast<const float4 *>(terms + ib[s] * kRow + e);
        acc[s] = __fmaf_rn(x.x, y.x, acc[s]);
        acc[s] = __fmaf_rn(x.y, y.y, acc[s]);
        acc[s] = __fmaf_rn(x.z, y.z, acc[s]);
        acc[s] = __fmaf_rn(x.w, y.w, acc[s]);
      }
    }
    __syncwarp();
  }
#pragma unroll
  for (int c = 0; c < Pass::kSums; ++c)
    sum[c] = __shfl_sync(kAll, acc[c / kGroup], c % kGroup, kGroup);
}

// A thread's list entries of the first round, loaded without waiting for the
// count (entries past it are whatever the list last held there, and unused).
template <typename Mem>
struct FirstEntries {
  uint2 j[kTwos];
  // c: nbr4, n and maxn of the lists (NbrCtx, RefLists)
  template <typename Lists>
  __device__ __forceinline__ FirstEntries(const Lists &c, uint32_t k) {
    const uint32_t l = lane_of_group();
#pragma unroll
    for (int u = 0; u < kTwos; ++u) j[u] = two(c, k, 2u * ((uint32_t)u * kGroup + l));
  }
  template <typename Lists>
  __device__ __forceinline__ static uint2 two(const Lists &c, uint32_t k, uint32_t e) {
    if (e >= c.maxn) return make_uint2(k, k);
    return Mem::ld(reinterpret_cast<const uint2 *>(&c.nbr4[(size_t)(e >> 2) * c.n + k]) +
                   (e >> 1 & 1u));
  }
  template <typename Lists>
  __device__ __forceinline__ uint2 get(const Lists &c, uint32_t k, uint32_t base, int u,
                                       uint32_t e) const {
    return base == 0 ? j[u] : two(c, k, e);
  }
};

// Particle p of the calling thread's group; past the end the last particle,
// computed along (the warp stays whole) and not written.
struct GroupIndex {
  uint32_t k;
  bool live, writes;  // writes: first thread of a particle's group
  __device__ __forceinline__ GroupIndex(uint32_t p, uint32_t n) {
    k = min(p, n - 1u);
    live = p < n;
    writes = live && lane_of_group() == 0;
  }
};

// Sums of a pass over the list of particle k, or over the set re-derived from
// the cells (by every thread of the group alike) when the list does not hold it.
template <typename Mem, typename Pass, typename Own, typename Lists, typename Rederive>
__device__ __forceinline__ void list_sums(const Pass &pass, const Own &own, const Lists &nc,
                                          uint32_t k, const FirstEntries<Mem> &first,
                                          float *terms, float (&sum)[Pass::kSums],
                                          Rederive &&rederive) {
  const uint32_t cnt = load_own(&nc.cnt[k]);
  const bool listed = cnt <= nc.maxn;
  group_sums(pass, own, k, listed ? cnt : 0u,
             [&](uint32_t base, int u, uint32_t e) { return first.get(nc, k, base, u, e); }, terms,
             sum);
  if (!listed) rederive(sum);
}

constexpr int kBuildChunks = 2 * kGroup;  // masks of 32 candidates a group holds
constexpr int kBuildList = 64;            // members a group's shared list holds

// The members of nine rows of slots for particle k (position pk) into the
// group's shared list of kBuildList entries, in row and slot order, the last
// four filled up with k.  Row q is [row[0].x, row[0].y) of the group's thread
// q, row 8 is row[1] of every thread.  A member has r^2 < h2 and, in row 4,
// r^2 >= low; kBySlot leaves out k itself by its slot.  The eight threads test
// 32 candidates of a row at a time (four each, from the position planes), join
// their bits into the row's mask, and thread q keeps mask q; each thread then
// writes its masks' members behind those of the masks before.  Returns their
// number, or kNotHeld when there are more masks or members than the group
// holds.  All 32 threads of the warp call it.
constexpr uint32_t kNotHeld = 0xffffffffu;
template <typename Mem, bool kBySlot, typename Entry>
__device__ __forceinline__ uint32_t group_scan_rows(uint32_t k, const float4 &pk,
                                                    const uint2 (&row)[2], const Planes &planes,
                                                    float low, float h2, Entry *list) {
  const uint32_t l = lane_of_group();
  const float2 px = make_float2(-pk.x, -pk.x), py = make_float2(-pk.y, -pk.y),
               pz = make_float2(-pk.z, -pk.z);
  uint32_t chunks = 0;
  uint2 mine[2] = {make_uint2(0u, 0u), make_uint2(0u, 0u)};  // (mask, first candidate + 31)
  for (int dz = 0; dz < 3; ++dz) {
    uint32_t a[3], b[3];
    float4 x[3], y[3], z[3];
#pragma unroll
    for (int dy = 0; dy < 3; ++dy) {  // the three rows' first candidates in flight together
      const int q = dz * 3 + dy;
      a[dy] = q < 8 ? __shfl_sync(kAll, row[0].x, q, kGroup) : row[1].x;
      b[dy] = q < 8 ? __shfl_sync(kAll, row[0].y, q, kGroup) : row[1].y;
      const uint32_t w = (a[dy] >> 2) + l;
      if (4u * w < b[dy]) {
        x[dy] = Mem::ld(planes.x + w);
        y[dy] = Mem::ld(planes.y + w);
        z[dy] = Mem::ld(planes.z + w);
      }
    }
#pragma unroll
    for (int dy = 0; dy < 3; ++dy) {
      const float least = dz * 3 + dy == 4 ? low : -1.f;
      for (uint32_t c0 = a[dy] & ~3u; __any_sync(kAll, c0 < b[dy]); c0 += 32u) {
        const uint32_t j = c0 + 4u * l;
        uint32_t m = 0;
        if (j < b[dy]) {
          if (c0 > a[dy]) {
            x[dy] = Mem::ld(planes.x + (j >> 2));
            y[dy] = Mem::ld(planes.y + (j >> 2));
            z[dy] = Mem::ld(planes.z + (j >> 2));
          }
          m = four_mask<true>(x[dy], y[dy], z[dy], px, py, pz, least, h2);
          if (j < a[dy]) m &= ~0u >> (a[dy] - j);
          if (b[dy] - j < 4u) m &= ~(~0u >> (b[dy] - j));
          m >>= 4u * l;
        }
        m |= __shfl_xor_sync(kAll, m, 1);
        m |= __shfl_xor_sync(kAll, m, 2);
        m |= __shfl_xor_sync(kAll, m, 4);
        if (kBySlot && k - c0 < 32u) m &= ~(0x80000000u >> (k - c0));
        if (m != 0u) {  // the same in the group's eight threads
          if (chunks == l) mine[0] = make_uint2(m, c0 + 31u);
          if (chunks == l + kGroup) mine[1] = make_uint2(m, c0 + 31u);
          ++chunks;
        }
      }
    }
  }
  // members before each thread's masks
  const uint32_t n0 = (uint32_t)__popc(mine[0].x), n1 = (uint32_t)__popc(mine[1].x);
  uint32_t s0 = n0, s1 = n1;
#pragma unroll
  for (int o = 1; o < kGroup; o <<= 1) {
    const uint32_t t0 = __shfl_up_sync(kAll, s0, o, kGroup), t1 = __shfl_up_sync(kAll, s1, o, kGroup);
    if (l >= (uint32_t)o) {
      s0 += t0;
      s1 += t1;
    }
  }
  const uint32_t all0 = __shfl_sync(kAll, s0, kGroup - 1, kGroup);
  const uint32_t cnt = all0 + __shfl_sync(kAll, s1, kGroup - 1, kGroup);
  const bool grouped = chunks <= (uint32_t)kBuildChunks && cnt <= (uint32_t)kBuildList;
  if (grouped) {
    uint32_t at = s0 - n0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (h == 1) at = all0 + s1 - n1;
      uint32_t m = mine[h].x;
      while (m) {
        const uint32_t top = 31u - (uint32_t)__clz((int)m);
        m ^= 1u << top;
        list[at++] = (Entry)(mine[h].y - top);
      }
    }
    if (l < (0u - cnt & 3u)) list[cnt + l] = (Entry)k;  // the last word's padding
  }
  __syncwarp();
  return grouped ? cnt : kNotHeld;
}

}  // namespace
}  // namespace pbf
