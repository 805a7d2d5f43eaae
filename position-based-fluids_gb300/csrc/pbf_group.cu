// Gather passes of the paper equations for scenes that do not fill the GPU:
// eight threads per particle.
//
// With one thread per particle (pbf_paper.cu) a pass over a small scene takes
// as long as one thread's walk of its list: about nine dependent rounds of
// loads for 33 neighbours, and nine rows of candidates in the list build,
// while most of the GPU idles.  Here the eight threads of a particle (four
// particles per warp) load all neighbours at once, evaluate a pair each, and
// put the pairs' terms in shared memory; then thread c of the eight sums
// component c over the pairs in list order.  A sum is therefore the same
// operations in the same order as the one-thread walk, and its bits are the
// same: only the components run side by side.  Shared memory is a warp's own
// (no CTA barrier anywhere).
//
// It costs about three times the instructions per particle, so it is the better
// form only while there are too few particles to keep the GPU busy: see
// kGroupParticles for the line and what both sides measured.  At 1,000
// particles (cold caches) the list build with the first lambda takes 8.3 us
// instead of 18.8, a delta-p pass 4.5 instead of 9.8, lambda 4.2 / 7.7,
// vorticity 4.4 / 9.7 and XSPH 4.2 / 9.4; an empty kernel takes 2.3.
#include "pbf_paper.cuh"

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
  static constexpr int kWords = kStride * kCtaParticles;
  static_assert(kStride >= kFloats * kRow && kRow % 4 == 0, "16-byte reads inside the region");
};

// A pair that is none contributes a * b with a = -0 and b = +0 (or the term
// -0) to every sum: x + (-0) is x, also for x = -0.
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
struct FirstEntries {
  uint2 j[kTwos];
  __device__ __forceinline__ FirstEntries(const NbrCtx &c, uint32_t k) {
    const uint32_t l = lane_of_group();
#pragma unroll
    for (int u = 0; u < kTwos; ++u) j[u] = two(c, k, 2u * ((uint32_t)u * kGroup + l));
  }
  __device__ __forceinline__ static uint2 two(const NbrCtx &c, uint32_t k, uint32_t e) {
    if (e >= c.maxn) return make_uint2(k, k);
    return __ldg(reinterpret_cast<const uint2 *>(&c.nbr4[(size_t)(e >> 2) * c.n + k]) +
                 (e >> 1 & 1u));
  }
  __device__ __forceinline__ uint2 get(const NbrCtx &c, uint32_t k, uint32_t base, int u,
                                       uint32_t e) const {
    return base == 0 ? j[u] : two(c, k, e);
  }
};

// ------------------------------------------------------------------ passes --
struct LambdaPass {
  const float4 *P;
  const PaperConsts &c;
  using Data = float4;
  static constexpr int kSums = 5, kFloats = 8;  // rho, g, s
  static constexpr bool kOnes = false;
  // rho += (poly6 t t) t; g += f r; s += (f f) r2
  __device__ __forceinline__ static int factor_a(int q) { return q == 0 ? 0 : (q == 4 ? 6 : 2); }
  __device__ __forceinline__ static int factor_b(int q) { return q == 0 ? 1 : (q == 4 ? 7 : 2 + q); }
  __device__ __forceinline__ float start(int q) const { return q == 0 ? c.w_self : 0.f; }
  __device__ __forceinline__ float4 load(uint32_t j) const { return __ldg(&P[j]); }
  __device__ __forceinline__ void pair(const float4 &pk, const float4 &pj, float (&v)[8]) const {
    const Sep r = separation(pk, pj);
    if (is_pair(r.r2, c.h2)) {
      const float t = __fsub_rn(c.h2, r.r2);
      const float f = spiky_factor(r.r2, c);
      v[0] = __fmul_rn(__fmul_rn(c.poly6, t), t);
      v[1] = t;
      v[2] = f;
      v[3] = r.x;
      v[4] = r.y;
      v[5] = r.z;
      v[6] = __fmul_rn(f, f);
      v[7] = r.r2;
    } else {
      v[0] = v[2] = v[6] = kNothing;
      v[1] = v[3] = v[4] = v[5] = v[7] = 0.f;
    }
  }
};

template <bool kTwelve>
struct DeltaPass {
  const float4 *Q;
  const PaperConsts &c;
  using Data = float4;
  static constexpr int kSums = 3, kFloats = 4;  // s += wgt r
  static constexpr bool kOnes = false;
  __device__ __forceinline__ static int factor_a(int) { return 0; }
  __device__ __forceinline__ static int factor_b(int q) { return 1 + q; }
  __device__ __forceinline__ float start(int) const { return 0.f; }
  __device__ __forceinline__ float4 load(uint32_t j) const { return __ldg(&Q[j]); }
  __device__ __forceinline__ void pair(const float4 &qk, const float4 &qj, float (&v)[4]) const {
    const Sep r = separation(qk, qj);
    const bool ok = is_pair(r.r2, c.h2);
    v[0] = ok ? delta_weight<kTwelve>(qk.w, qj.w, r.r2, c) : kNothing;
    v[1] = ok ? r.x : 0.f;
    v[2] = ok ? r.y : 0.f;
    v[3] = ok ? r.z : 0.f;
  }
};

struct VortPass {
  const float4 *P, *U;
  const PaperConsts &c;
  using Data = PU;
  // w += cross, s += g, x += wp u; the plain sums as 1 * term
  static constexpr int kSums = 9, kFloats = 10;
  static constexpr bool kOnes = true;
  __device__ __forceinline__ static int factor_a(int q) { return q < 6 ? -1 : 6; }
  __device__ __forceinline__ static int factor_b(int q) { return q < 6 ? q : 1 + q; }
  __device__ __forceinline__ float start(int) const { return 0.f; }
  __device__ __forceinline__ PU load(uint32_t j) const { return PU{__ldg(&P[j]), __ldg(&U[j])}; }
  __device__ __forceinline__ void pair(const PU &k, const PU &d, float (&v)[10]) const {
    const Sep r = separation(k.p, d.p);
    if (is_pair(r.r2, c.h2)) {
      const VortTerms t = vort_terms(r, k.u, d.u, c);
      v[0] = t.wx;
      v[1] = t.wy;
      v[2] = t.wz;
      v[3] = t.gx;
      v[4] = t.gy;
      v[5] = t.gz;
      v[6] = t.wp;
      v[7] = t.ux;
      v[8] = t.uy;
      v[9] = t.uz;
    } else {
#pragma unroll
      for (int q = 0; q < 7; ++q) v[q] = kNothing;
      v[7] = v[8] = v[9] = 0.f;
    }
  }
};

struct XsphPass {
  const float4 *PW;
  const PaperConsts &c;
  using Data = float4;
  static constexpr int kSums = 3, kFloats = 4;  // e += (f w) r
  static constexpr bool kOnes = false;
  __device__ __forceinline__ static int factor_a(int) { return 0; }
  __device__ __forceinline__ static int factor_b(int q) { return 1 + q; }
  __device__ __forceinline__ float start(int) const { return 0.f; }
  __device__ __forceinline__ float4 load(uint32_t j) const { return __ldg(&PW[j]); }
  __device__ __forceinline__ void pair(const float4 &pk, const float4 &pj, float (&v)[4]) const {
    const Sep r = separation(pk, pj);
    const bool ok = is_pair(r.r2, c.h2);
    v[0] = ok ? __fmul_rn(spiky_factor(r.r2, c), pj.w) : kNothing;
    v[1] = ok ? r.x : 0.f;
    v[2] = ok ? r.y : 0.f;
    v[3] = ok ? r.z : 0.f;
  }
};

// Particle of the calling thread's group; past the end the last particle,
// computed along (the warp stays whole) and not written.
struct GroupIndex {
  uint32_t k;
  bool writes;  // first thread of a particle's group
  __device__ __forceinline__ explicit GroupIndex(uint32_t n) {
    const uint32_t p = blockIdx.x * kCtaParticles + threadIdx.x / kGroup;
    k = min(p, n - 1u);
    writes = p < n && lane_of_group() == 0;
  }
};

// Sums of a pass over the list of particle k, or over the set re-derived from
// the cells (by every thread of the group alike) when the list does not hold it.
template <typename Pass, typename Own, typename Rederive>
__device__ __forceinline__ void list_sums(const Pass &pass, const Own &own, const NbrCtx &nc,
                                          uint32_t k, const FirstEntries &first, float *terms,
                                          float (&sum)[Pass::kSums], Rederive &&rederive) {
  const uint32_t cnt = load_own(&nc.cnt[k]);
  const bool listed = cnt <= nc.maxn;
  group_sums(pass, own, k, listed ? cnt : 0u,
             [&](uint32_t base, int u, uint32_t e) { return first.get(nc, k, base, u, e); }, terms,
             sum);
  if (!listed) rederive(sum);
}

__global__ void __launch_bounds__(kGroupThreads)
    k_group_lambda(const float4 *__restrict__ P, NbrCtx nc, PaperConsts c,
                   float4 *__restrict__ Q, float *__restrict__ R) {
  __shared__ __align__(16) float s_terms[Terms<8>::kWords];
  const GroupIndex g(c.n);
  const FirstEntries first(nc, g.k);
  const float4 pk = P[g.k];
  const LambdaPass pass{P, c};
  float s[5];
  list_sums(pass, pk, nc, g.k, first, s_terms + threadIdx.x / kGroup * Terms<8>::kStride, s,
            [&](float (&t)[5]) {
              LambdaAcc acc{c.w_self, 0.f, 0.f, 0.f, 0.f};
              visit_fallback(nc, g.k, [&](uint32_t j) { lambda_pair(acc, pk, __ldg(&P[j]), c); });
              t[0] = acc.rho;
              t[1] = acc.gx;
              t[2] = acc.gy;
              t[3] = acc.gz;
              t[4] = acc.s;
            });
  if (g.writes) lambda_commit(g.k, pk, LambdaAcc{s[0], s[1], s[2], s[3], s[4]}, c, Q, R);
}

template <bool kTwelve>
__global__ void __launch_bounds__(kGroupThreads)
    k_group_delta(const float4 *__restrict__ Q, NbrCtx nc, PaperConsts c,
                  float4 *__restrict__ D, float4 *__restrict__ P, const float *__restrict__ R,
                  float4 *__restrict__ U, int last) {
  __shared__ __align__(16) float s_terms[Terms<4>::kWords];
  const GroupIndex g(c.n);
  const FirstEntries first(nc, g.k);
  const float4 qk = Q[g.k];
  const float4 x = load_own(&nc.X2[g.k]), d0 = D[g.k];
  const float rho = R[g.k];
  const DeltaPass<kTwelve> pass{Q, c};
  float s[3];
  list_sums(pass, qk, nc, g.k, first, s_terms + threadIdx.x / kGroup * Terms<4>::kStride, s,
            [&](float (&t)[3]) {
              DeltaAcc acc{0.f, 0.f, 0.f};
              visit_fallback(nc, g.k, [&](uint32_t j) {
                acc.template pair<kTwelve>(qk, __ldg(&Q[j]), c);
              });
              t[0] = acc.sx;
              t[1] = acc.sy;
              t[2] = acc.sz;
            });
  if (g.writes)
    delta_store(g.k, DeltaAcc{s[0], s[1], s[2]}, x, d0, [&] { return rho; }, nc, c, D, P, U, last);
}

__global__ void __launch_bounds__(kGroupThreads)
    k_group_vorticity(const float4 *__restrict__ P, const float4 *__restrict__ U, NbrCtx nc,
                      PaperConsts c, float4 *__restrict__ Wo, float4 *__restrict__ PW,
                      float4 *__restrict__ XS, float4 *__restrict__ SS) {
  __shared__ __align__(16) float s_terms[Terms<10>::kWords];
  const GroupIndex g(c.n);
  const FirstEntries first(nc, g.k);
  const PU own{P[g.k], U[g.k]};
  const VortPass pass{P, U, c};
  float s[9];
  list_sums(pass, own, nc, g.k, first, s_terms + threadIdx.x / kGroup * Terms<10>::kStride, s,
            [&](float (&t)[9]) {
              VortAcc acc{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
              visit_fallback(nc, g.k, [&](uint32_t j) {
                acc.pair(own.p, own.u, PU{__ldg(&P[j]), __ldg(&U[j])}, c);
              });
              t[0] = acc.wx;
              t[1] = acc.wy;
              t[2] = acc.wz;
              t[3] = acc.sx;
              t[4] = acc.sy;
              t[5] = acc.sz;
              t[6] = acc.xx;
              t[7] = acc.xy;
              t[8] = acc.xz;
            });
  if (g.writes)
    vort_commit(g.k, own.p, own.u,
                VortAcc{s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7], s[8]}, Wo, PW, XS, SS);
}

__global__ void __launch_bounds__(kGroupThreads)
    k_group_xsph(const float4 *__restrict__ PW, const float4 *__restrict__ U,
                 const float4 *__restrict__ Wv, const float4 *__restrict__ XS,
                 const float4 *__restrict__ SS, NbrCtx nc, PaperConsts c,
                 const uint32_t *__restrict__ ID2, float4 *__restrict__ X,
                 float4 *__restrict__ V, uint32_t *__restrict__ ID) {
  __shared__ __align__(16) float s_terms[Terms<4>::kWords];
  const GroupIndex g(c.n);
  const FirstEntries first(nc, g.k);
  const float4 pk = PW[g.k];
  const float4 uk = load_own(&U[g.k]), wk = load_own(&Wv[g.k]), xs = load_own(&XS[g.k]),
               ss = load_own(&SS[g.k]);
  const float mass = nc.V2[g.k].w;
  const uint32_t id = load_own(&ID2[g.k]);
  const XsphPass pass{PW, c};
  float s[3];
  list_sums(pass, pk, nc, g.k, first, s_terms + threadIdx.x / kGroup * Terms<4>::kStride, s,
            [&](float (&t)[3]) {
              XsphAcc acc{0.f, 0.f, 0.f};
              visit_fallback(nc, g.k, [&](uint32_t j) { acc.pair(pk, __ldg(&PW[j]), c); });
              t[0] = acc.ex;
              t[1] = acc.ey;
              t[2] = acc.ez;
            });
  if (g.writes)
    xsph_store(g.k, pk, uk, wk, xs, ss, XsphAcc{s[0], s[1], s[2]}, c, mass, id, X, V, ID);
}

// ------------------------------------------------------------- list build --
constexpr int kBuildChunks = 2 * kGroup;  // masks of 32 candidates a group holds
constexpr int kBuildList = 64;            // members a group's shared list holds

// Neighbour lists and the first lambda, as k_nbr_lambda computes them: the
// eight threads of a particle test 32 candidates of a row at a time (four
// each, from the position planes), join their bits into the row's mask, and
// thread q keeps mask q; each thread then writes its masks' members to the
// shared list behind those of the masks before.  A set of more masks or
// members than the group holds is found by one thread, as k_nbr_lambda does.
__global__ void __launch_bounds__(kGroupThreads)
    k_group_nbr_lambda(const float4 *__restrict__ P, Planes planes, NbrCtx nc, PaperConsts c,
                       uint4 *__restrict__ nbr4, uint32_t *__restrict__ nbr_cnt,
                       float4 *__restrict__ Q, float *__restrict__ R) {
  __shared__ __align__(16) float s_terms[Terms<8>::kWords];
  __shared__ __align__(16) uint32_t s_list[kBuildList * kCtaParticles];
  const GroupIndex g(c.n);
  const uint32_t k = g.k, l = lane_of_group();
  uint32_t *list = s_list + threadIdx.x / kGroup * kBuildList;
  const float4 pk = P[k];
  const uint32_t key = nc.skeys[k];
  const SceneDesc &sc = scene_of(nc.scenes, nc.sid, k);
  const int nx = sc.ncell[0], ny = sc.ncell[1], nz = sc.ncell[2];
  const uint32_t local = key - sc.cell_base;
  const int cx = (int)(local % (uint32_t)nx);
  const uint32_t rest = local / (uint32_t)nx;
  const int cy = (int)(rest % (uint32_t)ny);
  const int cz = (int)(rest / (uint32_t)ny);
  const int x0 = cx > 0 ? cx - 1 : 0;
  const int x1 = cx + 1 < nx ? cx + 1 : nx - 1;
  // rows in (dz, dy) order: thread q holds the slots of row q, all hold row 8
  uint2 row[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int q = h == 0 ? (int)l : 8;
    const int y = cy + q % 3 - 1, z = cz + q / 3 - 1;
    row[h] = make_uint2(0u, 0u);
    if (y >= 0 && y < ny && z >= 0 && z < nz) {
      const uint32_t at =
          sc.cell_base + (uint32_t)nx * ((uint32_t)y + (uint32_t)ny * (uint32_t)z);
      row[h] = make_uint2(__ldg(&nc.off[at + x0]), __ldg(&nc.off[at + x1 + 1]));
    }
  }
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
        x[dy] = __ldg(planes.x + w);
        y[dy] = __ldg(planes.y + w);
        z[dy] = __ldg(planes.z + w);
      }
    }
#pragma unroll
    for (int dy = 0; dy < 3; ++dy) {
      const float low = dz * 3 + dy == 4 ? kMinPair2 : -1.f;  // r^2 > 0 in the own row only
      for (uint32_t c0 = a[dy] & ~3u; __any_sync(kAll, c0 < b[dy]); c0 += 32u) {
        const uint32_t j = c0 + 4u * l;
        uint32_t m = 0;
        if (j < b[dy]) {
          if (c0 > a[dy]) {
            x[dy] = __ldg(planes.x + (j >> 2));
            y[dy] = __ldg(planes.y + (j >> 2));
            z[dy] = __ldg(planes.z + (j >> 2));
          }
          m = four_mask<true>(x[dy], y[dy], z[dy], px, py, pz, low, c.h2);
          if (j < a[dy]) m &= ~0u >> (a[dy] - j);
          if (b[dy] - j < 4u) m &= ~(~0u >> (b[dy] - j));
          m >>= 4u * l;
        }
        m |= __shfl_xor_sync(kAll, m, 1);
        m |= __shfl_xor_sync(kAll, m, 2);
        m |= __shfl_xor_sync(kAll, m, 4);
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
  uint32_t cnt = all0 + __shfl_sync(kAll, s1, kGroup - 1, kGroup);
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
        list[at++] = mine[h].y - top;
      }
    }
    if (l < (0u - cnt & 3u)) list[cnt + l] = k;  // the last word's padding
  }
  __syncwarp();
  const bool live = blockIdx.x * kCtaParticles + threadIdx.x / kGroup < c.n;
  if (grouped && live)
    for (uint32_t w = l; 4u * w < min(cnt, c.maxn); w += kGroup)
      nbr4[(size_t)w * c.n + k] = *reinterpret_cast<const uint4 *>(list + 4u * w);
  const LambdaPass pass{P, c};
  float s[5];
  group_sums(pass, pk, k, grouped ? cnt : 0u, [&](uint32_t, int, uint32_t e) {
               return e < (uint32_t)kBuildList ? *reinterpret_cast<const uint2 *>(list + e)
                                               : make_uint2(k, k);
             },
             s_terms + threadIdx.x / kGroup * Terms<8>::kStride, s);
  if (g.writes) {
    LambdaAcc acc{s[0], s[1], s[2], s[3], s[4]};
    if (!grouped) {
      acc = LambdaAcc{c.w_self, 0.f, 0.f, 0.f, 0.f};
      cnt = scan_members_planes(pk, k, key, sc, nc.off, planes, c, [&](uint32_t w, const uint4 &j) {
        if (4u * w < c.maxn) nbr4[(size_t)w * c.n + k] = j;
        lambda_pair(acc, pk, __ldg(&P[j.x]), c);
        lambda_pair(acc, pk, __ldg(&P[j.y]), c);
        lambda_pair(acc, pk, __ldg(&P[j.z]), c);
        lambda_pair(acc, pk, __ldg(&P[j.w]), c);
      });
    }
    nbr_cnt[k] = cnt;
    record_count(nc.cnt_max, cnt);
    lambda_commit(k, pk, acc, c, Q, R);
  }
}

inline uint32_t group_ctas(uint32_t n) { return (n + kCtaParticles - 1) / kCtaParticles; }

}  // namespace

cudaError_t group_nbr_lambda(const DeviceState &d, const PaperConsts &c, const uint16_t *sid,
                             cudaStream_t st) {
  k_group_nbr_lambda<<<group_ctas(c.n), kGroupThreads, 0, st>>>(
      d.P, make_planes(d.W, c.n), make_ctx(d, c, sid), c, d.nbr, d.nbr_cnt, d.Q, d.R);
  return cudaGetLastError();
}

cudaError_t group_lambda(const DeviceState &d, const PaperConsts &c, const uint16_t *sid,
                         cudaStream_t st) {
  k_group_lambda<<<group_ctas(c.n), kGroupThreads, 0, st>>>(d.P, make_ctx(d, c, sid), c, d.Q, d.R);
  return cudaGetLastError();
}

cudaError_t group_delta(const DeviceState &d, const PaperConsts &c, const uint16_t *sid,
                        bool last, cudaStream_t st) {
  const auto kernel = c.scorr_n3 == 12 ? k_group_delta<true> : k_group_delta<false>;
  kernel<<<group_ctas(c.n), kGroupThreads, 0, st>>>(d.Q, make_ctx(d, c, sid), c, d.D, d.P, d.R,
                                                    d.U, last ? 1 : 0);
  return cudaGetLastError();
}

cudaError_t group_vorticity(const DeviceState &d, const PaperConsts &c, const uint16_t *sid,
                            cudaStream_t st) {
  k_group_vorticity<<<group_ctas(c.n), kGroupThreads, 0, st>>>(d.P, d.U, make_ctx(d, c, sid), c,
                                                               d.W, d.D, d.Q, d.S);
  return cudaGetLastError();
}

cudaError_t group_xsph_commit(const DeviceState &d, const PaperConsts &c, const uint16_t *sid,
                              cudaStream_t st) {
  k_group_xsph<<<group_ctas(c.n), kGroupThreads, 0, st>>>(d.D, d.U, d.W, d.Q, d.S,
                                                          make_ctx(d, c, sid), c, d.ID2, d.X, d.V,
                                                          d.ID);
  return cudaGetLastError();
}

}  // namespace pbf
