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
#include <type_traits>

#include "pbf_group.cuh"
#include "pbf_paper.cuh"

namespace pbf {

namespace {

// ------------------------------------------------------------------ passes --
template <typename Mem>
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
  __device__ __forceinline__ float4 load(uint32_t j) const { return Mem::ld(&P[j]); }
  __device__ __forceinline__ void pair(const float4 &pk, const float4 &pj, float (&v)[8]) const {
    const Sep r = separation(pk, pj);
    const bool ok = is_pair(r.r2, c.h2);
    const float t = __fsub_rn(c.h2, r.r2);
    const float f = spiky_factor(r.r2, c);
    v[0] = ok ? __fmul_rn(__fmul_rn(c.poly6, t), t) : kNothing;
    v[1] = ok ? t : 0.f;
    v[2] = ok ? f : kNothing;
    v[3] = ok ? r.x : 0.f;
    v[4] = ok ? r.y : 0.f;
    v[5] = ok ? r.z : 0.f;
    v[6] = ok ? __fmul_rn(f, f) : kNothing;
    v[7] = ok ? r.r2 : 0.f;
  }
};

template <typename Mem, bool kTwelve>
struct DeltaPass {
  const float4 *Q;
  const PaperConsts &c;
  using Data = float4;
  static constexpr int kSums = 3, kFloats = 4;  // s += wgt r
  static constexpr bool kOnes = false;
  __device__ __forceinline__ static int factor_a(int) { return 0; }
  __device__ __forceinline__ static int factor_b(int q) { return 1 + q; }
  __device__ __forceinline__ float start(int) const { return 0.f; }
  __device__ __forceinline__ float4 load(uint32_t j) const { return Mem::ld(&Q[j]); }
  __device__ __forceinline__ void pair(const float4 &qk, const float4 &qj, float (&v)[4]) const {
    const Sep r = separation(qk, qj);
    const bool ok = is_pair(r.r2, c.h2);
    v[0] = ok ? delta_weight<kTwelve>(qk.w, qj.w, r.r2, c) : kNothing;
    v[1] = ok ? r.x : 0.f;
    v[2] = ok ? r.y : 0.f;
    v[3] = ok ? r.z : 0.f;
  }
};

template <typename Mem>
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
  __device__ __forceinline__ PU load(uint32_t j) const { return PU{Mem::ld(&P[j]), Mem::ld(&U[j])}; }
  __device__ __forceinline__ void pair(const PU &k, const PU &d, float (&v)[10]) const {
    const Sep r = separation(k.p, d.p);
    const bool ok = is_pair(r.r2, c.h2);
    const VortTerms t = vort_terms(r, k.u, d.u, c);
    v[0] = ok ? t.wx : kNothing;
    v[1] = ok ? t.wy : kNothing;
    v[2] = ok ? t.wz : kNothing;
    v[3] = ok ? t.gx : kNothing;
    v[4] = ok ? t.gy : kNothing;
    v[5] = ok ? t.gz : kNothing;
    v[6] = ok ? t.wp : kNothing;
    v[7] = ok ? t.ux : 0.f;
    v[8] = ok ? t.uy : 0.f;
    v[9] = ok ? t.uz : 0.f;
  }
};

template <typename Mem>
struct XsphPass {
  const float4 *PW;
  const PaperConsts &c;
  using Data = float4;
  static constexpr int kSums = 3, kFloats = 4;  // e += (f w) r
  static constexpr bool kOnes = false;
  __device__ __forceinline__ static int factor_a(int) { return 0; }
  __device__ __forceinline__ static int factor_b(int q) { return 1 + q; }
  __device__ __forceinline__ float start(int) const { return 0.f; }
  __device__ __forceinline__ float4 load(uint32_t j) const { return Mem::ld(&PW[j]); }
  __device__ __forceinline__ void pair(const float4 &pk, const float4 &pj, float (&v)[4]) const {
    const Sep r = separation(pk, pj);
    const bool ok = is_pair(r.r2, c.h2);
    v[0] = ok ? __fmul_rn(spiky_factor(r.r2, c), pj.w) : kNothing;
    v[1] = ok ? r.x : 0.f;
    v[2] = ok ? r.y : 0.f;
    v[3] = ok ? r.z : 0.f;
  }
};

template <typename Mem>
__device__ __forceinline__ void group_lambda_of(uint32_t p, const float4 *P, const NbrCtx &nc,
                                                const PaperConsts &c, float4 *Q, float *R,
                                                float *terms) {
  const GroupIndex g(p, c.n);
  const FirstEntries<Mem> first(nc, g.k);
  const float4 pk = Mem::ld(&P[g.k]);
  const LambdaPass<Mem> pass{P, c};
  float s[5];
  list_sums<Mem>(pass, pk, nc, g.k, first, terms, s, [&](float (&t)[5]) {
    LambdaAcc acc{c.w_self, 0.f, 0.f, 0.f, 0.f};
    visit_fallback<Mem>(nc, g.k, [&](uint32_t j) { lambda_pair(acc, pk, Mem::ld(&P[j]), c); });
    t[0] = acc.rho;
    t[1] = acc.gx;
    t[2] = acc.gy;
    t[3] = acc.gz;
    t[4] = acc.s;
  });
  if (g.writes) lambda_commit(g.k, pk, LambdaAcc{s[0], s[1], s[2], s[3], s[4]}, c, Q, R);
}

template <typename Mem, bool kTwelve>
__device__ __forceinline__ void group_delta_of(uint32_t p, const float4 *Q, const NbrCtx &nc,
                                               const PaperConsts &c, float4 *D, float4 *P,
                                               const float *R, float4 *U, int last, float *terms) {
  const GroupIndex g(p, c.n);
  const FirstEntries<Mem> first(nc, g.k);
  const float4 qk = Mem::ld(&Q[g.k]);
  const float4 x = load_own(&nc.X2[g.k]), d0 = load_own(&D[g.k]);
  const float rho = load_own(&R[g.k]);
  const DeltaPass<Mem, kTwelve> pass{Q, c};
  float s[3];
  list_sums<Mem>(pass, qk, nc, g.k, first, terms, s, [&](float (&t)[3]) {
    DeltaAcc acc{0.f, 0.f, 0.f};
    visit_fallback<Mem>(nc, g.k, [&](uint32_t j) {
      acc.template pair<kTwelve>(qk, Mem::ld(&Q[j]), c);
    });
    t[0] = acc.sx;
    t[1] = acc.sy;
    t[2] = acc.sz;
  });
  if (g.writes)
    delta_store(g.k, DeltaAcc{s[0], s[1], s[2]}, x, d0, [&] { return rho; }, nc, c, D, P, U, last);
}

template <typename Mem>
__device__ __forceinline__ void group_vorticity_of(uint32_t p, const float4 *P, const float4 *U,
                                                   const NbrCtx &nc, const PaperConsts &c,
                                                   float4 *Wo, float4 *PW, float4 *XS, float4 *SS,
                                                   float *terms) {
  const GroupIndex g(p, c.n);
  const FirstEntries<Mem> first(nc, g.k);
  const PU own{Mem::ld(&P[g.k]), Mem::ld(&U[g.k])};
  const VortPass<Mem> pass{P, U, c};
  float s[9];
  list_sums<Mem>(pass, own, nc, g.k, first, terms, s, [&](float (&t)[9]) {
    VortAcc acc{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    visit_fallback<Mem>(nc, g.k, [&](uint32_t j) {
      acc.pair(own.p, own.u, PU{Mem::ld(&P[j]), Mem::ld(&U[j])}, c);
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

template <typename Mem>
__device__ __forceinline__ void group_xsph_of(uint32_t p, const float4 *PW, const float4 *U,
                                              const float4 *Wv, const float4 *XS, const float4 *SS,
                                              const NbrCtx &nc, const PaperConsts &c,
                                              const uint32_t *ID2, float4 *X, float4 *V,
                                              uint32_t *ID, float *terms) {
  const GroupIndex g(p, c.n);
  const FirstEntries<Mem> first(nc, g.k);
  const float4 pk = Mem::ld(&PW[g.k]);
  const float4 uk = load_own(&U[g.k]), wk = load_own(&Wv[g.k]), xs = load_own(&XS[g.k]),
               ss = load_own(&SS[g.k]);
  const float mass = load_own(&nc.V2[g.k]).w;
  const uint32_t id = load_own(&ID2[g.k]);
  const XsphPass<Mem> pass{PW, c};
  float s[3];
  list_sums<Mem>(pass, pk, nc, g.k, first, terms, s, [&](float (&t)[3]) {
    XsphAcc acc{0.f, 0.f, 0.f};
    visit_fallback<Mem>(nc, g.k, [&](uint32_t j) { acc.pair(pk, Mem::ld(&PW[j]), c); });
    t[0] = acc.ex;
    t[1] = acc.ey;
    t[2] = acc.ez;
  });
  if (g.writes)
    xsph_store(g.k, pk, uk, wk, xs, ss, XsphAcc{s[0], s[1], s[2]}, c, mass, id, X, V, ID);
}

// ------------------------------------------------------------- list build --
// The neighbours of particle k in the 27 cells around cell `key`: only the row
// of its own cell can hold k itself or a coincident particle.
template <typename Mem, typename Entry>
__device__ __forceinline__ uint32_t group_scan(uint32_t k, const float4 &pk, uint32_t key,
                                               const SceneDesc &sc, const uint32_t *off,
                                               const Planes &planes, float h2, Entry *list) {
  const uint32_t l = lane_of_group();
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
      row[h] = make_uint2(Mem::ld(&off[at + x0]), Mem::ld(&off[at + x1 + 1]));
    }
  }
  return group_scan_rows<Mem, false>(k, pk, row, planes, kMinPair2, h2, list);
}

// Neighbour list and first lambda of particle p, as k_nbr_lambda computes them.
// A set that the group does not hold is found by one thread, as there.
template <typename Mem>
__device__ __forceinline__ void group_nbr_lambda_of(uint32_t p, const float4 *P,
                                                    const Planes &planes, const NbrCtx &nc,
                                                    const PaperConsts &c, uint4 *nbr4,
                                                    uint32_t *nbr_cnt, float4 *Q, float *R,
                                                    float *terms, uint32_t *list) {
  const GroupIndex g(p, c.n);
  const uint32_t k = g.k;
  const float4 pk = Mem::ld(&P[k]);
  const uint32_t key = Mem::ld(&nc.skeys[k]);
  const SceneDesc &sc = scene_of(nc.scenes, nc.sid, k);
  uint32_t cnt = group_scan<Mem>(k, pk, key, sc, nc.off, planes, c.h2, list);
  const bool grouped = cnt != kNotHeld;
  if (grouped && g.live)
    for (uint32_t w = lane_of_group(); 4u * w < min(cnt, c.maxn); w += kGroup)
      nbr4[(size_t)w * c.n + k] = *reinterpret_cast<const uint4 *>(list + 4u * w);
  const LambdaPass<Mem> pass{P, c};
  float s[5];
  group_sums(pass, pk, k, grouped ? cnt : 0u, [&](uint32_t, int, uint32_t e) {
               return e < (uint32_t)kBuildList ? *reinterpret_cast<const uint2 *>(list + e)
                                               : make_uint2(k, k);
             },
             terms, s);
  if (g.writes) {
    LambdaAcc acc{s[0], s[1], s[2], s[3], s[4]};
    if (!grouped) {
      acc = LambdaAcc{c.w_self, 0.f, 0.f, 0.f, 0.f};
      cnt = scan_members_planes<Mem, false>(pk, k, key, sc, nc.off, planes, c, [&](uint32_t w, const uint4 &j) {
        if (4u * w < c.maxn) nbr4[(size_t)w * c.n + k] = j;
        lambda_pair(acc, pk, Mem::ld(&P[j.x]), c);
        lambda_pair(acc, pk, Mem::ld(&P[j.y]), c);
        lambda_pair(acc, pk, Mem::ld(&P[j.z]), c);
        lambda_pair(acc, pk, Mem::ld(&P[j.w]), c);
      });
    }
    nbr_cnt[k] = cnt;
    record_count(nc.cnt_max, cnt);
    lambda_commit(k, pk, acc, c, Q, R);
  }
}

// ----------------------------------------------------------------- kernels --
__device__ __forceinline__ uint32_t cta_particle() {
  return blockIdx.x * kCtaParticles + threadIdx.x / kGroup;
}

__global__ void __launch_bounds__(kGroupThreads)
    k_group_nbr_lambda(const float4 *__restrict__ P, Planes planes, NbrCtx nc, PaperConsts c,
                       uint4 *__restrict__ nbr4, uint32_t *__restrict__ nbr_cnt,
                       float4 *__restrict__ Q, float *__restrict__ R) {
  __shared__ __align__(16) float s_terms[Terms<8>::kStride * kCtaParticles];
  __shared__ __align__(16) uint32_t s_list[kBuildList * kCtaParticles];
  const uint32_t g = threadIdx.x / kGroup;
  group_nbr_lambda_of<EarlierKernel>(cta_particle(), P, planes, nc, c, nbr4, nbr_cnt, Q, R,
                                     s_terms + g * Terms<8>::kStride, s_list + g * kBuildList);
}

__global__ void __launch_bounds__(kGroupThreads)
    k_group_lambda(const float4 *__restrict__ P, NbrCtx nc, PaperConsts c,
                   float4 *__restrict__ Q, float *__restrict__ R) {
  __shared__ __align__(16) float s_terms[Terms<8>::kStride * kCtaParticles];
  group_lambda_of<EarlierKernel>(cta_particle(), P, nc, c, Q, R,
                                 s_terms + threadIdx.x / kGroup * Terms<8>::kStride);
}

template <bool kTwelve>
__global__ void __launch_bounds__(kGroupThreads)
    k_group_delta(const float4 *__restrict__ Q, NbrCtx nc, PaperConsts c,
                  float4 *__restrict__ D, float4 *__restrict__ P, const float *__restrict__ R,
                  float4 *__restrict__ U, int last) {
  __shared__ __align__(16) float s_terms[Terms<4>::kStride * kCtaParticles];
  group_delta_of<EarlierKernel, kTwelve>(cta_particle(), Q, nc, c, D, P, R, U, last,
                                         s_terms + threadIdx.x / kGroup * Terms<4>::kStride);
}

__global__ void __launch_bounds__(kGroupThreads)
    k_group_vorticity(const float4 *__restrict__ P, const float4 *__restrict__ U, NbrCtx nc,
                      PaperConsts c, float4 *__restrict__ Wo, float4 *__restrict__ PW,
                      float4 *__restrict__ XS, float4 *__restrict__ SS) {
  __shared__ __align__(16) float s_terms[Terms<10>::kStride * kCtaParticles];
  group_vorticity_of<EarlierKernel>(cta_particle(), P, U, nc, c, Wo, PW, XS, SS,
                                    s_terms + threadIdx.x / kGroup * Terms<10>::kStride);
}

__global__ void __launch_bounds__(kGroupThreads)
    k_group_xsph(const float4 *__restrict__ PW, const float4 *__restrict__ U,
                 const float4 *__restrict__ Wv, const float4 *__restrict__ XS,
                 const float4 *__restrict__ SS, NbrCtx nc, PaperConsts c,
                 const uint32_t *__restrict__ ID2, float4 *__restrict__ X,
                 float4 *__restrict__ V, uint32_t *__restrict__ ID) {
  report_count(nc);
  __shared__ __align__(16) float s_terms[Terms<4>::kStride * kCtaParticles];
  group_xsph_of<EarlierKernel>(cta_particle(), PW, U, Wv, XS, SS, nc, c, ID2, X, V, ID,
                               s_terms + threadIdx.x / kGroup * Terms<4>::kStride);
}

// --------------------------------------------------------- a step at once --
// The whole step of a scene of up to 1,024 particles as one launch of one
// cluster: a group of eight threads per particle through all passes, and a
// cluster barrier where the step would end a launch.  A pass of such a scene
// waits on launches and first loads from L2 (1,000 particles: 14 launches, 43
// us) and, with the state in global memory between the barriers, still on L2 and
// on writes to reach it (46 us).  So every CTA holds what the passes gather --
// P or (P, lambda) or (p, |omega|/rho), and the velocities -- for all particles
// in its own shared memory; a particle's group keeps its own state in
// registers and writes each pass's value into every CTA's copy (distributed
// shared memory).  Every CTA sorts the scene for itself at the start, so the
// sort ends in shared memory as well.  1,000 particles: 36.9 us a step alone, and
// three such scenes at once 13.8 us a step where the launches allowed 20.  Of its
// 71,000 clocks the sort takes 6,700, the scan for neighbours 7,300, each pass
// about 3,400 (four warps per scheduler of some 450 instructions) and each
// barrier with the stores it waits for about 2,300.
constexpr int kTinyThreads = 512;
constexpr int kTinyGroups = kTinyThreads / kGroup;  // 64 per CTA
constexpr uint32_t kTinyMaxCtas = kTinyParticles / kTinyGroups;
constexpr int kTinyEach = (int)kTinyParticles / kTinyThreads;  // particles a thread sorts
constexpr int kTinyWarps = kTinyThreads / 32;
// Shared memory: the terms of 64 groups, three arrays of float4, cell offsets,
// lists (first the unordered places), the sorted slots' particles, every warp's
// largest count (of the whole cluster, in the first CTA).
constexpr uint32_t kTinyArray = kTinyParticles * sizeof(float4);
constexpr uint32_t kTinyA = kTinyGroups * Terms<10>::kStride * sizeof(float);
constexpr uint32_t kTinyB = kTinyA + kTinyArray;
constexpr uint32_t kTinyU = kTinyB + kTinyArray;
constexpr uint32_t kTinyOff = kTinyU + kTinyArray;
constexpr uint32_t kTinyList = kTinyOff + (kTinyCells + 4) / 4 * 16;
constexpr uint32_t kTinySrc = kTinyList + kTinyGroups * kBuildList * sizeof(uint16_t);
constexpr uint32_t kTinyMax = kTinySrc + kTinyParticles * sizeof(uint16_t);
constexpr uint32_t kTinySmem = kTinyMax + kTinyMaxCtas * kTinyWarps * sizeof(uint32_t);
static_assert(kTinySmem <= 227 * 1024, "fits an SM");
static_assert(kTinyGroups * kBuildList >= (int)kTinyParticles, "the places fit the lists");
static_assert(3 * kTinyParticles * sizeof(float) <= kTinyArray, "the planes fit the velocities");
static_assert(Terms<10>::kStride >= Terms<8>::kStride, "one stride for all passes");

struct TinyStep {
  NbrCtx nc;
  PaperConsts c;
  float4 *X, *V, *X2, *V2;
  float *R;
  uint32_t *ID, *skeys, *off, *nbr_cnt, *cnt_max;
  uint4 *nbr;
  uint32_t ncells, iterations;
};

// What a pass gathers, in the CTA's own shared memory.
struct OwnCopy {
  template <typename T>
  __device__ __forceinline__ static T ld(const T *p) {
    return *p;
  }
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// Every thread of the cluster; what was written before it is visible after it.
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t shared_address(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// The address of the caller's shared address in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t peer_address(uint32_t address, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(address), "r"(rank));
  return r;
}
// The CTA's particles' values into every CTA's copy of `array`: gathered in
// `stage`, then a warp for each CTA, its lanes' stores side by side.  (Each
// group's threads storing its own value to the CTAs in turn, 64 bytes to eight
// CTAs per instruction: 38.9 us a step instead of 36.9.)
__device__ __forceinline__ void store_copies(float4 *array, uint32_t first, uint32_t n,
                                             const float4 &v, float4 *stage) {
  if (lane_of_group() == 0) stage[threadIdx.x / kGroup] = v;
  __syncthreads();
  const uint32_t ctas = cluster_size(), lane = threadIdx.x & 31u;
  for (uint32_t r = threadIdx.x / 32u; r < ctas; r += kTinyWarps)
#pragma unroll
    for (uint32_t i = lane; i < (uint32_t)kTinyGroups; i += 32u) {
      if (first + i >= n) continue;
      const float4 w = stage[i];
      asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(
                       peer_address(shared_address(array + first + i), r)),
                   "f"(w.x), "f"(w.y), "f"(w.z), "f"(w.w)
                   : "memory");
    }
}

// Prediction and cell sort of the whole scene into the CTA's shared memory:
// cell offsets, predicted positions by slot (and as planes) and the particle
// of each slot -- what k_predict_count to k_reorder compute.  The first CTA
// also writes the arrays that outlive the passes or re-derive a set.
__device__ __forceinline__ void tiny_sort(const TinyStep &t, unsigned char *smem, bool writes) {
  uint32_t *s_off = reinterpret_cast<uint32_t *>(smem + kTinyOff);  // counts, then offsets
  uint16_t *s_place = reinterpret_cast<uint16_t *>(smem + kTinyList);
  uint16_t *s_src = reinterpret_cast<uint16_t *>(smem + kTinySrc);
  float4 *s_pos = reinterpret_cast<float4 *>(smem + kTinyA);
  float *planes = reinterpret_cast<float *>(smem + kTinyU);
  __shared__ uint32_t s_warp[kTinyWarps];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, n = t.c.n;
  const SceneDesc &sc = t.nc.scenes[0];
  float4 x[kTinyEach], v[kTinyEach];
  uint32_t key[kTinyEach], place[kTinyEach];
#pragma unroll
  for (int u = 0; u < kTinyEach; ++u) {
    const uint32_t k = (uint32_t)u * kTinyThreads + tid;
    if (k < n) {
      x[u] = t.X[k];
      v[u] = gravity_velocity(t.V[k], t.c.dt, t.c.gy);
    }
  }
  for (uint32_t i = tid; i <= t.ncells; i += kTinyThreads) s_off[i] = 0u;
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kTinyEach; ++u) {
    const uint32_t k = (uint32_t)u * kTinyThreads + tid;
    if (k < n) {
      const float3 p = add3(x[u], displacement(v[u], t.c.dt));
      key[u] = scene_cell(p.x, p.y, p.z, sc);
      place[u] = atomicAdd(&s_off[key[u]], 1u);
    }
  }
  __syncthreads();
  // exclusive scan: consecutive cells per thread, warps, CTA
  const uint32_t per = (t.ncells + kTinyThreads - 1u) / kTinyThreads;
  const uint32_t c0 = min(tid * per, t.ncells), c1 = min(c0 + per, t.ncells);
  uint32_t sum = 0;
  for (uint32_t c = c0; c < c1; ++c) sum += s_off[c];
  uint32_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t up = __shfl_up_sync(kAll, incl, o);
    if (lane >= (uint32_t)o) incl += up;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  uint32_t run = incl - sum;
  for (uint32_t w = 0; w < warp; ++w) run += s_warp[w];
  for (uint32_t c = c0; c < c1; ++c) {
    const uint32_t m = s_off[c];
    s_off[c] = run;
    run += m;
  }
  if (tid == 0) s_off[t.ncells] = n;
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kTinyEach; ++u) {
    const uint32_t k = (uint32_t)u * kTinyThreads + tid;
    if (k < n) s_place[s_off[key[u]] + place[u]] = (uint16_t)k;
  }
  if (writes)
    for (uint32_t c = tid; c <= t.ncells; c += kTinyThreads) t.off[c] = s_off[c];
  __syncthreads();
  const uint32_t plane = plane_floats(n);
#pragma unroll
  for (int u = 0; u < kTinyEach; ++u) {
    const uint32_t k = (uint32_t)u * kTinyThreads + tid;
    if (k >= n) continue;
    // the place in index order among the cell's particles
    const uint32_t a = s_off[key[u]], b = s_off[key[u] + 1u];
    uint32_t q = a;
    for (uint32_t i = a; i < b; ++i) q += s_place[i] < k ? 1u : 0u;
    const float3 p = add3(x[u], displacement(v[u], t.c.dt));
    s_src[q] = (uint16_t)k;
    s_pos[q] = make_float4(p.x, p.y, p.z, 0.0f);
    planes[q] = p.x;
    planes[plane + q] = p.y;
    planes[2u * plane + q] = p.z;
    if (writes) {
      t.X2[q] = x[u];
      t.V2[q] = v[u];
      t.skeys[q] = key[u];
    }
  }
  __syncthreads();
}

template <bool kTwelve>
__global__ void __launch_bounds__(kTinyThreads, 1) k_tiny_step(TinyStep t) {
  extern __shared__ __align__(16) unsigned char s_tiny[];
  cluster_arrive();  // waited for before the first store into another CTA
  const uint32_t rank = cluster_rank(), group = threadIdx.x / kGroup;
  const PaperConsts &c = t.c;
  __shared__ float4 s_stage[2][kTinyGroups];
  const uint32_t first = rank * (uint32_t)kTinyGroups;
  float *terms = reinterpret_cast<float *>(s_tiny) + group * Terms<10>::kStride;
  uint16_t *list = reinterpret_cast<uint16_t *>(s_tiny + kTinyList) + group * kBuildList;
  float4 *A = reinterpret_cast<float4 *>(s_tiny + kTinyA);
  float4 *B = reinterpret_cast<float4 *>(s_tiny + kTinyB);
  float4 *U = reinterpret_cast<float4 *>(s_tiny + kTinyU);
  const uint32_t *s_off = reinterpret_cast<const uint32_t *>(s_tiny + kTinyOff);
  uint32_t *s_max = reinterpret_cast<uint32_t *>(s_tiny + kTinyMax);
  tiny_sort(t, s_tiny, rank == 0);
  // the group's particle, by slot
  const GroupIndex g(rank * (uint32_t)kTinyGroups + group, c.n);
  const uint32_t k = g.k, src = reinterpret_cast<const uint16_t *>(s_tiny + kTinySrc)[k];
  const SceneDesc &sc = t.nc.scenes[0];
  const float4 x = t.X[src], v0 = t.V[src];
  const uint32_t id = t.ID[src];
  float3 d = displacement(gravity_velocity(v0, c.dt, c.gy), c.dt);
  float4 pk = A[k];
  const uint32_t words = plane_floats(c.n) / 4u;
  const Planes planes = {U, U + words, U + 2u * words};
  uint32_t cnt = group_scan<OwnCopy>(k, pk, scene_cell(pk.x, pk.y, pk.z, sc), sc, s_off, planes,
                                     c.h2, list);
  if (!g.live) cnt = 0;  // (the list of its last particle is another warp's to write)
  const bool held = cnt != kNotHeld;
  // a set that the list does not hold is found by every thread of the group alike
  // and listed in global memory, with the first lambda summed on the way; one that
  // is too large for that as well is re-derived in each pass, as visit_fallback does
  LambdaAcc all{c.w_self, 0.f, 0.f, 0.f, 0.f};
  if (!held)
    cnt = scan_members_planes<OwnCopy, false>(
        pk, k, scene_cell(pk.x, pk.y, pk.z, sc), sc, s_off, planes, c,
        [&](uint32_t w, const uint4 &j) {
          if (g.writes && 4u * w < c.maxn) t.nbr[(size_t)w * c.n + k] = j;
          lambda_pair(all, pk, A[j.x], c);
          lambda_pair(all, pk, A[j.y], c);
          lambda_pair(all, pk, A[j.z], c);
          lambda_pair(all, pk, A[j.w], c);
        });
  __syncwarp();
  if (g.writes) t.nbr_cnt[k] = cnt;
  const bool far = !held && cnt <= c.maxn;
  const uint32_t listed = held ? cnt : 0u;
  const auto two = [&](uint32_t, int, uint32_t e) {
    if (e >= (uint32_t)kBuildList) return make_uint2(k, k);
    const ushort2 j = *reinterpret_cast<const ushort2 *>(list + e);
    return make_uint2(j.x, j.y);
  };
  // Sums of a pass for the warps with a set that its list does not hold: the far
  // lists by their groups (apart from the others: one way to read both took 5% of
  // an ordinary step), the rest by walk(sum).  1,000 particles of some 150 members
  // 115 us a step; with the sets re-derived in every pass 908.
  const bool all_held = __all_sync(kAll, held);
  const auto unheld = [&](const auto &pass, const auto &own, auto &sum, auto &&walk) {
    std::remove_reference_t<decltype(sum)> f;
    group_sums(pass, own, k, far ? cnt : 0u, [&](uint32_t, int, uint32_t e) {
                 return FirstEntries<EarlierPhase>::two(t.nc, k, e);
               },
               terms, f);
    if (held) return;
    if (!far) walk(f);
    for (uint32_t i = 0; i < sizeof f / sizeof f[0]; ++i) sum[i] = f[i];
  };
  const uint32_t most = __reduce_max_sync(kAll, cnt);
  cluster_wait();  // every CTA of the cluster runs
  if ((threadIdx.x & 31u) == 0u)
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(peer_address(
                     shared_address(s_max + rank * kTinyWarps + threadIdx.x / 32u), 0u)),
                 "r"(most)
                 : "memory");
  float rho = 0.f, lambda = 0.f;
  for (uint32_t it = 0; it < t.iterations; ++it) {
    {  // lambda from the positions in A to (P, lambda) in B
      const LambdaPass<OwnCopy> pass{A, c};
      float s[5];
      group_sums(pass, pk, k, listed, two, terms, s);
      if (!all_held && it > 0)
        unheld(pass, pk, s, [&](float (&f)[5]) {
          LambdaAcc acc{c.w_self, 0.f, 0.f, 0.f, 0.f};
          visit_fallback<EarlierPhase>(t.nc, k,
                                       [&](uint32_t j) { lambda_pair(acc, pk, A[j], c); });
          f[0] = acc.rho;
          f[1] = acc.gx;
          f[2] = acc.gy;
          f[3] = acc.gz;
          f[4] = acc.s;
        });
      const LambdaAcc acc = held || it > 0 ? LambdaAcc{s[0], s[1], s[2], s[3], s[4]} : all;
      lambda = acc.lambda(c);
      rho = acc.rho;
      store_copies(B, first, c.n, make_float4(pk.x, pk.y, pk.z, lambda), s_stage[0]);
    }
    cluster_arrive();
    cluster_wait();
    if (it == 0 && rank == 0 && threadIdx.x < 32) {
      uint32_t m = 0;
      for (uint32_t i = threadIdx.x; i < cluster_size() * kTinyWarps; i += 32u)
        m = max(m, s_max[i]);
      m = __reduce_max_sync(kAll, m);
      if (threadIdx.x == 0) {
        *t.cnt_max = m;
        *t.nc.host_max = m;
      }
    }
    const float4 qk = make_float4(pk.x, pk.y, pk.z, lambda);
    {  // delta-p from (P, lambda) in B to the positions in A
      const DeltaPass<OwnCopy, kTwelve> pass{B, c};
      float s[3];
      group_sums(pass, qk, k, listed, two, terms, s);
      if (!all_held)
        unheld(pass, qk, s, [&](float (&f)[3]) {
          DeltaAcc acc{0.f, 0.f, 0.f};
          visit_fallback<EarlierPhase>(t.nc, k, [&](uint32_t j) {
            acc.template pair<kTwelve>(qk, B[j], c);
          });
          f[0] = acc.sx;
          f[1] = acc.sy;
          f[2] = acc.sz;
        });
      const DeltaAcc acc{s[0], s[1], s[2]};
      const Moved m = delta_moved(acc, x, make_float4(d.x, d.y, d.z, 0.f), sc, c);
      d = m.d;
      pk = make_float4(m.p.x, m.p.y, m.p.z, 0.f);
      store_copies(A, first, c.n, pk, s_stage[1]);
      if (it + 1u == t.iterations)
        store_copies(U, first, c.n, delta_velocity(d, rho, c), s_stage[0]);
    }
    cluster_arrive();
    cluster_wait();
  }
  if (g.writes) t.R[k] = rho;
  // vorticity from A and U; (p, |omega|/rho) to B
  const PU own{pk, U[k]};
  VortAcc w;
  {
    const VortPass<OwnCopy> pass{A, U, c};
    float s[9];
    group_sums(pass, own, k, listed, two, terms, s);
    if (!all_held)
      unheld(pass, own, s, [&](float (&f)[9]) {
        VortAcc acc{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        visit_fallback<EarlierPhase>(
            t.nc, k, [&](uint32_t j) { acc.pair(own.p, own.u, PU{A[j], U[j]}, c); });
        f[0] = acc.wx;
        f[1] = acc.wy;
        f[2] = acc.wz;
        f[3] = acc.sx;
        f[4] = acc.sy;
        f[5] = acc.sz;
        f[6] = acc.xx;
        f[7] = acc.xy;
        f[8] = acc.xz;
      });
    w = VortAcc{s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7], s[8]};
  }
  const float wn = norm3(w.wx, w.wy, w.wz);
  const float4 pw = make_float4(pk.x, pk.y, pk.z, __fmul_rn(wn, own.u.w));
  store_copies(B, first, c.n, pw, s_stage[1]);
  cluster_arrive();
  cluster_wait();  // the last stores into another CTA lie behind it
  XsphAcc e;
  {
    const XsphPass<OwnCopy> pass{B, c};
    float s[3];
    group_sums(pass, pw, k, listed, two, terms, s);
    if (!all_held)
      unheld(pass, pw, s, [&](float (&f)[3]) {
        XsphAcc acc{0.f, 0.f, 0.f};
        visit_fallback<EarlierPhase>(t.nc, k, [&](uint32_t j) { acc.pair(pw, B[j], c); });
        f[0] = acc.ex;
        f[1] = acc.ey;
        f[2] = acc.ez;
      });
    e = XsphAcc{s[0], s[1], s[2]};
  }
  if (g.writes)
    xsph_store(k, pw, own.u, make_float4(w.wx, w.wy, w.wz, wn),
               make_float4(w.xx, w.xy, w.xz, 0.f), make_float4(w.sx, w.sy, w.sz, 0.f), e, c, v0.w,
               id, t.X, t.V, t.ID);
}

using TinyKernel = void (*)(TinyStep);

cudaLaunchConfig_t tiny_config(uint32_t ctas, cudaLaunchAttribute *attr, cudaStream_t st) {
  cudaLaunchConfig_t cfg{};
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = ctas;
  attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kTinyThreads);
  cfg.dynamicSmemBytes = kTinySmem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
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

uint32_t tiny_cluster() {
  for (TinyKernel k : {(TinyKernel)k_tiny_step<true>, (TinyKernel)k_tiny_step<false>}) {
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTinySmem) !=
            cudaSuccess ||
        cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
            cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
  }
  // 16 CTAs where the device places such a cluster, else the portable 8
  for (uint32_t size : {kTinyMaxCtas, 8u}) {
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = tiny_config(size, &attr, nullptr);
    int a = 0, b = 0;
    if (cudaOccupancyMaxActiveClusters(&a, k_tiny_step<true>, &cfg) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&b, k_tiny_step<false>, &cfg) == cudaSuccess && a > 0 &&
        b > 0)
      return size * (uint32_t)kTinyGroups;
    cudaGetLastError();
  }
  return 0;
}

cudaError_t tiny_step(const DeviceState &d, const PaperConsts &c, uint32_t ncells,
                      uint32_t iterations, cudaStream_t st) {
  TinyStep t;
  t.nc = make_ctx(d, c, nullptr);
  t.c = c;
  t.X = d.X;
  t.V = d.V;
  t.X2 = d.X2;
  t.V2 = d.V2;
  t.R = d.R;
  t.ID = d.ID;
  t.skeys = d.skeys;
  t.off = d.offsets;
  t.nbr_cnt = d.nbr_cnt;
  t.cnt_max = d.nbr_max;
  t.nbr = d.nbr;
  t.ncells = ncells;
  t.iterations = iterations;
  // as many CTAs as the particles need, a power of two of them
  uint32_t ctas = 1;
  while (ctas * (uint32_t)kTinyGroups < c.n) ctas *= 2;
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = tiny_config(ctas, &attr, st);
  return c.scorr_n3 == 12 ? cudaLaunchKernelEx(&cfg, k_tiny_step<true>, t)
                          : cudaLaunchKernelEx(&cfg, k_tiny_step<false>, t);
}

}  // namespace pbf
