// Device code shared by the gather passes of the paper equations
// (PBF_MODE_PAPER): the neighbour walks, the pair arithmetic of every pass
// and each pass's per-particle epilogue.  Both launch paths include it -- the
// passes that gather neighbours through L1 (pbf_paper.cu) and the passes that
// stage each tile's neighbourhood in shared memory (pbf_tile.cu) -- so a
// particle's arithmetic is the same operations in the same order whichever
// path runs it, and the two give the same bits.  nvcc only.
#pragma once

#include <type_traits>

#include "pbf_lists.cuh"

namespace pbf {
namespace {

struct NbrCtx {
  const uint4 *__restrict__ nbr4;
  const uint32_t *__restrict__ cnt;
  const uint32_t *__restrict__ skeys;
  const uint32_t *__restrict__ off;
  const float4 *__restrict__ X2;
  const float4 *__restrict__ V2;
  const SceneDesc *__restrict__ scenes;
  const uint16_t *__restrict__ sid;
  uint32_t *err;
  uint32_t *cnt_max;   // largest neighbour count of the step (may be null)
  uint32_t *host_max;  // where the host reads it (may be null)
  uint32_t n, maxn;
  float dt, h2;
};

// Folds the neighbour counts of the calling warp's active threads into the
// step's largest count: one atomic per warp.
__device__ __forceinline__ void record_count(uint32_t *cnt_max, uint32_t cnt) {
  const unsigned m = __activemask();
  const uint32_t mx = __reduce_max_sync(m, cnt);
  if (cnt_max && (threadIdx.x & 31u) == (unsigned)(__ffs(m) - 1)) atomicMax(cnt_max, mx);
}

// The step's last kernel: its largest count to the host.
__device__ __forceinline__ void report_count(const NbrCtx &c) {
  if (c.host_max && blockIdx.x == 0 && threadIdx.x == 0) *c.host_max = *c.cnt_max;
}

__device__ __forceinline__ const SceneDesc &scene_of(const SceneDesc *scenes,
                                                     const uint16_t *sid,
                                                     uint32_t k) {
  return scenes[sid ? sid[k] : 0];
}

// v' = v + dt g;  d = dt v';  p = x + d  -- rounded op by op (no
// contraction) so that every kernel that recomputes them gets the same bits.
__device__ __forceinline__ float4 gravity_velocity(float4 v, float dt, float gy) {
  v.y = __fadd_rn(v.y, __fmul_rn(dt, gy));
  return v;
}
__device__ __forceinline__ float3 displacement(float4 v1, float dt) {
  return make_float3(__fmul_rn(dt, v1.x), __fmul_rn(dt, v1.y), __fmul_rn(dt, v1.z));
}
__device__ __forceinline__ float3 add3(float4 x, float3 d) {
  return make_float3(__fadd_rn(x.x, d.x), __fadd_rn(x.y, d.y), __fadd_rn(x.z, d.z));
}

// Step-start predicted position of slot j (as written by the reorder).
template <typename Mem = EarlierKernel>
__device__ __forceinline__ float3 start_position(const NbrCtx &c, uint32_t j) {
  return add3(Mem::ld(&c.X2[j]), displacement(Mem::ld(&c.V2[j]), c.dt));
}

// Particles j != k closer than h form a pair.  Distances below
// sqrt(FLT_MIN) ~ 1.1e-19 count as coincident (like r = 0, whose direction
// is undefined), so r^2 is a normal number wherever a kernel is evaluated.
constexpr float kMinPair2 = 1.17549435e-38f;
__device__ __forceinline__ bool is_pair(float r2, float h2) {
  return r2 >= kMinPair2 && r2 < h2;
}

// All arithmetic on pair and particle values below is written with
// explicitly rounded operations (__fadd_rn, __fmul_rn, __fmaf_rn, ...): the
// compiler may not contract or reassociate them, so every kernel that
// evaluates a pair -- fused or not, any launch shape, staged or through L1 --
// rounds it the same way and gets the same bits.  (Left to itself, nvcc
// contracts a*b + c*d into an FMA on either product, and its choice can
// differ from one kernel to another.)
struct Sep {
  float x, y, z, r2;  // p_k - p_j and its squared length
};
__device__ __forceinline__ Sep separation(const float4 &a, const float4 &b) {
  Sep r;
  r.x = __fsub_rn(a.x, b.x);
  r.y = __fsub_rn(a.y, b.y);
  r.z = __fsub_rn(a.z, b.z);
  r.r2 = __fmaf_rn(r.z, r.z, __fmaf_rn(r.y, r.y, __fmul_rn(r.x, r.x)));
  return r;
}
__device__ __forceinline__ Sep separation(const float3 &a, const float3 &b) {
  return separation(make_float4(a.x, a.y, a.z, 0.f), make_float4(b.x, b.y, b.z, 0.f));
}

// Visits the 9 rows around the cell with key `key` (order: dz, dy, slot);
// f(q, j) gets the row index q = (dz+1)*3 + (dy+1) and the slot j != k.
template <typename Mem = EarlierKernel, typename F>
__device__ __forceinline__ void scan_rows(uint32_t k, uint32_t key, const SceneDesc &s,
                                          const uint32_t *__restrict__ off, F &&f) {
  const int nx = s.ncell[0], ny = s.ncell[1], nz = s.ncell[2];
  const uint32_t local = key - s.cell_base;
  const int cx = (int)(local % (uint32_t)nx);
  const uint32_t t = local / (uint32_t)nx;
  const int cy = (int)(t % (uint32_t)ny);
  const int cz = (int)(t / (uint32_t)ny);
  const int x0 = cx > 0 ? cx - 1 : 0;
  const int x1 = cx + 1 < nx ? cx + 1 : nx - 1;
  for (int dz = -1; dz <= 1; ++dz) {
    const int z = cz + dz;
    if (z < 0 || z >= nz) continue;
    for (int dy = -1; dy <= 1; ++dy) {
      const int y = cy + dy;
      if (y < 0 || y >= ny) continue;
      const int q = (dz + 1) * 3 + (dy + 1);
      const uint32_t row = s.cell_base + (uint32_t)nx * ((uint32_t)y + (uint32_t)ny * (uint32_t)z);
      const uint32_t a = Mem::ld(&off[row + x0]);
      const uint32_t b = Mem::ld(&off[row + x1 + 1]);
      for (uint32_t j = a; j < b; ++j)
        if (j != k) f(q, j);
    }
  }
}

// Re-derives N_k from the cells and the step-start positions (global loads).
template <typename Mem = EarlierKernel, typename F>
__device__ __forceinline__ void visit_fallback(const NbrCtx &c, uint32_t k, F &&f) {
  const SceneDesc &sc = scene_of(c.scenes, c.sid, k);
  const float3 pk = start_position<Mem>(c, k);
  scan_rows<Mem>(k, Mem::ld(&c.skeys[k]), sc, c.off, [&](int, uint32_t j) {
    if (is_pair(separation(pk, start_position<Mem>(c, j)).r2, c.h2)) f(j);
  });
}

// Calls f(load(slot)) for every neighbour of particle k (and, in the listed
// path, for k itself as the padding of the last group): from the list when
// k's set fits, otherwise re-derived.
template <int kBatch, typename Load, typename F>
__device__ __forceinline__ void visit_neighbours(const NbrCtx &c, uint32_t k, Load &&load,
                                                 F &&f) {
  const uint32_t cnt = load_own(&c.cnt[k]);
  if (cnt <= c.maxn) {
    for_each_listed<kBatch>(c.nbr4, c.n, k, cnt, load, f);
  } else {
    visit_fallback(c, k, [&](uint32_t j) { f(load(j)); });
  }
}

__device__ __forceinline__ float ipow(float b, int e) {
  float r = 1.0f;
  while (e > 0) {
    if (e & 1) r = __fmul_rn(r, b);
    b = __fmul_rn(b, b);
    e >>= 1;
  }
  return r;
}

// -k h^2 (W(r)/W(dq h))^n with W(r)/W(dq h) = ((h^2-r^2)/(h^2-dq^2 h^2))^3;
// kTwelve: the exponent 3n is 12 (n = 4, the paper's choice).
template <bool kTwelve>
__device__ __forceinline__ float scorr_term(float r2, const PaperConsts &c) {
  const float ratio = __fmul_rn(__fsub_rn(c.h2, r2), c.inv_scorr_den);
  if constexpr (kTwelve) {
    const float r3 = __fmul_rn(__fmul_rn(ratio, ratio), ratio);
    const float r6 = __fmul_rn(r3, r3);
    return __fmul_rn(-c.scorr_k, __fmul_rn(r6, r6));
  } else {
    return __fmul_rn(-c.scorr_k, ipow(ratio, c.scorr_n3));
  }
}

// Spiky gradient factor: grad_i W(r_vec) = f * r_vec, f = -S (h-r)^2 / r,
// for a pair (r^2 normal, so the MUFU reciprocal square root without the
// subnormal-input path equals rsqrtf).
__device__ __forceinline__ float spiky_factor(float r2, const PaperConsts &c) {
  float rinv;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(rinv) : "f"(r2));
  const float hr = __fmaf_rn(-r2, rinv, c.h);  // h - r, one rounding (r close to h cancels)
  return __fmul_rn(__fmul_rn(__fmul_rn(-c.spiky, hr), hr), rinv);
}

// Poly6 kernel value W(r) = poly6 (h^2 - r^2)^3.
__device__ __forceinline__ float poly6_value(float r2, const PaperConsts &c) {
  const float t = __fsub_rn(c.h2, r2);
  return __fmul_rn(__fmul_rn(__fmul_rn(c.poly6, t), t), t);
}

struct LambdaAcc {
  float rho, gx, gy, gz, s;
  __device__ __forceinline__ void add(const Sep &r, const PaperConsts &c) {
    const float t = __fsub_rn(c.h2, r.r2);
    rho = __fmaf_rn(__fmul_rn(__fmul_rn(c.poly6, t), t), t, rho);
    const float f = spiky_factor(r.r2, c);
    gx = __fmaf_rn(f, r.x, gx);
    gy = __fmaf_rn(f, r.y, gy);
    gz = __fmaf_rn(f, r.z, gz);
    s = __fmaf_rn(__fmul_rn(f, f), r.r2, s);
  }
  __device__ __forceinline__ float lambda(const PaperConsts &c) const {
    const float C = __fmaf_rn(rho, c.inv_rho0, -1.0f);
    const float g2 = __fmaf_rn(gz, gz, __fmaf_rn(gy, gy, __fmaf_rn(gx, gx, s)));
    const float den = __fmul_rn(g2, __fmul_rn(c.inv_rho0, c.inv_rho0));
    return __fdiv_rn(-C, __fadd_rn(den, c.relax_eps));
  }
};

// Calls member(j, sep) for every slot j that forms a pair with k
// (is_pair(r2 = |p_k - p_j|^2)) in the 27 cells around k's cell (key `key`),
// in the order the lists store and the re-derived path visits: rows by
// (dz, dy), each row's slots ascending.  The self pair and coincident
// particles drop out.
template <typename F>
__device__ __forceinline__ void scan_members(const float4 &pk, uint32_t key, const SceneDesc &s,
                                             const uint32_t *__restrict__ off,
                                             const float4 *__restrict__ P, const PaperConsts &c,
                                             F &&member) {
  const int nx = s.ncell[0], ny = s.ncell[1], nz = s.ncell[2];
  const uint32_t local = key - s.cell_base;
  const int cx = (int)(local % (uint32_t)nx);
  const uint32_t t = local / (uint32_t)nx;
  const int cy = (int)(t % (uint32_t)ny);
  const int cz = (int)(t / (uint32_t)ny);
  const int x0 = cx > 0 ? cx - 1 : 0;
  const int x1 = cx + 1 < nx ? cx + 1 : nx - 1;
  for (int dz = -1; dz <= 1; ++dz) {
    const int z = cz + dz;
    if (z < 0 || z >= nz) continue;
    for (int dy = -1; dy <= 1; ++dy) {
      const int y = cy + dy;
      if (y < 0 || y >= ny) continue;
      const uint32_t row = s.cell_base + (uint32_t)nx * ((uint32_t)y + (uint32_t)ny * (uint32_t)z);
      const uint32_t a = __ldg(&off[row + x0]);
      const uint32_t b = __ldg(&off[row + x1 + 1]);
      // whole groups of four candidates (loads at fixed offsets from one
      // pointer, no per-load bound), then the last one to three
      uint32_t j = a;
      for (; j + 4u <= b; j += 4) {
        const float4 *__restrict__ q = P + j;
        float4 d[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) d[e] = __ldg(q + e);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const Sep r = separation(pk, d[e]);
          if (is_pair(r.r2, c.h2)) member(j + e, r);
        }
      }
      if (j < b) {
        float4 d[3];
#pragma unroll
        for (int e = 0; e < 3; ++e) d[e] = __ldg(&P[min(j + e, b - 1u)]);
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          const Sep r = separation(pk, d[e]);
          if (j + e < b && is_pair(r.r2, c.h2)) member(j + e, r);
        }
      }
    }
  }
}

// The same members in the same order, found as masks: each row is tested up
// to 32 candidates at a time from the position planes, and the masks' members
// reach word(w, slots) in whole list words.  Returns the number of members.  Only
// the row of k's own cell can hold k itself or a coincident particle, so only there
// r^2 is tested against zero as well.  The candidate loop is 23 instructions per
// four candidates (12 of them packed), where one candidate at a time with its member
// work inside took about 18 each.  kWarp: all 32 lanes call it (MaskQueue).
template <typename Mem, bool kWarp, typename Word>
__device__ __forceinline__ uint32_t scan_members_planes(const float4 &pk, uint32_t k, uint32_t key,
                                                        const SceneDesc &s,
                                                        const uint32_t *__restrict__ off,
                                                        const Planes &planes,
                                                        const PaperConsts &c, Word &&word) {
  const int nx = s.ncell[0], ny = s.ncell[1], nz = s.ncell[2];
  const uint32_t local = key - s.cell_base;
  const int cx = (int)(local % (uint32_t)nx);
  const uint32_t t = local / (uint32_t)nx;
  const int cy = (int)(t % (uint32_t)ny);
  const int cz = (int)(t / (uint32_t)ny);
  const int x0 = cx > 0 ? cx - 1 : 0;
  const int x1 = cx + 1 < nx ? cx + 1 : nx - 1;
  const float2 px = make_float2(-pk.x, -pk.x), py = make_float2(-pk.y, -pk.y),
               pz = make_float2(-pk.z, -pk.z);
  MaskQueue<kMaskQueue> list;
  for (int dz = -1; dz <= 1; ++dz) {
    const int z = cz + dz;
    for (int dy = -1; dy <= 1; ++dy) {
      const int y = cy + dy;
      uint32_t a = 0, b = 0;  // a row outside the grid holds nothing
      if (z >= 0 && z < nz && y >= 0 && y < ny) {
        const uint32_t row =
            s.cell_base + (uint32_t)nx * ((uint32_t)y + (uint32_t)ny * (uint32_t)z);
        a = Mem::ld(&off[row + x0]);
        b = Mem::ld(&off[row + x1 + 1]);
      }
      const bool own = (dz | dy) == 0;
      list.template add_row<kWarp>(
          a, b,
          [&](uint32_t c0) {
            return own ? row_mask<true, Mem>(planes, c0, a, b, px, py, pz, kMinPair2, c.h2)
                       : row_mask<false, Mem>(planes, c0, a, b, px, py, pz, 0.f, c.h2);
          },
          word);
    }
  }
  const uint32_t cnt = list.count();
  list.finish(k, word);
  return cnt;
}

// ------------------------------------------------------------ pair terms --
// Lambda pass: density, constraint gradient sums over the pairs of k.
__device__ __forceinline__ void lambda_pair(LambdaAcc &acc, const float4 &pk, const float4 &pj,
                                            const PaperConsts &c) {
  const Sep r = separation(pk, pj);
  if (is_pair(r.r2, c.h2)) acc.add(r, c);
}
__device__ __forceinline__ void lambda_commit(uint32_t k, const float4 &pk, const LambdaAcc &acc,
                                              const PaperConsts &c, float4 *__restrict__ Q,
                                              float *__restrict__ R) {
  Q[k] = make_float4(pk.x, pk.y, pk.z, acc.lambda(c));
  R[k] = acc.rho;
}

// Delta-p pass: sum of (lambda_k + lambda_j + s_corr) grad W over the pairs.
template <bool kTwelve>
__device__ __forceinline__ float delta_weight(float lk, float lj, float r2, const PaperConsts &c) {
  return __fmul_rn(__fadd_rn(__fadd_rn(lk, lj), scorr_term<kTwelve>(r2, c)), spiky_factor(r2, c));
}
struct DeltaAcc {
  float sx, sy, sz;
  template <bool kTwelve>
  __device__ __forceinline__ void pair(const float4 &qk, const float4 &qj, const PaperConsts &c) {
    const Sep r = separation(qk, qj);
    if (is_pair(r.r2, c.h2)) {
      const float wgt = delta_weight<kTwelve>(qk.w, qj.w, r.r2, c);
      sx = __fmaf_rn(wgt, r.x, sx);
      sy = __fmaf_rn(wgt, r.y, sy);
      sz = __fmaf_rn(wgt, r.z, sz);
    }
  }
};
// delta-p, collision response (clamp to the admissible box with the moving
// x-min wall), Jacobi update of d and p; the last iteration also writes the
// velocity d/dt and 1/rho for the velocity passes.
struct Moved {
  float3 d, p;
};
// (x, d0: the particle's step-start position and displacement.)
__device__ __forceinline__ Moved delta_moved(const DeltaAcc &a, const float4 &x, const float4 &d0,
                                             const SceneDesc &sc, const PaperConsts &c) {
  float3 d = make_float3(__fmaf_rn(a.sx, c.inv_rho0, d0.x), __fmaf_rn(a.sy, c.inv_rho0, d0.y),
                         __fmaf_rn(a.sz, c.inv_rho0, d0.z));
  float3 p = add3(x, d);
  const float lo_x = __fadd_rn(sc.lo[0], sc.wave);
  if (p.x < lo_x) { d.x = __fsub_rn(lo_x, x.x); p.x = __fadd_rn(x.x, d.x); }
  else if (p.x > sc.hi[0]) { d.x = __fsub_rn(sc.hi[0], x.x); p.x = __fadd_rn(x.x, d.x); }
  if (p.y < sc.lo[1]) { d.y = __fsub_rn(sc.lo[1], x.y); p.y = __fadd_rn(x.y, d.y); }
  else if (p.y > sc.hi[1]) { d.y = __fsub_rn(sc.hi[1], x.y); p.y = __fadd_rn(x.y, d.y); }
  if (p.z < sc.lo[2]) { d.z = __fsub_rn(sc.lo[2], x.z); p.z = __fadd_rn(x.z, d.z); }
  else if (p.z > sc.hi[2]) { d.z = __fsub_rn(sc.hi[2], x.z); p.z = __fadd_rn(x.z, d.z); }
  return Moved{d, p};
}
// Velocity d/dt and 1/rho.
__device__ __forceinline__ float4 delta_velocity(const float3 &d, float rho, const PaperConsts &c) {
  return make_float4(__fdiv_rn(d.x, c.dt), __fdiv_rn(d.y, c.dt), __fdiv_rn(d.z, c.dt),
                     __fdiv_rn(1.0f, rho));
}
template <typename Rho>
__device__ __forceinline__ void delta_store(uint32_t k, const DeltaAcc &a, const float4 &x,
                                            const float4 &d0, Rho &&rho, const NbrCtx &nc,
                                            const PaperConsts &c, float4 *__restrict__ D,
                                            float4 *__restrict__ P, float4 *__restrict__ U,
                                            int last) {
  const Moved m = delta_moved(a, x, d0, scene_of(nc.scenes, nc.sid, k), c);
  D[k] = make_float4(m.d.x, m.d.y, m.d.z, 0.0f);
  P[k] = make_float4(m.p.x, m.p.y, m.p.z, 0.0f);
  if (last) U[k] = delta_velocity(m.d, rho(), c);
}
__device__ __forceinline__ void delta_commit(uint32_t k, const DeltaAcc &a, const NbrCtx &nc,
                                             const PaperConsts &c, float4 *__restrict__ D,
                                             float4 *__restrict__ P, const float *__restrict__ R,
                                             float4 *__restrict__ U, int last) {
  const float4 x = load_own(&nc.X2[k]);
  const float4 d0 = load_own(&D[k]);
  delta_store(k, a, x, d0, [&] { return load_own(&R[k]); }, nc, c, D, P, U, last);
}

// A neighbour's (position, velocity) as the velocity passes read it.
struct PU {
  float4 p, u;
};

// a x b, component by component with one rounding per product and sum.
__device__ __forceinline__ float cross_component(float a1, float b2, float a2, float b1) {
  return __fmaf_rn(a1, b2, __fmul_rn(-a2, b1));  // a1 b2 - a2 b1
}

// Vorticity pass, which also carries the neighbour sums the XSPH pass would
// otherwise gather velocities for:
//   omega_k = sum (1/rho_j) grad W x (v_j - v_k),
//   S_k     = sum (1/rho_j) grad W,
//   X_k     = sum (1/rho_j) W (v_j - v_k)   (XSPH viscosity).
// With |omega_j| / rho_j gathered in the next pass, the vorticity location
// vector eta_k = sum (1/rho_j)(|omega_j| - |omega_k|) grad W is
// sum (|omega_j|/rho_j) grad W - |omega_k| S_k, so that pass gathers one
// float4 per neighbour instead of two.
struct VortTerms {  // one pair's terms: w and s add theirs, X adds wp * u
  float wx, wy, wz, gx, gy, gz, wp, ux, uy, uz;
};
__device__ __forceinline__ VortTerms vort_terms(const Sep &r, const float4 &uk, const float4 &uj,
                                                const PaperConsts &c) {
  VortTerms t;
  const float f = __fmul_rn(spiky_factor(r.r2, c), uj.w);
  t.gx = __fmul_rn(f, r.x);
  t.gy = __fmul_rn(f, r.y);
  t.gz = __fmul_rn(f, r.z);
  t.ux = __fsub_rn(uj.x, uk.x);
  t.uy = __fsub_rn(uj.y, uk.y);
  t.uz = __fsub_rn(uj.z, uk.z);
  t.wx = cross_component(t.gy, t.uz, t.gz, t.uy);
  t.wy = cross_component(t.gz, t.ux, t.gx, t.uz);
  t.wz = cross_component(t.gx, t.uy, t.gy, t.ux);
  t.wp = __fmul_rn(poly6_value(r.r2, c), uj.w);
  return t;
}
struct VortAcc {
  float wx, wy, wz, sx, sy, sz, xx, xy, xz;
  __device__ __forceinline__ void pair(const float4 &pk, const float4 &uk, const PU &d,
                                       const PaperConsts &c) {
    const Sep r = separation(pk, d.p);
    if (is_pair(r.r2, c.h2)) {
      const VortTerms t = vort_terms(r, uk, d.u, c);
      wx = __fadd_rn(wx, t.wx);
      wy = __fadd_rn(wy, t.wy);
      wz = __fadd_rn(wz, t.wz);
      sx = __fadd_rn(sx, t.gx);
      sy = __fadd_rn(sy, t.gy);
      sz = __fadd_rn(sz, t.gz);
      xx = __fmaf_rn(t.wp, t.ux, xx);
      xy = __fmaf_rn(t.wp, t.uy, xy);
      xz = __fmaf_rn(t.wp, t.uz, xz);
    }
  }
};
__device__ __forceinline__ float norm3(float x, float y, float z) {
  return __fsqrt_rn(__fmaf_rn(z, z, __fmaf_rn(y, y, __fmul_rn(x, x))));
}
// Writes (omega_k, |omega_k|), (p_k, |omega_k| / rho_k) for the XSPH pass to
// gather, and k's own sums X_k and S_k.
__device__ __forceinline__ void vort_commit(uint32_t k, const float4 &pk, const float4 &uk,
                                            const VortAcc &a, float4 *__restrict__ Wo,
                                            float4 *__restrict__ PW, float4 *__restrict__ XS,
                                            float4 *__restrict__ SS) {
  const float wn = norm3(a.wx, a.wy, a.wz);
  Wo[k] = make_float4(a.wx, a.wy, a.wz, wn);
  PW[k] = make_float4(pk.x, pk.y, pk.z, __fmul_rn(wn, uk.w));
  XS[k] = make_float4(a.xx, a.xy, a.xz, 0.0f);
  SS[k] = make_float4(a.sx, a.sy, a.sz, 0.0f);
}

// XSPH + vorticity-confinement pass: E_k = sum (|omega_j|/rho_j) grad W over
// the pairs (pj.w = |omega_j|/rho_j).
struct XsphAcc {
  float ex, ey, ez;
  __device__ __forceinline__ void pair(const float4 &pk, const float4 &pj, const PaperConsts &c) {
    const Sep r = separation(pk, pj);
    if (is_pair(r.r2, c.h2)) {
      const float e = __fmul_rn(spiky_factor(r.r2, c), pj.w);
      ex = __fmaf_rn(e, r.x, ex);
      ey = __fmaf_rn(e, r.y, ey);
      ez = __fmaf_rn(e, r.z, ez);
    }
  }
};
// eta = E - |omega_k| S_k; v = v + dt f_vorticity + c_xsph X_k with
// f_vorticity = eps (eta/|eta|) x omega; commits x (.w = |v|), v (.w = mass)
// and the input index of slot k.
__device__ __forceinline__ void xsph_store(uint32_t k, const float4 &pk, const float4 &uk,
                                           const float4 &wk, const float4 &xs, const float4 &ss,
                                           const XsphAcc &a, const PaperConsts &c, float mass,
                                           uint32_t id, float4 *__restrict__ X,
                                           float4 *__restrict__ V, uint32_t *__restrict__ ID) {
  const float ex = __fmaf_rn(-wk.w, ss.x, a.ex), ey = __fmaf_rn(-wk.w, ss.y, a.ey),
              ez = __fmaf_rn(-wk.w, ss.z, a.ez);
  const float el2 = __fmaf_rn(ez, ez, __fmaf_rn(ey, ey, __fmul_rn(ex, ex)));
  float nx = 0.f, ny = 0.f, nz = 0.f;
  if (el2 > 0.0f) {
    const float inv = rsqrtf(el2);
    nx = __fmul_rn(ex, inv);
    ny = __fmul_rn(ey, inv);
    nz = __fmul_rn(ez, inv);
  }
  const float fx = __fmul_rn(c.vort_eps, cross_component(ny, wk.z, nz, wk.y));
  const float fy = __fmul_rn(c.vort_eps, cross_component(nz, wk.x, nx, wk.z));
  const float fz = __fmul_rn(c.vort_eps, cross_component(nx, wk.y, ny, wk.x));
  const float vx = __fmaf_rn(c.xsph_c, xs.x, __fmaf_rn(c.dt, fx, uk.x));
  const float vy = __fmaf_rn(c.xsph_c, xs.y, __fmaf_rn(c.dt, fy, uk.y));
  const float vz = __fmaf_rn(c.xsph_c, xs.z, __fmaf_rn(c.dt, fz, uk.z));
  X[k] = make_float4(pk.x, pk.y, pk.z, norm3(vx, vy, vz));
  V[k] = make_float4(vx, vy, vz, mass);
  ID[k] = id;
}

// The launch arguments shared by the passes over the L1 lists.
inline NbrCtx make_ctx(const DeviceState &d, const PaperConsts &c, const uint16_t *sid) {
  NbrCtx nc;
  nc.nbr4 = d.nbr;
  nc.cnt = d.nbr_cnt;
  nc.skeys = d.skeys;
  nc.off = d.offsets;
  nc.X2 = d.X2;
  nc.V2 = d.V2;
  nc.scenes = d.scenes;
  nc.sid = sid;
  nc.err = d.err;
  nc.cnt_max = d.nbr_max;
  nc.host_max = d.nbr_max_host;
  nc.n = c.n;
  nc.maxn = c.maxn;
  nc.dt = c.dt;
  nc.h2 = c.h2;
  return nc;
}

}  // namespace
}  // namespace pbf
