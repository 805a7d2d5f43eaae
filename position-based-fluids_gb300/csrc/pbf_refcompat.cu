// Solver kernels of the GB300 position-based-fluids step, reference
// equations (PBF_MODE_REF_COMPAT).  This translation unit is compiled with
// -fmad=false: every expression is evaluated operator by operator in IEEE
// binary32 with correctly rounded division and square root, in the operator
// order of the reference's kernels (MrMagne/position-based-fluids):
//   predict_positions.cl:8-9, update_cells.cl:10-15, compute_scaling.cl:11-140,
//   compute_delta.cl:13-152 + update_predicted.cl:7, update_velocities.cl:8,
//   apply_vorticity_and_viscosity.cl:12-104, update_positions.cl:9-12.
//
// State stays in input order (X, V, P = predicted with .w = density).  The
// reference visits the 27 cells around the particle's *current* cell with x
// outermost and z innermost, and each cell's particles in descending index --
// the order a sequential launch of update_cells.cl leaves in its linked
// lists.  The neighbour structure is laid out in exactly that order: cells
// are numbered with z fastest (rc_cell) and the particles are sorted in
// descending input index (sort element t is particle n - 1 - t), so the three
// cells of one (x, y) row are one contiguous run of sorted slots that is
// visited front to back.  Results then equal the reference's kernels bit for
// bit.  During the step the passes keep P, V and lambda by sorted slot as
// well (PS, VS, SS).
//
// The lambda and delta-p passes of one solver iteration evaluate the same
// pairs: lambda moves nothing.  So the lambda pass finds its members (the
// candidates of the nine rows tested into masks), sums their terms and leaves
// them in visiting order as neighbour lists, and the delta-p pass walks the
// list; the XSPH pass finds its own at the final positions.  With every pass
// testing and evaluating candidate by candidate, a warp ran the pair arithmetic
// (square roots and divisions) for nearly every one of ~216 candidates with
// 15 of 32 lanes active: 572, 537 and 443 us per lambda, delta-p and XSPH
// pass at 1,048,576 particles, against 257, 110 and 241 us now (lambda and
// delta-p issue instructions 73-79% of the time, over 90 per pair; XSPH's
// gathers keep L1's data path 90% busy).  A particle with more members than
// the list holds walks the cells in the delta-p pass instead.  (In a block at 4.6
// times the rest density, some 150 members each, 64,000 particles take 148, 234 and
// 108 us per pass; candidate by candidate they took 241, 219 and 199.)
#include "pbf_group.cuh"
#include "pbf_lists.cuh"

namespace pbf {

namespace {

constexpr int kThreads = 128;

// Calls row(a, b) for the slot range [a, b) of each of the nine rows of up to three
// cells around the current cell of position p, in visiting order.  Cells outside
// the grid hold nothing (the current cell itself may be outside).
template <typename Row>
__device__ __forceinline__ void ref_rows(float4 p, const RefConsts &k,
                                         const uint32_t *__restrict__ off, Row &&row) {
  const int nx = (int)k.ncell[0], ny = (int)k.ncell[1], nz = (int)k.ncell[2];
  // two cells outside is as far as any: keeps the sums below in range
  const int c0 = min(max((int)((p.x - k.min[0]) / k.clen[0]), -2), nx + 1);
  const int c1 = min(max((int)((p.y - k.min[1]) / k.clen[1]), -2), ny + 1);
  const int c2 = min(max((int)((p.z - k.min[2]) / k.clen[2]), -2), nz + 1);
  const int z0 = max(c2 - 1, 0), z1 = min(c2 + 1, nz - 1);
  for (int q = 0; q < 9; ++q) {
    const int x = c0 + q / 3 - 1, y = c1 + q % 3 - 1;
    uint32_t a = 0, b = 0;
    if (z0 <= z1 && x >= 0 && x < nx && y >= 0 && y < ny) {
      const uint32_t first = (uint32_t)nz * ((uint32_t)y + (uint32_t)ny * (uint32_t)x);
      a = __ldg(&off[first + z0]);
      b = __ldg(&off[first + z1 + 1]);
    }
    row(a, b);
  }
}

__device__ __forceinline__ float wider_h2(const RefConsts &k) {
  return k.h2 * 1.000001f + 1e-44f;
}

// The members of slot q (position p) in visiting order, from masks over the
// position planes, handed on four at a time as word(w, slots); the last word
// is filled up with q itself.  Returns their number.  The masks only have to
// hold every member: whoever takes the words applies the reference's own pair
// test, so r^2 is evaluated with FMAs here (12 packed instructions per four
// candidates instead of 16, and no lower bound) against an h^2 widened by more
// than both evaluations can differ, 6 * 2^-24 relative; q itself, which every
// scan meets, is taken out by its slot.
template <bool kWarp, typename Word>
__device__ __forceinline__ uint32_t scan_ref_members(uint32_t q, const float4 &p,
                                                     const RefConsts &k,
                                                     const uint32_t *__restrict__ off,
                                                     const Planes &planes, Word &&word) {
  const float2 px = make_float2(-p.x, -p.x), py = make_float2(-p.y, -p.y),
               pz = make_float2(-p.z, -p.z);
  const float h2 = wider_h2(k);
  MaskQueue<kMaskQueue> list;
  ref_rows(p, k, off, [&](uint32_t a, uint32_t b) {
    list.template add_row<kWarp>(
        a, b,
        [&](uint32_t c0) {
          uint32_t m = row_mask<false>(planes, c0, a, b, px, py, pz, 0.0f, h2);
          if (q - c0 < 32u) m &= ~(0x80000000u >> (q - c0));
          return m;
        },
        word);
  });
  const uint32_t cnt = list.count();
  list.finish(q, word);
  return cnt;
}

// Calls f(load(m)) for every candidate of the cells in visiting order, four loads in
// flight together.  (8,000 particles of some 150 members each: delta-p 158 -> 141 us.)
template <typename Load, typename F>
__device__ __forceinline__ void ref_candidates(float4 p, const RefConsts &k,
                                               const uint32_t *__restrict__ off, Load &&load,
                                               F &&f) {
  ref_rows(p, k, off, [&](uint32_t a, uint32_t b) {
    for (uint32_t m = a; m < b; m += 4) {
      decltype(load(0u)) d[4];
#pragma unroll
      for (uint32_t e = 0; e < 4; ++e) d[e] = load(min(m + e, b - 1u));
#pragma unroll
      for (uint32_t e = 0; e < 4; ++e)
        if (m + e < b) f(d[e]);
    }
  });
}

// Calls f(load(m)) for the members of slot q in visiting order (and for q
// itself as padding, which the pair test drops): from the list, or over all
// candidates of the cells when the list does not hold the set.
template <typename Load, typename F>
__device__ __forceinline__ void ref_members(uint32_t q, float4 p, const RefConsts &k,
                                            const RefLists &l, const uint32_t *__restrict__ off,
                                            Load &&load, F &&f) {
  const uint32_t cnt = l.maxn ? load_own(&l.cnt[q]) : 0u;
  if (l.maxn && cnt <= l.maxn)
    for_each_listed<4>(l.nbr4, l.n, q, cnt, load, f);
  else
    ref_candidates(p, k, off, load, f);
}

// Cell of a position with z fastest, as the passes' neighbour structure
// numbers the cells (scene_cell is the reference's numbering, x fastest).
__device__ __forceinline__ uint32_t rc_cell(float x, float y, float z, const SceneDesc &s) {
  const int cx = axis_cell(x, s.gmin[0], s.clen[0], s.ncell[0]);
  const int cy = axis_cell(y, s.gmin[1], s.clen[1], s.ncell[1]);
  const int cz = axis_cell(z, s.gmin[2], s.clen[2], s.ncell[2]);
  return (uint32_t)cz +
         (uint32_t)s.ncell[2] * ((uint32_t)cy + (uint32_t)s.ncell[1] * (uint32_t)cx);
}

__device__ __forceinline__ void store_planes(float *__restrict__ planes, uint32_t plane,
                                             uint32_t q, const float4 &p) {
  planes[q] = p.x;
  planes[plane + q] = p.y;
  planes[2 * (size_t)plane + q] = p.z;
}

// Prediction of sort element t (particle n - 1 - t) and its cell.
__device__ __forceinline__ uint32_t rc_predict(uint32_t t, uint32_t n, const float4 *X, float4 *V,
                                               float4 *P, const RefConsts &k,
                                               const SceneDesc &scene) {
  const uint32_t i = n - 1u - t;
  const float4 x = X[i];
  float4 v = V[i];
  v.x = v.x + k.dt * 0.0f;
  v.y = v.y + k.dt * -9.81f;
  v.z = v.z + k.dt * 0.0f;
  V[i] = v;
  float4 p = P[i];
  p.x = x.x + k.dt * v.x;
  p.y = x.y + k.dt * v.y;
  p.z = x.z + k.dt * v.z;
  P[i] = p;
  return rc_cell(p.x, p.y, p.z, scene);
}

// Prediction and cell of every particle, counted for the counting sort
// (grid-stride, whole warps iterate together).
__global__ void __launch_bounds__(256)
    k_rc_predict_count(const float4 *__restrict__ X, float4 *__restrict__ V,
                       float4 *__restrict__ P, uint32_t n, RefConsts k,
                       const SceneDesc *__restrict__ scenes, uint32_t *__restrict__ keys,
                       uint32_t *__restrict__ counts, uint32_t *__restrict__ pos) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride) {
    const uint32_t t[1] = {base + threadIdx.x};
    const bool valid[1] = {t[0] < n};
    uint32_t key[1] = {0};
    if (valid[0]) keys[t[0]] = key[0] = rc_predict(t[0], n, X, V, P, k, scenes[0]);
    count_cell_keys<false>(key, valid, t, counts, pos);
  }
}

__global__ void __launch_bounds__(256)
    k_rc_predict_hash(const float4 *__restrict__ X, float4 *__restrict__ V,
                      float4 *__restrict__ P, uint32_t n, RefConsts k,
                      const SceneDesc *__restrict__ scenes,
                      uint32_t *__restrict__ keys, uint32_t passes,
                      uint32_t digit_bits, uint32_t *__restrict__ hist) {
  __shared__ uint32_t s_hist[kMaxHistWords];
  const uint32_t hist_words = passes << digit_bits;
  for (uint32_t t = threadIdx.x; t < hist_words; t += blockDim.x) s_hist[t] = 0;
  __syncthreads();
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride) {
    const uint32_t t = base + threadIdx.x;
    const bool valid = t < n;
    uint32_t key = 0;
    if (valid) keys[t] = key = rc_predict(t, n, X, V, P, k, scenes[0]);
    warp_digit_histogram(key, valid, passes, digit_bits, s_hist);
  }
  __syncthreads();
  for (uint32_t t = threadIdx.x; t < hist_words; t += blockDim.x)
    if (s_hist[t]) atomicAdd(&hist[t], s_hist[t]);
}

// Predicted positions by slot (PS, planes) and each slot's input index.
// kRanked: as k_reorder (pbf_paper.cu), the cells of up to clear.rank_cell
// particles are put in order here, and the sort's control words left zero.
template <bool kRanked>
__global__ void __launch_bounds__(256)
    k_rc_gather(const float4 *__restrict__ P, const uint32_t *__restrict__ perm,
                const uint32_t *__restrict__ skeys, const uint32_t *__restrict__ off,
                StepClear clear, uint32_t n, float4 *__restrict__ PS, uint32_t *__restrict__ input,
                float *__restrict__ planes, uint32_t plane) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (kRanked)
    for (uint32_t i = t; i < clear.words; i += gridDim.x * blockDim.x) clear.ctl[i] = 0u;
  if (t >= n) return;
  // perm is a permutation of [0, n) unless the sort reported an error.
  const uint32_t element = min(perm[t], n - 1u);
  const uint32_t q = kRanked ? ordered_slot(perm, off, skeys[t], t, element, n, clear.rank_cell) : t;
  const uint32_t i = n - 1u - element;
  const float4 p = P[i];
  PS[q] = p;
  input[q] = i;
  store_planes(planes, plane, q, p);
}

// The terms of one pair in each pass; false: not a pair.
struct RefLambdaTerms {
  float poly, len, gx, gy, gz;
};
__device__ __forceinline__ bool ref_lambda_terms(const float4 &pi, const float4 &pj,
                                                 const RefConsts &k, RefLambdaTerms &t) {
  const float rx = pi.x - pj.x, ry = pi.y - pj.y, rz = pi.z - pj.z;
  const float r2 = rx * rx + ry * ry + rz * rz;
  if (!(r2 > 0.0f && r2 < k.h2)) return false;
  const float rl = sqrtf(r2);
  t.gx = rx / rl * k.spiky * (k.h - rl) * (k.h - rl);
  t.gy = ry / rl * k.spiky * (k.h - rl) * (k.h - rl);
  t.gz = rz / rl * k.spiky * (k.h - rl) * (k.h - rl);
  t.poly = k.poly6 * (k.h2 - r2) * (k.h2 - r2) * (k.h2 - r2);
  t.len = sqrtf(t.gx * t.gx + t.gy * t.gy + t.gz * t.gz);
  return true;
}
struct RefTerms {
  float x, y, z;
};
__device__ __forceinline__ bool ref_delta_terms(const float4 &pi, float si, const float4 &pj,
                                                float sj, const RefConsts &k, RefTerms &t) {
  const float rx = pi.x - pj.x, ry = pi.y - pj.y, rz = pi.z - pj.z;
  const float r2 = rx * rx + ry * ry + rz * rz;
  if (!(r2 > 0.0f && r2 < k.h2)) return false;
  const float rl = sqrtf(r2);
  const float gx = -1.0f * rx / rl * k.spiky * (k.h - rl) * (k.h - rl);
  const float gy = -1.0f * ry / rl * k.spiky * (k.h - rl) * (k.h - rl);
  const float gz = -1.0f * rz / rl * k.spiky * (k.h - rl) * (k.h - rl);
  const float sc = si + sj;
  t.x = sc * gx;
  t.y = sc * gy;
  t.z = sc * gz;
  return true;
}
// (vj.w is 1 / density)
__device__ __forceinline__ bool ref_xsph_terms(const float4 &pi, const float4 &vi,
                                               const float4 &pj, const float4 &vj,
                                               const RefConsts &k, RefTerms &t) {
  const float rx = pi.x - pj.x, ry = pi.y - pj.y, rz = pi.z - pj.z;
  const float r2 = rx * rx + ry * ry + rz * rz;
  if (!(r2 > 0.0f && r2 < k.h2)) return false;
  const float vx = vj.x - vi.x, vy = vj.y - vi.y, vz = vj.z - vi.z;
  const float poly = k.poly6 * (k.h2 - r2) * (k.h2 - r2) * (k.h2 - r2);
  const float inv = vj.w;
  t.x = inv * vx * poly;
  t.y = inv * vy * poly;
  t.z = inv * vz * poly;
  return true;
}

struct RefLambdaSums {
  float dens = 0.0f, gsum = 0.0f, gvx = 0.0f, gvy = 0.0f, gvz = 0.0f;
  __device__ __forceinline__ void add(const float4 &pi, const float4 &pj, const RefConsts &k) {
    RefLambdaTerms t;
    if (ref_lambda_terms(pi, pj, k, t)) {
      dens += t.poly;
      gsum += t.len;
      gvx += t.gx;
      gvy += t.gy;
      gvz += t.gz;
    }
  }
};
__device__ __forceinline__ void ref_lambda_commit(uint32_t q, RefLambdaSums s, const RefConsts &k,
                                                  float4 *__restrict__ PS,
                                                  float *__restrict__ SS) {
  s.gsum += sqrtf(s.gvx * s.gvx + s.gvy * s.gvy + s.gvz * s.gvz);
  // Only .w changes; concurrent readers use .xyz.
  reinterpret_cast<float *>(&PS[q])[3] = s.dens;
  const float c = s.dens / k.rest_density - 1.0f;
  SS[q] = -1.0f * c / (s.gsum * s.gsum / (k.rest_density * k.rest_density) + 10000.0f);
}

// Lambda of every particle, and the neighbour lists for the delta-p pass of the
// iteration: the members of slot q in visiting order, found by row masks,
// their terms summed as each list word of four is handed on.  (48 registers:
// 3% faster than the 56 it takes unbounded, which leave 9 CTAs an SM.)
__global__ void __launch_bounds__(kThreads, 10)
    k_rc_lambda(float4 *__restrict__ PS, Planes planes, float *__restrict__ SS,
                const uint32_t *__restrict__ off, uint32_t n, RefConsts k, uint32_t maxn,
                uint4 *__restrict__ nbr4, uint32_t *__restrict__ nbr_cnt) {
  // past the end the last particle once more: the warp stays whole
  const uint32_t q = min(blockIdx.x * blockDim.x + threadIdx.x, n - 1u);
  const float4 pi = PS[q];
  RefLambdaSums s;
  const uint32_t cnt = scan_ref_members<true>(
      q, pi, k, off, planes, [&](uint32_t w, const uint4 &j) {
        if (4u * w < maxn) nbr4[(size_t)w * n + q] = j;
        const float4 d[4] = {PS[j.x], PS[j.y], PS[j.z], PS[j.w]};
#pragma unroll
        for (int e = 0; e < 4; ++e) s.add(pi, d[e], k);
      });
  if (maxn) nbr_cnt[q] = cnt;
  ref_lambda_commit(q, s, k, PS, SS);
}

// Future position, wall clamp, Jacobi update; the last iteration also writes
// the predicted position and the velocity by input index.
struct RcDeltaOut {
  float4 *PS2, *V, *P, *VS;
  const float4 *X;
  const uint32_t *input;
  float *planes;
  uint32_t plane;
  const SceneDesc *scenes;
  int last;
};
__device__ __forceinline__ void ref_delta_commit(uint32_t q, const float4 &pi, float sx, float sy,
                                                 float sz, const RefConsts &k,
                                                 const RcDeltaOut &o) {
  const float wave = o.scenes[0].wave;
  float fx = pi.x + sx / k.rest_density;
  float fy = pi.y + sy / k.rest_density;
  float fz = pi.z + sz / k.rest_density;
  if ((fx - k.h) < (k.min[0] + wave)) fx = k.min[0] + wave + k.h;
  else if ((fx + k.h) > k.max[0]) fx = k.max[0] - k.h;
  if ((fy - k.h) < k.min[1]) fy = k.min[1] + k.h;
  else if ((fy + k.h) > k.max[1]) fy = k.max[1] - k.h;
  if ((fz - k.h) < k.min[2]) fz = k.min[2] + k.h;
  else if ((fz + k.h) > k.max[2]) fz = k.max[2] - k.h;
  // computeDelta writes delta = future - predicted; updatePredicted adds it.
  const float dx = fx - pi.x, dy = fy - pi.y, dz = fz - pi.z;
  const float4 np = make_float4(pi.x + dx, pi.y + dy, pi.z + dz, pi.w);
  o.PS2[q] = np;
  store_planes(o.planes, o.plane, q, np);
  if (o.last) {
    const uint32_t i = o.input[q];
    o.P[i] = np;
    // updateVelocities
    const float4 x = o.X[i];
    float4 v = o.V[i];
    v.x = (np.x - x.x) / k.dt;
    v.y = (np.y - x.y) / k.dt;
    v.z = (np.z - x.z) / k.dt;
    o.V[i] = v;
    o.VS[q] = make_float4(v.x, v.y, v.z, 1.0f / np.w);
  }
}

struct PSl {
  float4 p;
  float s;
};

__global__ void __launch_bounds__(kThreads)
    k_rc_delta(const float4 *__restrict__ PS, const float *__restrict__ SS, RefLists lists,
               const uint32_t *__restrict__ off, uint32_t n, RefConsts k, RcDeltaOut out) {
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const float4 pi = PS[q];
  const float si = SS[q];
  float sx = 0.0f, sy = 0.0f, sz = 0.0f;
  ref_members(
      q, pi, k, lists, off, [&](uint32_t m) { return PSl{__ldg(&PS[m]), __ldg(&SS[m])}; },
      [&](const PSl &d) {
        RefTerms t;
        if (ref_delta_terms(pi, si, d.p, d.s, k, t)) {
          sx += t.x;
          sy += t.y;
          sz += t.z;
        }
      });
  ref_delta_commit(q, pi, sx, sy, sz, k, out);
}

struct PV {
  float4 p, v;
};

__global__ void __launch_bounds__(kThreads)
    k_rc_xsph(const float4 *__restrict__ PS, Planes planes, const float4 *__restrict__ VS,
              float4 *__restrict__ DV, const uint32_t *__restrict__ input,
              const uint32_t *__restrict__ off, uint32_t n, RefConsts k) {
  // past the end the last particle once more: the warp stays whole
  const uint32_t q = min(blockIdx.x * blockDim.x + threadIdx.x, n - 1u);
  const float4 pi = PS[q];
  const float4 vi = VS[q];
  float sx = 0.0f, sy = 0.0f, sz = 0.0f;
  const auto pair = [&](const float4 &pj, const float4 &vj) {
    RefTerms t;
    if (ref_xsph_terms(pi, vi, pj, vj, k, t)) {
      sx += t.x;
      sy += t.y;
      sz += t.z;
    }
  };
  scan_ref_members<true>(q, pi, k, off, planes, [&](uint32_t, const uint4 &j) {
    const float4 p[4] = {__ldg(&PS[j.x]), __ldg(&PS[j.y]), __ldg(&PS[j.z]), __ldg(&PS[j.w])};
    const float4 v[4] = {__ldg(&VS[j.x]), __ldg(&VS[j.y]), __ldg(&VS[j.z]), __ldg(&VS[j.w])};
#pragma unroll
    for (int e = 0; e < 4; ++e) pair(p[e], v[e]);
  });
  DV[input[q]] = make_float4(0.01f * sx, 0.01f * sy, 0.01f * sz, 0.0f);
}

// ------------------------------------------ eight threads per particle --
// The same passes for scenes that do not fill the GPU (pbf_group.cuh): the
// group's threads evaluate a pair each and sum each component in visiting
// order.  See kRefGroupParticles for the line.
constexpr int kRefStride = Terms<5>::kStride;

// Rows of the group's particle, as ref_rows visits them: thread q holds row q,
// all hold row 8.
__device__ __forceinline__ void group_ref_rows(const float4 &p, const RefConsts &k,
                                               const uint32_t *__restrict__ off, uint2 (&row)[2]) {
  const int nx = (int)k.ncell[0], ny = (int)k.ncell[1], nz = (int)k.ncell[2];
  const int c0 = min(max((int)((p.x - k.min[0]) / k.clen[0]), -2), nx + 1);
  const int c1 = min(max((int)((p.y - k.min[1]) / k.clen[1]), -2), ny + 1);
  const int c2 = min(max((int)((p.z - k.min[2]) / k.clen[2]), -2), nz + 1);
  const int z0 = max(c2 - 1, 0), z1 = min(c2 + 1, nz - 1);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int q = h == 0 ? (int)lane_of_group() : 8;
    const int x = c0 + q / 3 - 1, y = c1 + q % 3 - 1;
    row[h] = make_uint2(0u, 0u);
    if (z0 <= z1 && x >= 0 && x < nx && y >= 0 && y < ny) {
      const uint32_t first = (uint32_t)nz * ((uint32_t)y + (uint32_t)ny * (uint32_t)x);
      row[h] = make_uint2(__ldg(&off[first + z0]), __ldg(&off[first + z1 + 1]));
    }
  }
}
// The group's list of the particle's members (and what scan_ref_members adds).
__device__ __forceinline__ uint32_t group_ref_scan(uint32_t q, const float4 &p, const RefConsts &k,
                                                   const uint32_t *__restrict__ off,
                                                   const Planes &planes, uint32_t *list) {
  uint2 row[2];
  group_ref_rows(p, k, off, row);
  return group_scan_rows<EarlierKernel, true>(q, p, row, planes, -1.0f, wider_h2(k), list);
}

// Every component is a plain sum of the pairs' terms.
template <int kCount>
struct RefSums {
  static constexpr int kSums = kCount, kFloats = kCount;
  static constexpr bool kOnes = true;
  __device__ __forceinline__ static int factor_a(int) { return -1; }
  __device__ __forceinline__ static int factor_b(int c) { return c; }
  __device__ __forceinline__ float start(int) const { return 0.0f; }
};
struct RcLambdaPass : RefSums<5> {
  const float4 *PS;  // .w is written meanwhile
  const RefConsts &k;
  using Data = float4;
  __device__ __forceinline__ RcLambdaPass(const float4 *ps, const RefConsts &c) : PS(ps), k(c) {}
  __device__ __forceinline__ float4 load(uint32_t j) const { return PS[j]; }
  __device__ __forceinline__ void pair(const float4 &pi, const float4 &pj, float (&v)[5]) const {
    RefLambdaTerms t;
    const bool ok = ref_lambda_terms(pi, pj, k, t);
    v[0] = ok ? t.poly : kNothing;
    v[1] = ok ? t.len : kNothing;
    v[2] = ok ? t.gx : kNothing;
    v[3] = ok ? t.gy : kNothing;
    v[4] = ok ? t.gz : kNothing;
  }
};
struct RcDeltaPass : RefSums<3> {
  const float4 *PS;
  const float *SS;
  const RefConsts &k;
  using Data = PSl;
  __device__ __forceinline__ RcDeltaPass(const float4 *ps, const float *ss, const RefConsts &c)
      : PS(ps), SS(ss), k(c) {}
  __device__ __forceinline__ PSl load(uint32_t j) const {
    return PSl{__ldg(&PS[j]), __ldg(&SS[j])};
  }
  __device__ __forceinline__ void pair(const PSl &i, const PSl &d, float (&v)[3]) const {
    RefTerms t;
    const bool ok = ref_delta_terms(i.p, i.s, d.p, d.s, k, t);
    v[0] = ok ? t.x : kNothing;
    v[1] = ok ? t.y : kNothing;
    v[2] = ok ? t.z : kNothing;
  }
};
struct RcXsphPass : RefSums<3> {
  const float4 *PS, *VS;
  const RefConsts &k;
  using Data = PV;
  __device__ __forceinline__ RcXsphPass(const float4 *ps, const float4 *vs, const RefConsts &c)
      : PS(ps), VS(vs), k(c) {}
  __device__ __forceinline__ PV load(uint32_t j) const { return PV{__ldg(&PS[j]), __ldg(&VS[j])}; }
  __device__ __forceinline__ void pair(const PV &i, const PV &d, float (&v)[3]) const {
    RefTerms t;
    const bool ok = ref_xsph_terms(i.p, i.v, d.p, d.v, k, t);
    v[0] = ok ? t.x : kNothing;
    v[1] = ok ? t.y : kNothing;
    v[2] = ok ? t.z : kNothing;
  }
};

__device__ __forceinline__ uint32_t group_particle() {
  return blockIdx.x * kCtaParticles + threadIdx.x / kGroup;
}
// Two entries of the group's shared list.
__device__ __forceinline__ uint2 list_two(const uint32_t *list, uint32_t q, uint32_t e) {
  return e < (uint32_t)kBuildList ? *reinterpret_cast<const uint2 *>(list + e) : make_uint2(q, q);
}

__global__ void __launch_bounds__(kGroupThreads)
    k_rc_group_lambda(float4 *PS, Planes planes, float *__restrict__ SS,
                      const uint32_t *__restrict__ off, uint32_t n, RefConsts k, uint32_t maxn,
                      uint4 *__restrict__ nbr4, uint32_t *__restrict__ nbr_cnt) {
  __shared__ __align__(16) float s_terms[kRefStride * kCtaParticles];
  __shared__ __align__(16) uint32_t s_list[kBuildList * kCtaParticles];
  const GroupIndex g(group_particle(), n);
  const uint32_t q = g.k, group = threadIdx.x / kGroup;
  uint32_t *list = s_list + group * kBuildList;
  const float4 pi = PS[q];
  uint32_t cnt = group_ref_scan(q, pi, k, off, planes, list);
  const bool held = cnt != kNotHeld;
  if (held && g.live)
    for (uint32_t w = lane_of_group(); 4u * w < min(cnt, maxn); w += kGroup)
      nbr4[(size_t)w * n + q] = *reinterpret_cast<const uint4 *>(list + 4u * w);
  const RcLambdaPass pass(PS, k);
  float t[5];
  group_sums(pass, pi, q, held ? cnt : 0u,
             [&](uint32_t, int, uint32_t e) { return list_two(list, q, e); },
             s_terms + group * kRefStride, t);
  if (!g.writes) return;
  RefLambdaSums s;
  if (held) {
    s.dens = t[0];
    s.gsum = t[1];
    s.gvx = t[2];
    s.gvy = t[3];
    s.gvz = t[4];
  } else {  // found by one thread
    cnt = scan_ref_members<false>(q, pi, k, off, planes, [&](uint32_t w, const uint4 &j) {
      if (4u * w < maxn) nbr4[(size_t)w * n + q] = j;
      const float4 d[4] = {PS[j.x], PS[j.y], PS[j.z], PS[j.w]};
#pragma unroll
      for (int e = 0; e < 4; ++e) s.add(pi, d[e], k);
    });
  }
  if (maxn) nbr_cnt[q] = cnt;
  ref_lambda_commit(q, s, k, PS, SS);
}

__global__ void __launch_bounds__(kGroupThreads)
    k_rc_group_delta(const float4 *__restrict__ PS, const float *__restrict__ SS, RefLists lists,
                     const uint32_t *__restrict__ off, RefConsts k, RcDeltaOut out) {
  __shared__ __align__(16) float s_terms[Terms<3>::kStride * kCtaParticles];
  const GroupIndex g(group_particle(), lists.n);
  const FirstEntries<EarlierKernel> first(lists, g.k);
  const PSl own{PS[g.k], SS[g.k]};
  const RcDeltaPass pass(PS, SS, k);
  float s[3];
  list_sums<EarlierKernel>(pass, own, lists, g.k, first,
                           s_terms + threadIdx.x / kGroup * Terms<3>::kStride, s,
                           [&](float (&t)[3]) {
                             t[0] = t[1] = t[2] = 0.0f;
                             ref_candidates(
                                 own.p, k, off, [&](uint32_t m) { return pass.load(m); },
                                 [&](const PSl &d) {
                                   RefTerms x;
                                   if (ref_delta_terms(own.p, own.s, d.p, d.s, k, x)) {
                                     t[0] += x.x;
                                     t[1] += x.y;
                                     t[2] += x.z;
                                   }
                                 });
                           });
  if (g.writes) ref_delta_commit(g.k, own.p, s[0], s[1], s[2], k, out);
}

__global__ void __launch_bounds__(kGroupThreads)
    k_rc_group_xsph(const float4 *__restrict__ PS, Planes planes, const float4 *__restrict__ VS,
                    float4 *__restrict__ DV, const uint32_t *__restrict__ input,
                    const uint32_t *__restrict__ off, uint32_t n, RefConsts k) {
  __shared__ __align__(16) float s_terms[Terms<3>::kStride * kCtaParticles];
  __shared__ __align__(16) uint32_t s_list[kBuildList * kCtaParticles];
  const GroupIndex g(group_particle(), n);
  const uint32_t q = g.k, group = threadIdx.x / kGroup;
  uint32_t *list = s_list + group * kBuildList;
  const PV own{PS[q], VS[q]};
  const uint32_t cnt = group_ref_scan(q, own.p, k, off, planes, list);
  const bool held = cnt != kNotHeld;
  const RcXsphPass pass(PS, VS, k);
  float s[3];
  group_sums(pass, own, q, held ? cnt : 0u,
             [&](uint32_t, int, uint32_t e) { return list_two(list, q, e); },
             s_terms + group * Terms<3>::kStride, s);
  if (!g.writes) return;
  if (!held) {
    s[0] = s[1] = s[2] = 0.0f;
    scan_ref_members<false>(q, own.p, k, off, planes, [&](uint32_t, const uint4 &j) {
      const uint32_t slot[4] = {j.x, j.y, j.z, j.w};
      for (int e = 0; e < 4; ++e) {
        RefTerms t;
        if (ref_xsph_terms(own.p, own.v, __ldg(&PS[slot[e]]), __ldg(&VS[slot[e]]), k, t)) {
          s[0] += t.x;
          s[1] += t.y;
          s[2] += t.z;
        }
      }
    });
  }
  DV[input[q]] = make_float4(0.01f * s[0], 0.01f * s[1], 0.01f * s[2], 0.0f);
}

// Keys of the sort elements (cells with z fastest, descending input index) as the
// cells of the particles with x fastest.
__global__ void __launch_bounds__(256)
    k_rc_view_keys(const uint32_t *__restrict__ keys, uint32_t n, uint32_t nx, uint32_t ny,
                   uint32_t nz, uint32_t *__restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t k = keys[n - 1u - i];
  const uint32_t z = k % nz, y = k / nz % ny, x = k / nz / ny;
  out[i] = x + nx * (y + ny * z);
}

__global__ void __launch_bounds__(256)
    k_rc_commit(float4 *__restrict__ X, float4 *__restrict__ V,
                const float4 *__restrict__ P, const float4 *__restrict__ DV,
                uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 p = P[i];
  const float4 dv = DV[i];
  float4 v = V[i];
  v.x += dv.x;
  v.y += dv.y;
  v.z += dv.z;
  V[i] = v;
  X[i] = make_float4(p.x, p.y, p.z, sqrtf(v.x * v.x + v.y * v.y + v.z * v.z));
}

inline uint32_t blocks_for(uint64_t n, uint32_t t) {
  return (uint32_t)((n + t - 1) / t);
}

}  // namespace

cudaError_t rc_predict_hash(float4 *X, float4 *V, float4 *P, uint32_t n,
                            const RefConsts &k, const SceneDesc *scenes,
                            uint32_t *keys, const SortPlan &plan,
                            uint32_t *sort_scratch, cudaStream_t st) {
  k_rc_predict_hash<<<min(blocks_for(n, 256), kStrideCtas), 256, 0, st>>>(
      X, V, P, n, k, scenes, keys, plan.passes, plan.digit_bits,
      sort_scratch + plan.off_hist);
  return cudaGetLastError();
}

cudaError_t rc_predict_count(float4 *X, float4 *V, float4 *P, uint32_t n, const RefConsts &k,
                             const SceneDesc *scenes, uint32_t *keys, const CellSortPlan &plan,
                             uint32_t *cell_scratch, cudaStream_t st) {
  k_rc_predict_count<<<min(blocks_for(n, 256), kStrideCtas), 256, 0, st>>>(
      X, V, P, n, k, scenes, keys, cell_scratch + plan.off_counts, cell_scratch + plan.off_pos);
  return cudaGetLastError();
}

cudaError_t rc_gather(const DeviceState &d, uint32_t n, const StepClear *clear, cudaStream_t st) {
  const auto kernel = clear ? k_rc_gather<true> : k_rc_gather<false>;
  kernel<<<blocks_for(n, 256), 256, 0, st>>>(d.P, d.perm, d.skeys, d.offsets,
                                             clear ? *clear : StepClear{}, n, d.PS, d.ID2,
                                             reinterpret_cast<float *>(d.io_pos), plane_floats(n));
  return cudaGetLastError();
}

cudaError_t rc_lambda(float4 *PS, const float4 *planes, float *SS, const uint32_t *offsets,
                      uint32_t n, const RefConsts &k, uint32_t maxn, uint4 *nbr,
                      uint32_t *nbr_cnt, cudaStream_t st) {
  if (n <= kRefGroupParticles)
    k_rc_group_lambda<<<blocks_for(n, kCtaParticles), kGroupThreads, 0, st>>>(
        PS, make_planes(planes, n), SS, offsets, n, k, maxn, nbr, nbr_cnt);
  else
    k_rc_lambda<<<blocks_for(n, kThreads), kThreads, 0, st>>>(PS, make_planes(planes, n), SS,
                                                              offsets, n, k, maxn, nbr, nbr_cnt);
  return cudaGetLastError();
}

cudaError_t rc_delta(const float4 *PS, float4 *PS2, const float *SS, const RefLists &lists,
                     const uint32_t *input, const uint32_t *offsets, const float4 *X, float4 *V,
                     float4 *P, float4 *VS, float4 *planes, uint32_t n, const RefConsts &k,
                     const SceneDesc *scenes, bool last, cudaStream_t st) {
  const RcDeltaOut out{PS2, V, P, VS, X, input, reinterpret_cast<float *>(planes),
                       plane_floats(n), scenes, last ? 1 : 0};
  if (n <= kRefGroupParticles && lists.maxn)
    k_rc_group_delta<<<blocks_for(n, kCtaParticles), kGroupThreads, 0, st>>>(PS, SS, lists,
                                                                             offsets, k, out);
  else
    k_rc_delta<<<blocks_for(n, kThreads), kThreads, 0, st>>>(PS, SS, lists, offsets, n, k, out);
  return cudaGetLastError();
}

cudaError_t rc_xsph(const float4 *PS, const float4 *planes, const float4 *VS, float4 *DV,
                    const uint32_t *input, const uint32_t *offsets, uint32_t n, const RefConsts &k,
                    cudaStream_t st) {
  if (n <= kRefGroupParticles)
    k_rc_group_xsph<<<blocks_for(n, kCtaParticles), kGroupThreads, 0, st>>>(
        PS, make_planes(planes, n), VS, DV, input, offsets, n, k);
  else
    k_rc_xsph<<<blocks_for(n, kThreads), kThreads, 0, st>>>(PS, make_planes(planes, n), VS, DV,
                                                            input, offsets, n, k);
  return cudaGetLastError();
}

cudaError_t rc_view_keys(const uint32_t *keys, uint32_t n, const SceneDesc &scene, uint32_t *out,
                         cudaStream_t st) {
  k_rc_view_keys<<<blocks_for(n, 256), 256, 0, st>>>(keys, n, (uint32_t)scene.ncell[0],
                                                     (uint32_t)scene.ncell[1],
                                                     (uint32_t)scene.ncell[2], out);
  return cudaGetLastError();
}

cudaError_t rc_commit(float4 *X, float4 *V, const float4 *P, const float4 *DV,
                      uint32_t n, cudaStream_t st) {
  k_rc_commit<<<blocks_for(n, 256), 256, 0, st>>>(X, V, P, DV, n);
  return cudaGetLastError();
}

}  // namespace pbf
