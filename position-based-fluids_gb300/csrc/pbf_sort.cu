// Neighbour structure for the GB300 position-based-fluids step: cell hash,
// onesweep LSD radix sort of 32-bit cell keys, CSR cell offsets and the
// reference's inclusive cell ranges.
//
// Reference semantics this implements (MrMagne/position-based-fluids):
//   - cell hash: src/kernels/update_cells.cl:10-15 (and calc_hash.cl:15-20);
//   - a stable LSD radix sort of (cell, particle index) pairs, the intent of
//     src/kernels/radix_histogram.cl, radix_scan.cl, radix_paste.cl and
//     radix_reorder.cl driven by src/Simulation.cpp:351-435 (that code does
//     not run as shipped: radix_reorder.cl:28-41 uses an uninitialised
//     counter);
//   - inclusive [first,last] cell ranges with -1 for empty cells, the intent
//     of init_cells.cl and find_cells.cl.
//
// The sort is the onesweep scheme (one upfront histogram pass for every
// digit, then one pass per digit that ranks a tile of keys with warp-level
// multisplit, publishes per-digit tile counts and resolves its global
// offsets by decoupled look-back).  Digits are 8 bits wide, or 9 where that
// saves a pass within two passes: the 18-bit cell keys of a 64^3-cell grid
// take two 9-bit passes instead of three 8-bit ones.  Tiles are numbered by an atomic
// counter in the order CTAs start, so a CTA only ever waits on tiles that
// are already resident; every wait is additionally bounded, and a wait that
// runs out sets a device error bit instead of spinning on.
#include <algorithm>

#include "pbf_device.cuh"

namespace pbf {

namespace {

constexpr uint32_t kLbMask = (1u << 30) - 1u;
constexpr uint32_t kLbAggregate = 1u << 30;
constexpr uint32_t kLbInclusive = 2u << 30;
constexpr uint32_t kSpinLimit = 1u << 22;
constexpr int kSortWarps = kSortThreads / 32;
static_assert(kSortThreads == (1 << kMinDigitBits), "at least one digit per scan thread");
// A digit pass takes its tile with more threads of fewer keys: the ranking is a
// serial round per key of a warp, and a tile's time is the pass's latency while
// there are only a few tiles per SM (1M keys: 245 tiles).
constexpr int kSweepThreads = 512;
constexpr int kSweepItems = kSortTile / kSweepThreads;  // 8
constexpr int kSweepWarps = kSweepThreads / 32;
static_assert(kSweepThreads >= (1 << kMaxDigitBits), "a thread per digit");

__device__ __forceinline__ uint32_t ld_volatile(const uint32_t *p) {
  return *reinterpret_cast<const volatile uint32_t *>(p);
}
__device__ __forceinline__ void st_volatile(uint32_t *p, uint32_t v) {
  *reinterpret_cast<volatile uint32_t *>(p) = v;
}

// Exclusive scan of one value per thread over a block of kWarps warps.
template <int kWarps = kSortWarps>
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v,
                                                         uint32_t *s_warp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < kWarps ? s_warp[lane] : 0u;
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < kWarps; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    if (lane < kWarps) s_warp[lane] = wi - w;
  }
  __syncthreads();
  return incl - v + s_warp[warp];
}

// Two CTAs per SM: each adds its whole histogram to the global one, so more and
// smaller CTAs (1216 before) spend their time in those atomics.
constexpr uint32_t kHistThreads = 512;
constexpr uint32_t kHistCtas = 152u * 2u;
__global__ void __launch_bounds__(kHistThreads)
    k_sort_histogram(const uint32_t *__restrict__ keys, uint32_t n,
                     uint32_t passes, uint32_t digit_bits, uint32_t *__restrict__ hist) {
  __shared__ uint32_t s_hist[kMaxHistWords];
  const uint32_t hist_words = passes << digit_bits;
  for (uint32_t i = threadIdx.x; i < hist_words; i += blockDim.x) s_hist[i] = 0;
  __syncthreads();
  const uint32_t stride = gridDim.x * blockDim.x;
  // Whole warps iterate together.  Four keys per thread where the keys are
  // 16-byte aligned, then the rest one by one.
  const uint32_t words = (reinterpret_cast<uintptr_t>(keys) & 15u) == 0u ? n >> 2 : 0u;
  for (uint32_t base = blockIdx.x * blockDim.x; base < words; base += stride) {
    const uint32_t i = base + threadIdx.x;
    const bool valid = i < words;
    const uint4 k = valid ? __ldg(reinterpret_cast<const uint4 *>(keys) + i) : make_uint4(0, 0, 0, 0);
    warp_digit_histogram(k.x, valid, passes, digit_bits, s_hist);
    warp_digit_histogram(k.y, valid, passes, digit_bits, s_hist);
    warp_digit_histogram(k.z, valid, passes, digit_bits, s_hist);
    warp_digit_histogram(k.w, valid, passes, digit_bits, s_hist);
  }
  for (uint32_t base = 4u * words + blockIdx.x * blockDim.x; base < n; base += stride) {
    const uint32_t i = base + threadIdx.x;
    const bool valid = i < n;
    warp_digit_histogram(valid ? keys[i] : 0u, valid, passes, digit_bits, s_hist);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < hist_words; i += blockDim.x)
    if (s_hist[i]) atomicAdd(&hist[i], s_hist[i]);
}

// Look-back over groups of kLookGroup tiles.  A tile's word is its count
// (kLbAggregate), then the count of everything up to it (kLbInclusive); the last
// tile of a group gives its whole group's count instead of its own, which no
// other tile needs.  So a tile adds up to kLookGroup - 1 words of its own group,
// all in flight together, then the groups' words, again as many in flight: two
// or three L2 round trips after the last of them has its counts, where tiles
// that all start at once -- a sort of one wave -- walked up to 244 words behind
// each other, four at a time.  Sort of 1M keys of 18 bits 47.0 -> 43.2 us.
constexpr uint32_t kLookGroup = 16;

// Adds `count` words from `at` downwards, `step` words apart, as they are
// published; true when one of them was inclusive, or the wait gave up.
__device__ __forceinline__ bool look_back(const uint32_t *at, size_t step, uint32_t count,
                                          uint32_t &excl, uint32_t &spins, uint32_t spin_limit,
                                          uint32_t *err) {
  while (count > 0u) {
    uint32_t v[kLookGroup];
#pragma unroll
    for (uint32_t w = 0; w < kLookGroup; ++w) v[w] = w < count ? ld_volatile(at - w * step) : 0u;
    uint32_t taken = 0;
#pragma unroll
    for (uint32_t w = 0; w < kLookGroup; ++w) {
      if (taken != w || (v[w] & ~kLbMask) == 0u) continue;
      excl += v[w] & kLbMask;
      if ((v[w] & ~kLbMask) == kLbInclusive) return true;
      ++taken;
    }
    at -= taken * step;
    count -= taken;
    if (count == 0u) break;
    if (taken == 0u && ++spins >= spin_limit) {
      atomicOr(err, kDevErrLookback);
      return true;
    }
    if (spins > 64) __nanosleep(32);
  }
  return false;
}

// Publishes tile `tile`'s count of digit d and returns the count of all tiles
// before it.  Gives up (and reports through *err) after spin_limit polls without
// a new word, so a missing one cannot hang the GPU.
__device__ __forceinline__ uint32_t lookback_prefix(uint32_t *lookback, uint32_t radix,
                                                    uint32_t tile, uint32_t d, uint32_t count,
                                                    uint32_t spin_limit, uint32_t *err) {
  const uint32_t group = tile / kLookGroup, place = tile % kLookGroup;
  const bool leads = place == kLookGroup - 1u;
  uint32_t *mine = lookback + (size_t)tile * radix + d;
  uint32_t excl = 0, spins = 0;
  if (!leads) st_volatile(mine, (tile == 0 ? kLbInclusive : kLbAggregate) | count);
  if (tile == 0) return 0u;
  bool done = look_back(mine - radix, radix, place, excl, spins, spin_limit, err);
  if (!done && group > 0u) {
    if (leads) st_volatile(mine, kLbAggregate | (excl + count));
    look_back(lookback + ((size_t)group * kLookGroup - 1u) * radix + d,
              (size_t)kLookGroup * radix, group, excl, spins, spin_limit, err);
  }
  st_volatile(mine, kLbInclusive | ((excl + count) & kLbMask));
  return excl;
}

// Runs the look-back wait of one digit against a predecessor tile that
// never publishes (the words are zero): the wait must give up after
// spin_limit polls and report through *err.
__global__ void k_wait_selftest(uint32_t *lookback, uint32_t spin_limit, uint32_t *err) {
  if (threadIdx.x == 0) lookback_prefix(lookback, 1u << kMinDigitBits, 1u, 0u, 0u, spin_limit, err);
}

// Dynamic shared memory of one digit pass with 2^kBits digits.
constexpr size_t onesweep_smem_bytes(uint32_t bits) {
  return ((size_t)2u * kSweepWarps * (1u << bits) + 2u * (1u << bits) + 2u * kSortTile) *
         sizeof(uint32_t);
}

template <uint32_t kBits, bool kIota>
__global__ void __launch_bounds__(kSweepThreads)
    k_onesweep(const uint32_t *__restrict__ keys_in,
               const uint32_t *__restrict__ vals_in,
               uint32_t *__restrict__ keys_out, uint32_t *__restrict__ vals_out,
               uint32_t n, uint32_t shift,
               const uint32_t *__restrict__ hist,
               uint32_t *lookback, uint32_t *tile_counter, uint32_t *err) {
  constexpr uint32_t R = 1u << kBits;
  extern __shared__ __align__(16) uint32_t s_dyn[];
  uint32_t(*s_wcnt)[R] = reinterpret_cast<uint32_t(*)[R]>(s_dyn);  // [kSweepWarps][R]
  uint32_t(*s_match)[R] = s_wcnt + kSweepWarps;
  uint32_t *s_dexcl = s_dyn + 2u * kSweepWarps * R;
  uint32_t *s_gbase = s_dexcl + R;
  uint32_t *s_keys = s_gbase + R;
  uint32_t *s_vals = s_keys + kSortTile;
  __shared__ uint32_t s_tile;
  __shared__ uint32_t s_warp[kSweepWarps];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) s_tile = atomicAdd(tile_counter, 1u);
  for (uint32_t i = tid; i < 2u * kSweepWarps * R / 4u; i += kSweepThreads)
    reinterpret_cast<uint4 *>(s_dyn)[i] = make_uint4(0u, 0u, 0u, 0u);
  const uint32_t d = (uint32_t)tid;  // the digit this thread sees to after the ranks
  const uint32_t total = d < R ? __ldg(&hist[d]) : 0u;
  __syncthreads();

  const uint32_t tile = s_tile;
  const uint32_t tile_base = tile * (uint32_t)kSortTile;
  // Each warp owns a contiguous segment of 32*kSweepItems keys and reads it
  // lane-striped; the warp-local order (item, lane) is the input order.
  const uint32_t seg = tile_base + (uint32_t)warp * (32u * kSweepItems);

  uint32_t key[kSweepItems], val[kSweepItems], rank[kSweepItems];
#pragma unroll
  for (int it = 0; it < kSweepItems; ++it) {
    const uint32_t idx = seg + (uint32_t)it * 32u + lane;
    const bool ok = idx < n;
    key[it] = ok ? keys_in[idx] : 0u;
    val[it] = ok ? (kIota ? idx : vals_in[idx]) : 0u;
  }

  // Keys of lower digits in all tiles, while this tile's keys are on their way
  // (a launch of its own for this scan took 3.4 us and its gap).
  const uint32_t global_excl = block_exclusive_scan<kSweepWarps>(total, s_warp);

  // Warp-level multisplit: stable rank of each key among the warp's keys of
  // the same digit, item by item; the lanes of a digit find each other through
  // a word of shared memory.  (With a ballot per digit bit the ranks took 3,640
  // cycles of a tile, 6,500 with two tiles on the SM: 12 cycles a ballot.  1M
  // keys of 18 bits 43.2 -> 39.0 us, 4M 111 -> 100; __match_any_sync, a round
  // per distinct value, was slower still.)
  const unsigned lt_mask = (1u << lane) - 1u;
#pragma unroll
  for (int it = 0; it < kSweepItems; ++it) {
    const uint32_t idx = seg + (uint32_t)it * 32u + lane;
    const bool ok = idx < n;
    const uint32_t dg = (key[it] >> shift) & (R - 1);
    // one digit throughout (keys in order): known without 32 turns at one word
    // (4M equal keys 109 -> 85 us, random ones 100 -> 101)
    const uint32_t dg0 = __shfl_sync(0xffffffffu, dg, 0);
    if (__all_sync(0xffffffffu, ok && dg == dg0)) {
      const uint32_t before = s_wcnt[warp][dg];
      __syncwarp();
      rank[it] = before + (uint32_t)lane;
      if (lane == 31) s_wcnt[warp][dg] = before + 32u;
      __syncwarp();
      continue;
    }
    if (ok) atomicOr(&s_match[warp][dg], 1u << lane);
    __syncwarp();
    const unsigned peers = s_match[warp][dg];
    const uint32_t before = s_wcnt[warp][dg];
    __syncwarp();
    rank[it] = before + (uint32_t)__popc(peers & lt_mask);
    if (ok && lane == 31 - __clz(peers)) {
      s_match[warp][dg] = 0u;
      s_wcnt[warp][dg] = before + (uint32_t)__popc(peers);
    }
    __syncwarp();
  }
  __syncthreads();

  // Per digit (one thread each): the tile's count, and each warp's exclusive
  // offset.
  uint32_t tile_count = 0, excl = 0;
  if (d < R) {
    uint32_t x[kSweepWarps];
#pragma unroll
    for (int w = 0; w < kSweepWarps; ++w) x[w] = s_wcnt[w][d];
#pragma unroll
    for (int w = 0; w < kSweepWarps; ++w) {
      s_wcnt[w][d] = tile_count;
      tile_count += x[w];
    }
    excl = lookback_prefix(lookback, R, tile, d, tile_count, kSpinLimit, err);
  }
  const uint32_t e = block_exclusive_scan<kSweepWarps>(tile_count, s_warp);
  if (d < R) {
    s_gbase[d] = global_excl + excl;
    s_dexcl[d] = e;
  }
  __syncthreads();

  // Stage the tile in digit order in shared memory, then write it out with
  // consecutive threads on consecutive destinations.
#pragma unroll
  for (int it = 0; it < kSweepItems; ++it) {
    const uint32_t idx = seg + (uint32_t)it * 32u + lane;
    if (idx < n) {
      const uint32_t dg = (key[it] >> shift) & (R - 1);
      const uint32_t lp = s_dexcl[dg] + s_wcnt[warp][dg] + rank[it];
      s_keys[lp] = key[it];
      s_vals[lp] = val[it];
    }
  }
  __syncthreads();
  const uint32_t tile_n = min((uint32_t)kSortTile, n - tile_base);
#pragma unroll
  for (uint32_t it = 0; it < kSweepItems; ++it) {
    const uint32_t i = it * kSweepThreads + tid;
    key[it] = i < tile_n ? s_keys[i] : 0u;
    val[it] = i < tile_n ? s_vals[i] : 0u;
    const uint32_t dg = (key[it] >> shift) & (R - 1);
    rank[it] = i < tile_n ? s_gbase[dg] + (i - s_dexcl[dg]) : n;
  }
#pragma unroll
  for (uint32_t it = 0; it < kSweepItems; ++it) {
    // (also when a look-back wait gave up: error flag set)
    if (rank[it] >= n) continue;
    keys_out[rank[it]] = key[it];
    vals_out[rank[it]] = val[it];
  }
}

// Every instantiation takes its tile's shared memory dynamically (above the
// 48 KB static limit: 66 KB with 8-bit digits, 100 KB with 9-bit ones); the limit
// is raised once on each device.
OncePerDevice g_onesweep_once;

template <uint32_t kBits>
cudaError_t allow_onesweep_smem() {
  const int bytes = (int)onesweep_smem_bytes(kBits);
  cudaError_t e = cudaFuncSetAttribute(k_onesweep<kBits, false>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_onesweep<kBits, true>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  return e;
}

cudaError_t onesweep_init() {
  int device = 0;
  const cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  return g_onesweep_once.run(device, [] {
    const cudaError_t e = allow_onesweep_smem<8>();
    return e == cudaSuccess ? allow_onesweep_smem<9>() : e;
  });
}

template <uint32_t kBits>
void launch_onesweep(bool iota, uint32_t tiles, cudaStream_t stream, const uint32_t *ksrc,
                     const uint32_t *vsrc, uint32_t *kdst, uint32_t *vdst, uint32_t n,
                     uint32_t shift, const uint32_t *hist, uint32_t *lb, uint32_t *ctr,
                     uint32_t *err) {
  const size_t smem = onesweep_smem_bytes(kBits);
  if (iota)
    k_onesweep<kBits, true><<<tiles, kSweepThreads, smem, stream>>>(ksrc, nullptr, kdst, vdst, n,
                                                                  shift, hist, lb, ctr, err);
  else
    k_onesweep<kBits, false><<<tiles, kSweepThreads, smem, stream>>>(ksrc, vsrc, kdst, vdst, n,
                                                                   shift, hist, lb, ctr, err);
}

// off[c] = number of sorted keys < c, for c in [0, ncells]: one thread per
// cell, binary search over the sorted keys.  Neighbouring cells search
// neighbouring key ranges, so the probes of a warp share cache lines.
__global__ void k_cell_offsets(const uint32_t *__restrict__ skeys, uint32_t n,
                               uint32_t ncells, uint32_t *__restrict__ off) {
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c > ncells) return;
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = lo + ((hi - lo) >> 1);
    if (__ldg(&skeys[mid]) < c) lo = mid + 1;
    else hi = mid;
  }
  off[c] = lo;
}

constexpr uint32_t kShortRun = 64;    // cells a boundary thread writes itself
constexpr uint32_t kRunChunk = 4096;  // cells per queued chunk

// One thread per key boundary i in [0, n]: the cells (key[i-1], key[i]]
// (key[-1] = -1, key[n] = ncells) all take the value i -- the number of keys
// below each of them.  Short runs are written here, long ones queued.
__global__ void k_offset_runs(const uint32_t *__restrict__ skeys, uint32_t n, uint32_t ncells,
                              uint32_t *__restrict__ off, uint4 *__restrict__ runs,
                              uint32_t *__restrict__ runs_count, uint32_t runs_cap) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > n) return;
  const uint32_t lo = i == 0 ? 0u : min(skeys[i - 1], ncells - 1u) + 1u;
  const uint32_t hi = i == n ? ncells : min(skeys[i], ncells - 1u);
  if (hi < lo) return;
  const uint32_t count = hi - lo + 1u;
  if (count <= kShortRun) {
    for (uint32_t c = lo; c <= hi; ++c) off[c] = i;
    return;
  }
  const uint32_t chunks = (count + kRunChunk - 1u) / kRunChunk;
  const uint32_t slot = atomicAdd(runs_count, chunks);
  for (uint32_t q = 0; q < chunks; ++q) {
    const uint32_t a = lo + q * kRunChunk;
    const uint32_t len = min(kRunChunk, hi + 1u - a);
    if (slot + q < runs_cap) {
      runs[slot + q] = make_uint4(a, len, i, 0u);
    } else {  // beyond the capacity bound (keys out of order): write it here
      for (uint32_t c = a; c < a + len; ++c) off[c] = i;
    }
  }
}

// One CTA per queued chunk (grid-stride over the chunks).
__global__ void __launch_bounds__(256)
    k_offset_fill(const uint4 *__restrict__ runs, const uint32_t *__restrict__ runs_count,
                  uint32_t runs_cap, uint32_t *__restrict__ off) {
  const uint32_t total = min(*runs_count, runs_cap);
  for (uint32_t r = blockIdx.x; r < total; r += gridDim.x) {
    const uint4 e = runs[r];
    for (uint32_t t = threadIdx.x; t < e.y; t += blockDim.x) off[e.x + t] = e.z;
  }
}

__global__ void k_find_cells(const uint32_t *__restrict__ off, uint32_t ncells,
                             int2 *__restrict__ out) {
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncells) return;
  const uint32_t a = off[c], b = off[c + 1];
  out[c] = a < b ? make_int2((int)a, (int)(b - 1)) : make_int2(-1, -1);
}

// kHashItems positions of a thread on their way together (4.2M particles 17.7 ->
// 13.8 us; with fewer than a wave of threads each, one).
template <uint32_t kHashItems>
__global__ void __launch_bounds__(256)
    k_cell_hash(const float4 *__restrict__ pred, uint32_t n, SceneDesc scene,
                uint32_t *__restrict__ hash) {
  const uint32_t first = blockIdx.x * (256u * kHashItems) + threadIdx.x;
  float4 p[kHashItems];
#pragma unroll
  for (uint32_t e = 0; e < kHashItems; ++e)
    if (first + 256u * e < n) p[e] = __ldg(&pred[first + 256u * e]);
#pragma unroll
  for (uint32_t e = 0; e < kHashItems; ++e)
    if (first + 256u * e < n)
      hash[first + 256u * e] = scene.cell_base + scene_cell(p[e].x, p[e].y, p[e].z, scene);
}

inline uint32_t blocks_for(uint64_t n, uint32_t t) {
  return (uint32_t)((n + t - 1) / t);
}

// ------------------------------------------------- counting sort by cell --
// Cell keys sorted in one pass: each cell's particles are counted
// (count_cell_keys: one atomic per run of a warp's equal keys, each particle keeping
// its place among the increments of its cell) by the step's predict kernel or, for
// the operator, by k_count_keys; k_count_scan turns the counts into the cell offsets
// (and zeroes them for the next sort), and k_count_scatter puts every particle at
// its cell's offset plus its place.  The places of particles counted by different
// warps follow the order of their atomics, so the cells are then put back in index
// order -- the order a stable sort gives.  In a step the gather of the state does
// that for most cells (ordered_slot) and the scan lists the larger ones for
// k_cell_fix_big.  The operator runs k_cell_fix over all cells, which sorts those of
// up to 16 particles in registers (up to kLightCell on sparse grids) and lists the
// others.  k_cell_fix_big sorts listed cells of up to kBigCell in shared memory (one
// CTA per cell) and larger ones through a per-CTA bitmap of the particle indices.
constexpr uint32_t kScanItems = 8;                            // counts per thread and chunk
constexpr uint32_t kScanChunk = kSortThreads * kScanItems;   // 2048
constexpr uint32_t kScanChunks = 4;    // chunks per scan tile, where there are many
// Grids of few cells take one chunk per tile: the scan is then one chunk and
// the look-back over at most these tiles (they fit the control words).
constexpr uint32_t kFewTiles = 56;
constexpr uint32_t kSmallCell = 16;
// Cells of up to this many particles are sorted where sparse grids test them:
// listing a cell is an atomic on one word.  1M random keys in 2M cells 28.3 ->
// 11.9 us, 4.2M in 4.2M cells nearly in order 76 -> 22.
constexpr uint32_t kLightCell = 4;
constexpr uint32_t kWarpCell = 64;  // cells of 17..64 particles: one warp each
// control words: [0] scan tiles started, [1] big cells, [2] huge cells,
// [3] the operator's error word, [4] out-of-order small cells, [5] cells
// for one warp
constexpr uint32_t kCtlHeader = 8;
constexpr uint32_t kBigCell = 8192;

// Exclusive prefix of tile `tile` from the look-back words of the tiles
// before it, 32 tiles per round (lane l reads tile t - l; the nearest
// inclusive word ends the walk).  Runs on one full warp; a wait of more than
// spin_limit polls sets kDevErrLookback in *err and gives up.
__device__ __forceinline__ uint32_t warp_lookback(uint32_t *lookback, uint32_t tile,
                                                  uint32_t spin_limit, uint32_t *err) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t excl = 0;
  int t = (int)tile - 1;
  while (t >= 0) {
    const int p = t - (int)lane;
    uint32_t v = p >= 0 ? ld_volatile(&lookback[p]) : kLbInclusive;
    uint32_t spins = 0;
    bool gave_up = false;
    while (!__all_sync(0xffffffffu, (v & ~kLbMask) != 0u)) {
      if ((v & ~kLbMask) == 0u) v = ld_volatile(&lookback[p]);
      if (++spins >= spin_limit) {
        gave_up = true;
        break;
      }
      if (spins > 64) __nanosleep(32);
    }
    if (gave_up) {
      if (lane == 0) atomicOr(err, kDevErrLookback);
      break;
    }
    const unsigned inc = __ballot_sync(0xffffffffu, (v & ~kLbMask) == kLbInclusive);
    const uint32_t stop = inc ? (uint32_t)(__ffs(inc) - 1) : 31u;
    uint32_t part = lane <= stop ? (v & kLbMask) : 0u;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    excl += part;
    if (inc) break;
    t -= 32;
  }
  return excl;
}

// off[c] = particles in cells below c, for c in [0, ncells]; counts[c] -> 0.
// Tiles of kScanChunks chunks of 2048 counts (each thread holding 8
// consecutive counts of every chunk) are numbered in the order CTAs start.
// kList: cells of more than kRankCell particles are listed for k_cell_fix_big.
template <uint32_t kScanChunks, bool kList>
__global__ void __launch_bounds__(kSortThreads)
    k_count_scan(uint32_t *__restrict__ counts, uint32_t ncells, uint32_t total,
                 uint32_t *__restrict__ off, uint32_t *ctl, uint32_t *err,
                 uint32_t *__restrict__ big, uint32_t big_cap, uint32_t *__restrict__ huge,
                 uint32_t huge_cap) {
  constexpr uint32_t kScanTile = kScanChunk * kScanChunks;
  __shared__ uint32_t s_tile, s_excl;
  __shared__ uint32_t s_chunk[kScanChunks];
  __shared__ uint32_t s_warp[kScanChunks][kSortWarps];
  uint32_t *lookback = ctl + kCtlHeader;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  if (tid == 0) s_tile = atomicAdd(&ctl[0], 1u);
  __syncthreads();
  const uint32_t tile = s_tile;
  // every chunk's counts on their way together, then one scan of all chunks (a
  // step's cell sort at 1M 22.4 -> 20.8 us, at 4M 30.2 -> 28.4)
  uint32_t v[kScanChunks][kScanItems], sum[kScanChunks], texcl[kScanChunks];
#pragma unroll
  for (uint32_t q = 0; q < kScanChunks; ++q) {
    const uint32_t base = tile * kScanTile + q * kScanChunk + tid * kScanItems;
    // two 16-byte loads where the counts are 16-byte aligned (base is a
    // multiple of 8)
    if (whole_items(base, kScanItems, ncells) &&
        (reinterpret_cast<uintptr_t>(counts + base) & 15u) == 0u) {
      const uint4 a = *reinterpret_cast<const uint4 *>(counts + base);
      const uint4 b = *reinterpret_cast<const uint4 *>(counts + base + 4);
      v[q][0] = a.x; v[q][1] = a.y; v[q][2] = a.z; v[q][3] = a.w;
      v[q][4] = b.x; v[q][5] = b.y; v[q][6] = b.z; v[q][7] = b.w;
    } else {
#pragma unroll
      for (uint32_t j = 0; j < kScanItems; ++j) v[q][j] = base + j < ncells ? counts[base + j] : 0u;
    }
  }
#pragma unroll
  for (uint32_t q = 0; q < kScanChunks; ++q) {
    const uint32_t base = tile * kScanTile + q * kScanChunk + tid * kScanItems;
    uint32_t any = 0;
    sum[q] = 0;
#pragma unroll
    for (uint32_t j = 0; j < kScanItems; ++j) {
      any |= v[q][j];
      sum[q] += v[q][j];
    }
    if (any) {
      if (whole_items(base, kScanItems, ncells) &&
          (reinterpret_cast<uintptr_t>(counts + base) & 15u) == 0u) {
        *reinterpret_cast<uint4 *>(counts + base) = make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4 *>(counts + base + 4) = make_uint4(0, 0, 0, 0);
      } else {
#pragma unroll
        for (uint32_t j = 0; j < kScanItems; ++j)
          if (v[q][j]) counts[base + j] = 0u;
      }
    }
    if (kList) {
#pragma unroll
      for (uint32_t j = 0; j < kScanItems; ++j) {
        if (v[q][j] <= kRankCell) continue;
        if (v[q][j] <= kBigCell) {
          const uint32_t at = atomicAdd(&ctl[1], 1u);
          if (at < big_cap) big[at] = base + j;
        } else {
          const uint32_t at = atomicAdd(&ctl[2], 1u);
          if (at < huge_cap) huge[at] = base + j;
        }
      }
    }
    texcl[q] = sum[q];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, texcl[q], o);
      if (lane >= (uint32_t)o) texcl[q] += t;
    }
    if (lane == 31u) s_warp[q][warp] = texcl[q];
  }
  __syncthreads();
  if (warp < kScanChunks) {  // a chunk's warps by one warp
    const uint32_t w = lane < (uint32_t)kSortWarps ? s_warp[warp][lane] : 0u;
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < kSortWarps; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= (uint32_t)o) wi += t;
    }
    if (lane < (uint32_t)kSortWarps) s_warp[warp][lane] = wi - w;
    if (lane == (uint32_t)kSortWarps - 1u) s_chunk[warp] = wi;
  }
  __syncthreads();
#pragma unroll
  for (uint32_t q = 0; q < kScanChunks; ++q) texcl[q] += s_warp[q][warp] - sum[q];
  if (tid < 32) {
    uint32_t tot = 0;
#pragma unroll
    for (uint32_t q = 0; q < kScanChunks; ++q) tot += s_chunk[q];
    if (tile == 0) {
      if (tid == 0) {
        st_volatile(&lookback[0], kLbInclusive | tot);
        s_excl = 0;
        off[ncells] = total;
      }
    } else {
      if (tid == 0) st_volatile(&lookback[tile], kLbAggregate | tot);
      __syncwarp();
      const uint32_t excl = warp_lookback(lookback, tile, kSpinLimit, err);
      if (tid == 0) {
        st_volatile(&lookback[tile], kLbInclusive | ((excl + tot) & kLbMask));
        s_excl = excl;
      }
    }
  }
  __syncthreads();
  uint32_t carry = s_excl;
#pragma unroll
  for (uint32_t q = 0; q < kScanChunks; ++q) {
    const uint32_t base = tile * kScanTile + q * kScanChunk + tid * kScanItems;
    uint32_t run = carry + texcl[q];
    uint32_t o[kScanItems];
#pragma unroll
    for (uint32_t j = 0; j < kScanItems; ++j) {
      o[j] = run;
      run += v[q][j];
    }
    if (whole_items(base, kScanItems, ncells) &&
        (reinterpret_cast<uintptr_t>(off + base) & 15u) == 0u) {
      *reinterpret_cast<uint4 *>(off + base) = make_uint4(o[0], o[1], o[2], o[3]);
      *reinterpret_cast<uint4 *>(off + base + 4) = make_uint4(o[4], o[5], o[6], o[7]);
    } else {
#pragma unroll
      for (uint32_t j = 0; j < kScanItems; ++j)
        if (base + j < ncells) off[base + j] = o[j];
    }
    carry += s_chunk[q];
  }
}

// Every particle at its cell's offset plus its place among the cell's (four
// per thread where one per thread would be several waves of CTAs).
template <int kKeys>
__global__ void __launch_bounds__(256)
    k_count_scatter(const uint32_t *__restrict__ keys, const uint32_t *__restrict__ pos,
                    const uint32_t *__restrict__ off, uint32_t n, uint32_t ncells,
                    uint32_t *__restrict__ skeys, uint32_t *__restrict__ perm) {
  // kKeys keys per thread, their loads in flight together
  const uint32_t first = blockIdx.x * blockDim.x * kKeys + threadIdx.x;
  uint32_t k[kKeys], place[kKeys], d[kKeys];
#pragma unroll
  for (int u = 0; u < kKeys; ++u) {
    const uint32_t i = first + (uint32_t)u * blockDim.x;
    k[u] = i < n ? __ldg(&keys[i]) : 0xffffffffu;
    place[u] = i < n ? __ldg(&pos[i]) : 0u;
  }
#pragma unroll
  for (int u = 0; u < kKeys; ++u)  // a key not below ncells was not counted (error flag set)
    d[u] = k[u] < ncells ? __ldg(&off[k[u]]) + place[u] : 0xffffffffu;
#pragma unroll
  for (int u = 0; u < kKeys; ++u) {
    // always true unless the scan's look-back gave up (error flag set)
    if (d[u] < n) {
      skeys[d[u]] = k[u];
      perm[d[u]] = first + (uint32_t)u * blockDim.x;
    }
  }
}

// The counts and the control words to zero in one launch (a memset each: hash,
// sort and ranges of 4.2M particles 74.6 us instead of 73.9).
__global__ void __launch_bounds__(256)
    k_cell_clear(uint32_t *__restrict__ counts, uint32_t cells, uint32_t *__restrict__ ctl,
                 uint32_t words) {
  const uint32_t first = blockIdx.x * 256u + threadIdx.x, stride = gridDim.x * 256u;
  for (uint32_t i = first; i < cells; i = stride_next(i, stride, cells)) counts[i] = 0u;
  for (uint32_t i = first; i < words; i = stride_next(i, stride, words)) ctl[i] = 0u;
}

// The counting of the predict kernel, from a key array (the operator).
// A key outside [0, ncells) is not counted and sets kDevErrKey in *err.
__global__ void __launch_bounds__(256)
    k_count_keys(const uint32_t *__restrict__ keys, uint32_t n, uint32_t ncells,
                 uint32_t *__restrict__ counts, uint32_t *__restrict__ pos, uint32_t *err) {
  const uint32_t stride = gridDim.x * blockDim.x * kCountKeys;
  for (uint32_t base = blockIdx.x * blockDim.x * kCountKeys; base < n; base += stride) {
    uint32_t i[kCountKeys], key[kCountKeys];
    bool valid[kCountKeys];
#pragma unroll
    for (int u = 0; u < kCountKeys; ++u) {
      i[u] = base + (uint32_t)u * blockDim.x + threadIdx.x;
      key[u] = i[u] < n ? keys[i[u]] : 0u;
    }
#pragma unroll
    for (int u = 0; u < kCountKeys; ++u) {
      valid[u] = i[u] < n && key[u] < ncells;
      if (i[u] < n && !valid[u]) atomicOr(err, kDevErrKey);
    }
    count_cell_keys<true>(key, valid, i, counts, pos);
  }
}

// Steps kFrom, 2 kFrom, ... below kN of Batcher's odd-even merge sort of v: with
// kFrom = 1 a sort, with kFrom = kN / 2 the merge of two sorted halves.
template <uint32_t kFrom, uint32_t kN>
__device__ __forceinline__ void merge_steps(uint32_t *v) {
#pragma unroll
  for (uint32_t p = kFrom; p < kN; p <<= 1)
#pragma unroll
    for (uint32_t k = p; k > 0; k >>= 1)
#pragma unroll
      for (uint32_t i = 0; i + k < kN; ++i)
        if (i >= k % p && (i - k % p) % (2u * k) < k && i / (2u * p) == (i + k) / (2u * p)) {
          const uint32_t x = v[i], y = v[i + k];
          v[i] = min(x, y);
          v[i + k] = max(x, y);
        }
}

// The m <= kMost indices from perm[a] in order, in registers: all loaded
// together, none stored when they were in order, the upper half of the network
// left out where it is empty.  Cells of 4.2M particles in 15.2 -> 11 us against
// four loads at a time and a bitonic network of 80 exchanges (this one has 19
// for 8 indices, 63 for 16); bounded by its instructions, and slower with fewer
// than its 62 registers.
template <uint32_t kMost>
__device__ __forceinline__ void sort_cell(uint32_t *__restrict__ perm, uint32_t a, uint32_t m) {
  constexpr uint32_t kHalf = kMost / 2;
  uint32_t v[kMost];
#pragma unroll
  for (uint32_t j = 0; j < kMost; ++j) v[j] = j < m ? perm[a + j] : 0xffffffffu;
  bool sorted = true;
#pragma unroll
  for (uint32_t j = 1; j < kMost; ++j) sorted = sorted && v[j] >= v[j - 1];
  if (sorted) return;
  merge_steps<1, kHalf>(v);
  if (m > kHalf) {
    merge_steps<1, kHalf>(v + kHalf);
    merge_steps<kHalf, kMost>(v);
  }
#pragma unroll
  for (uint32_t j = 0; j < kMost; ++j)
    if (j < m) perm[a + j] = v[j];
}

// One thread per cell.  A cell of 2..kSmallCell particles whose indices are
// out of order (most are in order: their particles were counted by one warp)
// is sorted here (kSortHere, on grids with at least two particles per cell)
// or, on sparse grids, where this kernel runs over mostly empty cells and is
// kept light in registers, sorted here up to kLightCell particles and listed
// for k_cell_fix_big above; larger cells are listed by size.
template <bool kSortHere>
__global__ void __launch_bounds__(256)
    k_cell_fix(const uint32_t *__restrict__ off, uint32_t ncells, uint32_t *__restrict__ perm,
               uint32_t *__restrict__ small, uint32_t small_cap, uint32_t *__restrict__ med,
               uint32_t med_cap, uint32_t *__restrict__ big, uint32_t big_cap,
               uint32_t *__restrict__ huge, uint32_t huge_cap, uint32_t *ctl) {
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncells) return;
  const uint32_t a = off[c], m = off[c + 1] - a;
  if (m <= 1u) return;
  if (m > kSmallCell) {
    if (m <= kWarpCell) {
      const uint32_t q = atomicAdd(&ctl[5], 1u);
      if (q < med_cap) med[q] = c;
    } else if (m <= kBigCell) {
      const uint32_t q = atomicAdd(&ctl[1], 1u);
      if (q < big_cap) big[q] = c;
    } else {
      const uint32_t q = atomicAdd(&ctl[2], 1u);
      if (q < huge_cap) huge[q] = c;
    }
    return;
  }
  if (kSortHere) {
    sort_cell<kSmallCell>(perm, a, m);
    return;
  }
  if (m <= kLightCell) {
    sort_cell<kLightCell>(perm, a, m);
    return;
  }
  // four indices in flight at a time (past the cell's end its last one)
  uint32_t prev = perm[a];
  bool sorted = true;
#pragma unroll 1
  for (uint32_t j = 1; j < m && sorted; j += 4) {
    uint32_t x[4];
#pragma unroll
    for (uint32_t e = 0; e < 4; ++e) x[e] = perm[a + min(j + e, m - 1u)];
#pragma unroll
    for (uint32_t e = 0; e < 4; ++e) {
      sorted = sorted && x[e] >= prev;
      prev = x[e];
    }
  }
  if (sorted) return;
  const uint32_t q = atomicAdd(&ctl[4], 1u);
  if (q < small_cap) small[q] = c;
}

// A cell of up to 64 particles put back in index order by one warp: lane l
// holds entries l and l + 32, bitonic network across the warp.
__device__ __forceinline__ void warp_sort_cell(uint32_t *__restrict__ perm, uint32_t a,
                                               uint32_t m) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t v[2];
  v[0] = lane < m ? perm[a + lane] : 0xffffffffu;
  v[1] = lane + 32u < m ? perm[a + lane + 32u] : 0xffffffffu;
#pragma unroll
  for (uint32_t k = 2; k <= 64; k <<= 1)
#pragma unroll
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      if (j == 32) {  // entries lane and lane + 32, in this thread
        const uint32_t lo = min(v[0], v[1]), hi = max(v[0], v[1]);
        v[0] = lo;  // k = 64: ascending for every entry below 64
        v[1] = hi;
      } else {
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
          const uint32_t i = lane + 32u * h;
          const uint32_t y = __shfl_xor_sync(0xffffffffu, v[h], (int)j);
          const bool keep_min = ((i & j) == 0u) == ((i & k) == 0u);
          v[h] = keep_min ? min(v[h], y) : max(v[h], y);
        }
      }
    }
  if (lane < m) perm[a + lane] = v[0];
  if (lane + 32u < m) perm[a + lane + 32u] = v[1];
}

constexpr uint32_t kHugeCtas = 4;  // CTAs that take the huge cells (one bitmap each)

// The listed cells: up to kBigCell particles sorted in shared memory (one
// CTA per cell, bitonic); more through a bitmap of the particle indices
// (bm_words words per CTA, kHugeCtas CTAs): mark every index of the cell,
// then write the marked indices in ascending order.
__global__ void __launch_bounds__(kSortThreads)
    k_cell_fix_big(const uint32_t *__restrict__ off, uint32_t *__restrict__ perm,
                   const uint32_t *__restrict__ small, uint32_t small_cap,
                   const uint32_t *__restrict__ med, uint32_t med_cap,
                   const uint32_t *__restrict__ big, uint32_t big_cap,
                   const uint32_t *__restrict__ huge, uint32_t huge_cap, const uint32_t *ctl,
                   uint32_t *__restrict__ bitmap, uint32_t bm_words, uint32_t bm_stride) {
  __shared__ uint32_t s[kBigCell];
  __shared__ uint32_t s_warp[kSortWarps];
  __shared__ uint32_t s_total;
  const uint32_t tid = threadIdx.x;
  const uint32_t nsmall = min(ctl[4], small_cap);
  const uint32_t nbig = min(ctl[1], big_cap), nhuge = min(ctl[2], huge_cap);
  // the listed small cells: one thread each
  for (uint32_t w = blockIdx.x * kSortThreads + tid; w < nsmall; w += gridDim.x * kSortThreads) {
    const uint32_t c = small[w];
    const uint32_t a = off[c];
    sort_cell<kSmallCell>(perm, a, off[c + 1] - a);
  }
  // cells of 17..64: one warp each
  const uint32_t nmed = min(ctl[5], med_cap);
  for (uint32_t w = (blockIdx.x * kSortThreads + tid) >> 5; w < nmed;
       w += gridDim.x * kSortWarps) {
    const uint32_t c = med[w];
    const uint32_t a = off[c];
    warp_sort_cell(perm, a, off[c + 1] - a);
  }
  for (uint32_t b = blockIdx.x; b < nbig; b += gridDim.x) {
    const uint32_t c = big[b];
    const uint32_t a = off[c], m = off[c + 1] - a;
    uint32_t P = 1;
    while (P < m) P <<= 1;
    for (uint32_t i = tid; i < P; i += kSortThreads) s[i] = i < m ? perm[a + i] : 0xffffffffu;
    __syncthreads();
    for (uint32_t k = 2; k <= P; k <<= 1)
      for (uint32_t j = k >> 1; j > 0; j >>= 1) {
        for (uint32_t i = tid; i < P; i += kSortThreads) {
          const uint32_t l = i ^ j;
          if (l > i) {
            const uint32_t x = s[i], y = s[l];
            const bool up = (i & k) == 0u;
            if ((x > y) == up) {
              s[i] = y;
              s[l] = x;
            }
          }
        }
        __syncthreads();
      }
    for (uint32_t i = tid; i < m; i += kSortThreads) perm[a + i] = s[i];
    __syncthreads();
  }
  if (blockIdx.x >= kHugeCtas) return;
  uint32_t *bm = bitmap + (size_t)blockIdx.x * bm_stride;
  for (uint32_t h = blockIdx.x; h < nhuge; h += kHugeCtas) {
    const uint32_t c = huge[h];
    const uint32_t a = off[c], m = off[c + 1] - a;
    for (uint32_t w = tid; w < bm_words; w += kSortThreads) bm[w] = 0u;
    __syncthreads();
    for (uint32_t i = tid; i < m; i += kSortThreads) {
      const uint32_t x = perm[a + i];
      atomicOr(&bm[x >> 5], 1u << (x & 31u));
    }
    __syncthreads();
    uint32_t carry = 0;
    for (uint32_t w0 = 0; w0 < bm_words; w0 += kSortThreads) {
      const uint32_t w = w0 + tid;
      uint32_t word = w < bm_words ? bm[w] : 0u;
      const uint32_t cnt = (uint32_t)__popc(word);
      uint32_t at = a + carry + block_exclusive_scan(cnt, s_warp);
      if (tid == kSortThreads - 1) s_total = at - a - carry + cnt;
      while (word) {
        const uint32_t bit = (uint32_t)(__ffs(word) - 1);
        if (at < a + m) perm[at] = (w << 5) + bit;
        ++at;
        word &= word - 1u;
      }
      __syncthreads();
      carry += s_total;
      __syncthreads();
    }
  }
}

}  // namespace

uint32_t bits_for(uint32_t max_key_exclusive) {
  uint32_t b = 1;
  while (b < 32 && (1ull << b) < (uint64_t)max_key_exclusive) ++b;
  return b;
}

cudaError_t wait_selftest(uint32_t *scratch, uint32_t spin_limit, uint32_t *err,
                          cudaStream_t stream) {
  k_wait_selftest<<<1, 32, 0, stream>>>(scratch, spin_limit, err);
  return cudaGetLastError();
}

cudaError_t sort_clear(const SortPlan &plan, uint32_t *scratch,
                       cudaStream_t stream) {
  return cudaMemsetAsync(scratch + plan.off_hist, 0,
                         plan.clear_words * sizeof(uint32_t), stream);
}

cudaError_t sort_histogram(const SortPlan &plan, const uint32_t *keys,
                           uint32_t *scratch, cudaStream_t stream) {
  if (plan.n == 0) return cudaSuccess;
  const uint32_t blocks = min(blocks_for(plan.n, kHistThreads), kHistCtas);
  k_sort_histogram<<<blocks, kHistThreads, 0, stream>>>(keys, plan.n, plan.passes, plan.digit_bits,
                                               scratch + plan.off_hist);
  return cudaGetLastError();
}

cudaError_t sort_passes(const SortPlan &plan, const uint32_t *keys_in,
                        const uint32_t *vals_in, uint32_t *keys_out,
                        uint32_t *vals_out, uint32_t *scratch, uint32_t *err,
                        cudaStream_t stream) {
  if (plan.n == 0) return cudaSuccess;
  if (plan.digit_bits < kMinDigitBits || plan.digit_bits > kMaxDigitBits ||
      plan.passes > (uint32_t)kMaxSortPasses)
    return cudaErrorInvalidValue;
  const cudaError_t init = onesweep_init();
  if (init != cudaSuccess) return init;
  uint32_t *kalt = scratch + plan.off_keys_alt;
  uint32_t *valt = scratch + plan.off_vals_alt;
  // Arrange the ping-pong so the last pass writes keys_out/vals_out and the
  // inputs are never written.
  const uint32_t *ksrc = keys_in;
  const uint32_t *vsrc = vals_in;
  for (uint32_t p = 0; p < plan.passes; ++p) {
    const bool to_out = ((plan.passes - 1 - p) % 2) == 0;
    uint32_t *kdst = to_out ? keys_out : kalt;
    uint32_t *vdst = to_out ? vals_out : valt;
    uint32_t *hist = scratch + plan.off_hist + (size_t)p * plan.radix;
    uint32_t *lb = scratch + plan.off_lookback + (size_t)p * plan.tiles * plan.radix;
    uint32_t *ctr = scratch + plan.off_counter + p;
    const bool iota = p == 0 && vsrc == nullptr;
    const uint32_t shift = p * plan.digit_bits;
    if (plan.digit_bits == 8)
      launch_onesweep<8>(iota, plan.tiles, stream, ksrc, vsrc, kdst, vdst, plan.n, shift, hist,
                         lb, ctr, err);
    else
      launch_onesweep<9>(iota, plan.tiles, stream, ksrc, vsrc, kdst, vdst, plan.n, shift, hist,
                         lb, ctr, err);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    ksrc = kdst;
    vsrc = vdst;
  }
  return cudaSuccess;
}

cudaError_t cell_offsets(const uint32_t *sorted_keys, uint32_t n,
                         uint32_t ncells, uint32_t *offsets,
                         cudaStream_t stream) {
  if (n == 0) return cudaMemsetAsync(offsets, 0, (ncells + 1ull) * 4, stream);
  k_cell_offsets<<<blocks_for(ncells + 1ull, 256), 256, 0, stream>>>(
      sorted_keys, n, ncells, offsets);
  return cudaGetLastError();
}

uint32_t offset_runs_capacity(uint32_t ncells) {
  // every queued run is longer than kShortRun cells and adds one chunk per
  // kRunChunk cells or part of it
  const uint64_t cells = (uint64_t)ncells + 1u;
  return (uint32_t)(cells / (kShortRun + 1u) + cells / kRunChunk + 2u);
}

cudaError_t cell_offsets_runs(const uint32_t *sorted_keys, uint32_t n, uint32_t ncells,
                              uint32_t *offsets, uint4 *runs, uint32_t *runs_count,
                              cudaStream_t stream) {
  const uint32_t cap = offset_runs_capacity(ncells);
  cudaError_t e = cudaMemsetAsync(runs_count, 0, sizeof(uint32_t), stream);
  if (e != cudaSuccess) return e;
  k_offset_runs<<<blocks_for(n + 1ull, 256), 256, 0, stream>>>(sorted_keys, n, ncells, offsets,
                                                               runs, runs_count, cap);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_offset_fill<<<min(cap, kStrideCtas / 2u), 256, 0, stream>>>(runs, runs_count, cap, offsets);
  return cudaGetLastError();
}

cudaError_t find_cells(const uint32_t *offsets, uint32_t ncells,
                       int32_t *first_last, cudaStream_t stream) {
  if (ncells == 0) return cudaSuccess;
  k_find_cells<<<blocks_for(ncells, 256), 256, 0, stream>>>(
      offsets, ncells, reinterpret_cast<int2 *>(first_last));
  return cudaGetLastError();
}

cudaError_t cell_hash(const float4 *pred, uint32_t n, const SceneDesc &scene,
                      uint32_t *hash, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  if (n > kStrideCtas * 256u)
    k_cell_hash<4><<<blocks_for(n, 1024), 256, 0, stream>>>(pred, n, scene, hash);
  else
    k_cell_hash<1><<<blocks_for(n, 256), 256, 0, stream>>>(pred, n, scene, hash);
  return cudaGetLastError();
}

static void set_scan_tiles(CellSortPlan &p) {
  static_assert(kCtlHeader + kFewTiles <= 64, "the control words are padded to 64");
  const uint32_t few = (uint32_t)(((uint64_t)p.ncells + kScanChunk - 1) / kScanChunk);
  p.scan_chunks = few <= kFewTiles ? 1u : kScanChunks;
  p.tiles = (few + p.scan_chunks - 1) / p.scan_chunks;
  p.ctl_words = kCtlHeader + (size_t)p.tiles;
}

CellSortPlan make_cell_sort_plan(uint32_t n, uint32_t ncells) {
  CellSortPlan p;
  p.n = n;
  p.ncells = ncells;
  set_scan_tiles(p);
  p.rank_all = n <= kRankAllParticles;
  p.small_cap = (uint32_t)std::min<uint64_t>(ncells, (uint64_t)n / 2 + 1);
  p.med_cap = (uint32_t)std::min<uint64_t>(ncells, (uint64_t)n / (kSmallCell + 1) + 1);
  p.big_cap = (uint32_t)std::min<uint64_t>(ncells, (uint64_t)n / (kWarpCell + 1) + 1);
  p.huge_cap = n / (kBigCell + 1) + 1;
  p.bm_words = (n + 31u) / 32u;
  p.bm_stride = p.bm_words;
  size_t w = 0;
  p.off_counts = w;
  w += ncells;
  w = (w + 63) & ~size_t(63);
  p.off_pos = w;
  w += n;
  w = (w + 63) & ~size_t(63);
  p.off_ctl = w;
  // room for tiles of either size (kFewTiles of the small ones fit 64 words)
  w += kCtlHeader + (size_t)(((uint64_t)ncells + kScanChunk * kScanChunks - 1) /
                             (kScanChunk * kScanChunks));
  w = (w + 63) & ~size_t(63);
  p.off_small = w;
  w += p.small_cap;
  p.off_med = w;
  w += p.med_cap;
  p.off_big = w;
  w += p.big_cap;
  p.off_huge = w;
  w += p.huge_cap;
  w = (w + 63) & ~size_t(63);
  p.off_bitmap = w;
  w += (size_t)kHugeCtas * p.bm_stride;
  p.words = w;
  return p;
}

CellSortPlan resize_cell_sort_plan(const CellSortPlan &cap, uint32_t n, uint32_t ncells) {
  CellSortPlan p = cap;
  p.n = std::min(n, cap.n);
  p.ncells = std::min(ncells, cap.ncells);
  set_scan_tiles(p);
  p.bm_words = (p.n + 31u) / 32u;
  return p;
}

cudaError_t cell_sort_clear(const CellSortPlan &plan, uint32_t *scratch, cudaStream_t stream) {
  const uint32_t ctl = (uint32_t)cell_sort_clear_words(plan);
  k_cell_clear<<<min(blocks_for(max(plan.ncells, ctl), 1024), kStrideCtas), 256, 0, stream>>>(
      scratch + plan.off_counts, plan.ncells, scratch + plan.off_ctl, ctl);
  return cudaGetLastError();
}

// The offsets from the counts and every particle at its place.
template <bool kList>
static cudaError_t scan_and_scatter(const CellSortPlan &plan, const uint32_t *keys,
                                    uint32_t *scratch, uint32_t *offsets, uint32_t *skeys,
                                    uint32_t *perm, uint32_t *err, cudaStream_t stream) {
  if (plan.ncells == 0) return cudaErrorInvalidValue;
  const auto scan =
      plan.scan_chunks == 1 ? k_count_scan<1, kList> : k_count_scan<kScanChunks, kList>;
  scan<<<plan.tiles, kSortThreads, 0, stream>>>(
      scratch + plan.off_counts, plan.ncells, plan.n, offsets, scratch + plan.off_ctl, err,
      scratch + plan.off_big, plan.big_cap, scratch + plan.off_huge, plan.huge_cap);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || plan.n == 0) return e;
  const bool many = plan.n > kStrideCtas * 256u;
  const auto scatter = many ? k_count_scatter<kCountKeys> : k_count_scatter<1>;
  scatter<<<blocks_for(plan.n, many ? 256 * kCountKeys : 256), 256, 0, stream>>>(
      keys, scratch + plan.off_pos, offsets, plan.n, plan.ncells, skeys, perm);
  return cudaGetLastError();
}

static cudaError_t fix_big(const CellSortPlan &plan, uint32_t *scratch, const uint32_t *offsets,
                           uint32_t *perm, uint32_t ctas, cudaStream_t stream) {
  k_cell_fix_big<<<ctas, kSortThreads, 0, stream>>>(
      offsets, perm, scratch + plan.off_small, plan.small_cap, scratch + plan.off_med,
      plan.med_cap, scratch + plan.off_big, plan.big_cap, scratch + plan.off_huge, plan.huge_cap,
      scratch + plan.off_ctl, scratch + plan.off_bitmap, plan.bm_words, plan.bm_stride);
  return cudaGetLastError();
}

cudaError_t cell_sort_place(const CellSortPlan &plan, const uint32_t *keys, uint32_t *scratch,
                            uint32_t *offsets, uint32_t *skeys, uint32_t *perm, uint32_t *err,
                            cudaStream_t stream) {
  const cudaError_t e = scan_and_scatter<true>(plan, keys, scratch, offsets, skeys, perm, err,
                                               stream);
  if (e != cudaSuccess || plan.rank_all || plan.n == 0) return e;
  // at most n / (kRankCell + 1) cells are listed
  const uint32_t ctas = min(kStrideCtas / 4u, max(kHugeCtas, plan.n / (kRankCell + 1u) + 1u));
  return fix_big(plan, scratch, offsets, perm, ctas, stream);
}

cudaError_t cell_sort_finish(const CellSortPlan &plan, const uint32_t *keys, uint32_t *scratch,
                             uint32_t *offsets, uint32_t *skeys, uint32_t *perm, uint32_t *err,
                             cudaStream_t stream) {
  uint32_t *ctl = scratch + plan.off_ctl;
  cudaError_t e = scan_and_scatter<false>(plan, keys, scratch, offsets, skeys, perm, err, stream);
  if (e != cudaSuccess || plan.n == 0) return e;
  // dense grids sort their small cells in the pass over the cells, sparse
  // ones list them (measured: 1M particles in 64^3 cells, 14.6M in 14.6M)
  if ((uint64_t)plan.ncells * 2u <= plan.n)
    k_cell_fix<true><<<blocks_for(plan.ncells, 256), 256, 0, stream>>>(
        offsets, plan.ncells, perm, scratch + plan.off_small, plan.small_cap,
        scratch + plan.off_med, plan.med_cap, scratch + plan.off_big, plan.big_cap,
        scratch + plan.off_huge, plan.huge_cap, ctl);
  else
    k_cell_fix<false><<<blocks_for(plan.ncells, 256), 256, 0, stream>>>(
        offsets, plan.ncells, perm, scratch + plan.off_small, plan.small_cap,
        scratch + plan.off_med, plan.med_cap, scratch + plan.off_big, plan.big_cap,
        scratch + plan.off_huge, plan.huge_cap, ctl);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return fix_big(plan, scratch, offsets, perm, kStrideCtas / 4u, stream);
}

cudaError_t cell_sort_count(const CellSortPlan &plan, const uint32_t *keys, uint32_t *scratch,
                            uint32_t *err, cudaStream_t stream) {
  if (plan.n == 0) return cudaSuccess;
  k_count_keys<<<min(blocks_for(plan.n, 256 * kCountKeys), kStrideCtas), 256, 0, stream>>>(
      keys, plan.n, plan.ncells, scratch + plan.off_counts, scratch + plan.off_pos, err);
  return cudaGetLastError();
}

}  // namespace pbf
