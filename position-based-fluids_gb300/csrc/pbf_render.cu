// Headless particle renderer: the reference's point-sprite drawing restated
// as CUDA kernels writing an RGB8 image (no graphics stack).
//
// Reference: the particle pass of CVisual::visualizeParticles
// (src/visual/visual.cpp:270-330) with the camera of
// CVisual::resolveCamPosition / calcLookAtMatrix (:86-125) and the matrices
// set up at :217-227 (glm::perspective(45, w/h, 0.1, 1000), the box moved to
// be centred on the origin); the vertex shader
// (src/shaders/particlevertex.glsl: gl_PointSize = 200 / clip.w) and the
// fragment shader (src/shaders/particlefragment.glsl: a sphere normal from
// gl_PointCoord, discard outside the unit disc, colour (|v|, |v|, 1) times
// clamp(dot(n, (1,1,1)), 0, 1)); depth test GL_LESS with depth cleared to 1
// and colour cleared to 0.05 grey.
//
// The translation unit is compiled with -fmad=false (and its host code
// without floating-point contraction): every expression rounds operator by
// operator in IEEE binary32, with correctly rounded division and square
// root, so the image is reproducible bit for bit by a restatement that
// evaluates the same expressions in the same order.
//
// GL rasterises points in submission order; here each pixel keeps the
// fragment of least depth, ties to the lowest input index (the particle GL
// would have drawn first), through a 64-bit atomicMin on (depth bits, index),
// so the image does not depend on thread scheduling.  A second pass shades
// every pixel from its winning particle.
#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <cstring>

#include "pbf_host.hpp"

namespace pbf {
namespace {

struct RenderView {
  float m[16];        // clip = m * (p, 1), column-major like glm
  float width, height;
  float max_size;     // largest point size in pixels
  float half[3];      // box centre offset (model-to-world translation)
};

// Sprite of particle position p: window centre (x, y), window depth z and
// point size s.  False if GL would clip the point (centre outside the view
// volume).
__device__ __forceinline__ bool sprite(const RenderView &v, float px, float py, float pz,
                                       float &x, float &y, float &z, float &s) {
  const float wx = px + v.half[0], wy = py + v.half[1], wz = pz + v.half[2];
  const float cx = v.m[0] * wx + v.m[4] * wy + v.m[8] * wz + v.m[12];
  const float cy = v.m[1] * wx + v.m[5] * wy + v.m[9] * wz + v.m[13];
  const float cz = v.m[2] * wx + v.m[6] * wy + v.m[10] * wz + v.m[14];
  const float cw = v.m[3] * wx + v.m[7] * wy + v.m[11] * wz + v.m[15];
  if (!(cw > 0.0f) || fabsf(cx) > cw || fabsf(cy) > cw || fabsf(cz) > cw) return false;
  const float inv = 1.0f / cw;
  x = (cx * inv + 1.0f) * 0.5f * v.width;
  y = (cy * inv + 1.0f) * 0.5f * v.height;
  z = (cz * inv + 1.0f) * 0.5f;
  s = fminf(200.0f * inv, v.max_size);
  return true;
}

// gl_PointCoord mapped to [-1, 1]^2 for the pixel whose lower-left corner is
// (ix, iy) in window coordinates (origin lower left; point coordinates have
// their origin at the sprite's upper left).
__device__ __forceinline__ void point_coord(float x, float y, float s, int ix, int iy,
                                            float &mx, float &my) {
  const float u = ((float)ix + 0.5f - (x - 0.5f * s)) / s;
  const float w = ((y + 0.5f * s) - ((float)iy + 0.5f)) / s;
  mx = u * 2.0f - 1.0f;
  my = w * 2.0f - 1.0f;
}

// An empty image, and the slot of each input index (ID null: not needed), in one
// launch: frames of 152k particles at 1280 x 720 162.5 -> 154.9 us.
__global__ void k_render_clear(unsigned long long *__restrict__ zbuf, uint32_t pixels,
                               const uint32_t *__restrict__ ID, uint32_t n,
                               uint32_t *__restrict__ slot_of) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < pixels) zbuf[i] = ~0ull;
  if (ID && i < n) slot_of[min(ID[i], n - 1u)] = i;
}

// One sprite by eight threads: a thread's column, and rows eight at a time with
// each row's coordinate computed by one of the threads -- two divisions per
// thread and 64 pixels, where a thread per sprite divided twice per pixel.  A
// pixel is only written when its key beats what is there by now: in a fluid
// most particles lie behind others, and the atomics on pixels that can no
// longer change were the cost.  The first `count` particles of an order unlike
// their places are taken: an order from back to front would still write every
// pixel every time.  All of 152k particles at 1280 x 720, some 300 pixels each:
// 322 -> 91 us (99 in slot order), bound by its instructions, 37 per warp and
// pixel row.  An eighth of them takes 28 us: with every sprite in flight at
// once most of their pixels are atomics.
__global__ void __launch_bounds__(kSpriteCta)
    k_render_splat(const float4 *__restrict__ X, const uint32_t *__restrict__ ID, uint32_t n,
                   uint32_t count, uint32_t stride, RenderView v, unsigned long long *zbuf) {
  const uint32_t lane = threadIdx.x & (kSpriteThreads - 1u);
  const unsigned group = 0xffu << (threadIdx.x & 31u & ~(kSpriteThreads - 1u));
  const uint32_t i = sprite_of_thread(blockIdx.x, threadIdx.x);
  if (i >= count) return;
  const uint32_t k = (uint32_t)((uint64_t)i * stride % n);
  const float4 p = X[k];
  float x, y, z, s;
  if (!sprite(v, p.x, p.y, p.z, x, y, z, s)) return;  // the eight threads alike
  const uint32_t idx = ID ? ID[k] : k;
  const unsigned long long key = ((unsigned long long)__float_as_uint(z) << 32) | idx;
  const int W = (int)v.width, H = (int)v.height;
  // pixels whose centres fall inside the sprite square
  const int x0 = max(0, (int)ceilf(x - 0.5f * s - 0.5f));
  const int x1 = min(W - 1, (int)floorf(x + 0.5f * s - 0.5f));
  const int y0 = max(0, (int)ceilf(y - 0.5f * s - 0.5f));
  const int y1 = min(H - 1, (int)floorf(y + 0.5f * s - 0.5f));
  for (int ya = y0; ya <= y1; ya += (int)kSpriteThreads) {
    float unused, my_lane;
    point_coord(x, y, s, 0, ya + (int)lane, unused, my_lane);
    const float my2_lane = my_lane * my_lane;
    for (int xa = x0; xa <= x1; xa += (int)kSpriteThreads) {
      const int ix = xa + (int)lane;
      float mx, unused2;
      point_coord(x, y, s, ix, 0, mx, unused2);
      const float mx2 = mx * mx;
      const int rows = min((int)kSpriteThreads, y1 + 1 - ya);
      for (int r = 0; r < rows; ++r) {
        const float my2 = __shfl_sync(group, my2_lane, r, (int)kSpriteThreads);
        if (ix > x1 || mx2 + my2 > 1.0f) continue;
        unsigned long long *px = &zbuf[(size_t)(ya + r) * W + ix];
        if (key < __ldcg(px)) atomicMin(px, key);
      }
    }
  }
}

// The other sprites of the order, in blocks of eight by eight pixels of the
// image: only those not behind all of every block they touch (`far`: the largest
// depth of each block when the first sprites were drawn), and of those only the
// blocks they are not behind.  Depths only fall, so a block skipped could not
// change.  A warp takes 32 sprites, a lane each to place it (eight lanes placing
// the same sprite took 39 us instead of 27), then draws four at a time with
// eight threads as above, the eight rows' keys loaded together.  Frame of 152k
// particles at 1280 x 720: 185 -> 151 us, of which the copy of the image is half.
constexpr int kBlockSide = 8;
__global__ void __launch_bounds__(128)
    k_render_splat_rest(const float4 *__restrict__ X, const uint32_t *__restrict__ ID, uint32_t n,
                        uint32_t first, uint32_t count, uint32_t stride, RenderView v,
                        const uint32_t *__restrict__ far, unsigned long long *zbuf) {
  constexpr unsigned kWarp = 0xffffffffu;
  const uint32_t in_warp = threadIdx.x & 31u, lane = in_warp & (kSpriteThreads - 1u);
  const uint32_t shift = in_warp & ~(kSpriteThreads - 1u);
  const unsigned group = 0xffu << shift;
  const int W = (int)v.width, H = (int)v.height;
  const int across = (W + kBlockSide - 1) / kBlockSide;  // blocks of an image row
  const uint32_t i = blockIdx.x * 128u + threadIdx.x;
  float own_x = 0.f, own_y = 0.f, own_s = 0.f;
  uint32_t own_depth = 0, own_idx = 0, own_cols = 0, own_rows = 0;
  bool ok = i < count;
  if (ok) {
    const uint32_t k = (uint32_t)((uint64_t)(first + i) * stride % n);
    const float4 p = X[k];
    float z;
    ok = sprite(v, p.x, p.y, p.z, own_x, own_y, z, own_s);
    if (ok) {
      own_depth = __float_as_uint(z);
      own_idx = ID ? ID[k] : k;
      // pixels whose centres fall inside the sprite square
      const int x0 = max(0, (int)ceilf(own_x - 0.5f * own_s - 0.5f));
      const int x1 = min(W - 1, (int)floorf(own_x + 0.5f * own_s - 0.5f));
      const int y0 = max(0, (int)ceilf(own_y - 0.5f * own_s - 0.5f));
      const int y1 = min(H - 1, (int)floorf(own_y + 0.5f * own_s - 0.5f));
      ok = x0 <= x1 && y0 <= y1;
      own_cols = (uint32_t)x0 | (uint32_t)x1 << 16;  // (an image side is at most 16384)
      own_rows = (uint32_t)y0 | (uint32_t)y1 << 16;
      if (ok) {
        ok = false;
        for (int yb = y0 / kBlockSide; yb <= y1 / kBlockSide && !ok; ++yb)
          for (int xb = x0 / kBlockSide; xb <= x1 / kBlockSide; ++xb)
            ok = ok || own_depth <= far[yb * across + xb];
      }
    }
  }
  unsigned todo = __ballot_sync(kWarp, ok);
  while (todo) {
    // this group's sprite: the lowest of `todo`, the next one, ...
    unsigned left = todo;
#pragma unroll
    for (uint32_t g = 0; g < 3; ++g)
      if (g < shift / kSpriteThreads) left &= left - 1u;
    const int src = __ffs((int)left) - 1;
    const float x = __shfl_sync(kWarp, own_x, src), y = __shfl_sync(kWarp, own_y, src),
                s = __shfl_sync(kWarp, own_s, src);
    const uint32_t depth = __shfl_sync(kWarp, own_depth, src),
                   idx = __shfl_sync(kWarp, own_idx, src),
                   cols = __shfl_sync(kWarp, own_cols, src),
                   rows_of = __shfl_sync(kWarp, own_rows, src);
#pragma unroll
    for (int g = 0; g < 4; ++g) todo &= todo - 1u;
    const unsigned long long key = ((unsigned long long)depth << 32) | idx;
    const int x0 = (int)(cols & 0xffffu), x1 = (int)(cols >> 16);
    const int y0 = (int)(rows_of & 0xffffu), y1 = src < 0 ? -1 : (int)(rows_of >> 16);
    for (int ya = y0 & ~(kBlockSide - 1); ya <= y1; ya += kBlockSide) {
      float unused, my_lane;
      point_coord(x, y, s, 0, ya + (int)lane, unused, my_lane);
      const float my2_lane = my_lane * my_lane;
      const uint32_t rows =
          (0xffu << max(y0 - ya, 0)) & (0xffu >> max(ya + kBlockSide - 1 - y1, 0));
      for (int xs = x0 / kBlockSide; xs <= x1 / kBlockSide; xs += (int)kSpriteThreads) {
        const int xb = xs + (int)lane;
        bool draw = xb <= x1 / kBlockSide;
        if (draw) draw = depth <= far[ya / kBlockSide * across + xb];
        for (unsigned b = __ballot_sync(group, draw) >> shift & 0xffu; b; b &= b - 1u) {
          const int ix = (xs + __ffs((int)b) - 1) * kBlockSide + (int)lane;
          float mx, unused2;
          point_coord(x, y, s, ix, 0, mx, unused2);
          const float mx2 = mx * mx;
          const uint32_t mine = ix < x0 || ix > x1 ? 0u : rows;  // of the sprite's square
          unsigned long long *px = &zbuf[(size_t)ya * W + ix];
          unsigned long long now[kBlockSide];
#pragma unroll
          for (int r = 0; r < kBlockSide; ++r) {
            const float my2 = __shfl_sync(group, my2_lane, r, (int)kSpriteThreads);
            now[r] = !(mine >> r & 1u) || mx2 + my2 > 1.0f ? 0ull : __ldcg(px + (size_t)r * W);
          }
#pragma unroll
          for (int r = 0; r < kBlockSide; ++r)
            if (key < now[r]) atomicMin(px + (size_t)r * W, key);
        }
      }
    }
    __syncwarp();
  }
}

// The largest depth of each block of the image, eight threads per block.
__global__ void __launch_bounds__(256)
    k_render_far(const unsigned long long *__restrict__ zbuf, int W, int H, uint32_t blocks,
                 uint32_t *__restrict__ far) {
  const uint32_t t = blockIdx.x * 256u + threadIdx.x;
  const uint32_t block = t / 8u;
  const int across = (W + kBlockSide - 1) / kBlockSide;
  const int ix = (int)(block % (uint32_t)across) * kBlockSide + (int)(t & 7u);
  const int ya = (int)(block / (uint32_t)across) * kBlockSide;
  uint32_t most = 0;
  if (block < blocks && ix < W)
#pragma unroll
    for (int r = 0; r < kBlockSide; ++r)
      if (ya + r < H) most = max(most, (uint32_t)(zbuf[(size_t)(ya + r) * W + ix] >> 32));
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
  if (block < blocks && (t & 7u) == 0u) far[block] = most;
}

// Shades every pixel from its winning particle; rows are written top first.
__global__ void k_render_shade(const float4 *__restrict__ X, const uint32_t *__restrict__ ID,
                               const uint32_t *__restrict__ slot_of, uint32_t n, RenderView v,
                               const unsigned long long *__restrict__ zbuf,
                               uint8_t *__restrict__ rgb) {
  const int W = (int)v.width, H = (int)v.height;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint32_t)(W * H)) return;
  const int ix = (int)(i % (uint32_t)W), iy = (int)(i / (uint32_t)W);
  float r = 0.05f, g = 0.05f, b = 0.05f;
  const unsigned long long key = zbuf[i];
  if (key != ~0ull) {
    const uint32_t idx = (uint32_t)(key & 0xffffffffu);
    const uint32_t k = min(ID ? slot_of[idx] : idx, n - 1u);
    const float4 p = X[k];
    float x, y, z, s, mx, my;
    if (sprite(v, p.x, p.y, p.z, x, y, z, s)) {
      point_coord(x, y, s, ix, iy, mx, my);
      const float l2 = mx * mx + my * my;
      const float nz = sqrtf(fmaxf(0.0f, 1.0f - l2));
      const float inv = 1.0f / sqrtf(fmaxf(l2 + nz * nz, 1e-30f));
      const float cosang = fminf(fmaxf((mx + my + nz) * inv, 0.0f), 1.0f);
      r = p.w * cosang;
      g = p.w * cosang;
      b = cosang;
    }
  }
  const size_t o = ((size_t)(H - 1 - iy) * W + ix) * 3;
  rgb[o + 0] = (uint8_t)__float2int_rn(fminf(fmaxf(r, 0.0f), 1.0f) * 255.0f);
  rgb[o + 1] = (uint8_t)__float2int_rn(fminf(fmaxf(g, 0.0f), 1.0f) * 255.0f);
  rgb[o + 2] = (uint8_t)__float2int_rn(fminf(fmaxf(b, 0.0f), 1.0f) * 255.0f);
}

// A step through the n particles that visits each once, in an order unlike
// their places: near 0.618 n and without a common factor.
uint32_t sprite_stride(uint32_t n) {
  uint32_t s = (uint32_t)(0.6180339887 * n) | 1u;
  const auto gcd = [](uint32_t a, uint32_t b) {
    while (b) {
      const uint32_t t = a % b;
      a = b;
      b = t;
    }
    return a;
  };
  while (gcd(s, n) != 1u) ++s;
  return s;
}

// glm-style column-major 4x4 helpers (host).
void mat_mul(const float a[16], const float b[16], float out[16]) {
  float r[16];
  for (int c = 0; c < 4; ++c)
    for (int row = 0; row < 4; ++row) {
      float acc = 0.f;
      for (int k = 0; k < 4; ++k) acc += a[k * 4 + row] * b[c * 4 + k];
      r[c * 4 + row] = acc;
    }
  std::memcpy(out, r, sizeof r);
}

}  // namespace

void render_view_matrix(const pbf_camera &cam, float aspect, float out[16]) {
  // camera position on the sphere around the target (visual.cpp:89-100)
  const double phi = M_PI / 180.0 * (cam.phi_deg - 90.0);
  const double theta = M_PI / 180.0 * (cam.theta_deg + 90.0);
  const float dir[3] = {(float)(std::sin(theta) * std::cos(phi)), (float)std::cos(theta),
                        (float)(std::sin(theta) * std::sin(phi))};
  float eye[3], look[3];
  for (int a = 0; a < 3; ++a) eye[a] = dir[a] * cam.distance + cam.target[a];
  for (int a = 0; a < 3; ++a) look[a] = cam.target[a] - eye[a];
  auto normalize = [](float v[3]) {
    const float l = std::sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    for (int a = 0; a < 3; ++a) v[a] /= l;
  };
  normalize(look);
  float up[3] = {0.f, 1.f, 0.f};
  float right[3] = {look[1] * up[2] - look[2] * up[1], look[2] * up[0] - look[0] * up[2],
                    look[0] * up[1] - look[1] * up[0]};
  normalize(right);
  const float pup[3] = {right[1] * look[2] - right[2] * look[1],
                        right[2] * look[0] - right[0] * look[2],
                        right[0] * look[1] - right[1] * look[0]};
  // view = R * T (visual.cpp:104-125)
  float view[16] = {right[0], pup[0], -look[0], 0.f, right[1], pup[1], -look[1], 0.f,
                    right[2], pup[2], -look[2], 0.f, 0.f,      0.f,    0.f,      1.f};
  float trans[16] = {1.f, 0.f, 0.f, 0.f, 0.f, 1.f, 0.f, 0.f,
                     0.f, 0.f, 1.f, 0.f, -eye[0], -eye[1], -eye[2], 1.f};
  mat_mul(view, trans, view);
  // perspective (glm::perspective with fovy in degrees)
  const float f = 1.0f / (float)std::tan(M_PI / 180.0 * cam.fovy_deg / 2.0);
  const float zn = cam.znear, zf = cam.zfar;
  float proj[16] = {0.f};
  proj[0] = f / aspect;
  proj[5] = f;
  proj[10] = -(zf + zn) / (zf - zn);
  proj[11] = -1.f;
  proj[14] = -(2.f * zf * zn) / (zf - zn);
  mat_mul(proj, view, out);
}

constexpr uint32_t kFirstSprites = 8;  // of two parts, the first: one sprite in so many

// More scratch than this is not kept from one image to the next.
constexpr size_t kRenderKeep = (size_t)256 << 20;

int render_particles(const float4 *X, const uint32_t *ID, uint32_t n, const pbf_params &prm,
                     const pbf_camera &cam, uint32_t width, uint32_t height, uint8_t *rgb,
                     RenderScratch &scratch, cudaStream_t st) {
  if (width == 0 || height == 0 || width > 16384 || height > 16384) return PBF_ERR_INVALID;
  RenderView v;
  render_view_matrix(cam, (float)width / (float)height, v.m);
  v.width = (float)width;
  v.height = (float)height;
  v.max_size = cam.max_point_size > 0.f ? cam.max_point_size : 64.f;
  // model-to-world: the box moved by minus half its extent (visual.cpp:219-223)
  v.half[0] = -(prm.x_max - prm.x_min) / 2.0f;
  v.half[1] = -(prm.y_max - prm.y_min) / 2.0f;
  v.half[2] = -(prm.z_max - prm.z_min) / 2.0f;
  const uint32_t pixels = width * height;
  int rc = PBF_OK;
  auto cuda = [&](cudaError_t e, const char *where) {
    if (e != cudaSuccess && rc == PBF_OK) rc = cuda_status(e, where);
    return rc == PBF_OK;
  };
  // depth keys, image (whole 16-byte words), depth of each block, slot of each
  // input index
  const uint32_t blocks = (width + kBlockSide - 1) / kBlockSide *
                          ((height + kBlockSide - 1) / kBlockSide);
  const size_t img_at = (size_t)pixels * 8, far_at = img_at + ((size_t)pixels * 3 + 15) / 16 * 16,
               slot_at = far_at + (size_t)blocks * 4;
  if (!cuda(scratch.reserve(slot_at + (ID ? (size_t)n * 4 : 0)), "render alloc")) return rc;
  unsigned char *base = static_cast<unsigned char *>(scratch.data);
  auto *zbuf = reinterpret_cast<unsigned long long *>(base);
  uint8_t *img = base + img_at;
  auto *far = reinterpret_cast<uint32_t *>(base + far_at);
  auto *slot_of = reinterpret_cast<uint32_t *>(base + slot_at);
  k_render_clear<<<((ID && n > pixels ? n : pixels) + 255) / 256, 256, 0, st>>>(zbuf, pixels, ID,
                                                                                n, slot_of);
  // (a sprite's size at the camera's target)
  const float size = std::fmin(200.0f / std::fabs(cam.distance), v.max_size);
  const bool cull = draws_in_two_parts(n, pixels, size);
  const uint32_t drawn = cull ? n / kFirstSprites : n;
  if (n)
    k_render_splat<<<sprite_ctas(drawn), kSpriteCta, 0, st>>>(
        X, ID, n, drawn, sprite_stride(n), v, zbuf);
  if (cull) {
    k_render_far<<<(blocks * 8u + 255u) / 256u, 256, 0, st>>>(zbuf, (int)width, (int)height,
                                                              blocks, far);
    k_render_splat_rest<<<(n - drawn + 127u) / 128u, 128, 0, st>>>(
        X, ID, n, drawn, n - drawn, sprite_stride(n), v, far, zbuf);
  }
  k_render_shade<<<(pixels + 255) / 256, 256, 0, st>>>(X, ID, slot_of, n ? n : 1u, v, zbuf, img);
  if (cuda(cudaGetLastError(), "render launch"))
    cuda(cudaMemcpyAsync(rgb, img, (size_t)pixels * 3, cudaMemcpyDeviceToHost, st), "render copy");
  cuda(cudaStreamSynchronize(st), "render sync");
  if (scratch.bytes > kRenderKeep) scratch.release();
  return rc;
}

}  // namespace pbf

extern "C" void pbf_camera_default(const pbf_params *p, pbf_camera *out) {
  if (!out) return;
  std::memset(out, 0, sizeof *out);
  // CVisual's initial camera sphere (visual.cpp:38-39) with the distance set
  // from the box depth (:225)
  out->phi_deg = 0.0f;
  out->theta_deg = 20.0f;
  out->distance = p ? -(p->z_max - p->z_min) * 2.0f : -1.0f;
  out->fovy_deg = 45.0f;
  out->znear = 0.1f;
  out->zfar = 1000.0f;
  out->max_point_size = 64.0f;
}
