// Host-side helpers shared by the C-ABI translation units (no device code).
#pragma once

#include <cuda_runtime.h>

#include <string>

#include "pbf.h"
#include "pbf_internal.cuh"

namespace pbf {

// Records the text of a CUDA error for pbf_last_error_message and maps it to
// a status code.
int cuda_status(cudaError_t e, const char *where);
void set_error_message(const std::string &msg);

// The reference's constant baking (src/main.cpp:149-168): a value printed
// with std::showpoint at precision 6 and read back as a float literal.
float baked6(double v);

// Derived constants.  `h` is (x_max - x_min) / x_n in float arithmetic, as
// src/main.cpp:164 computes it.
float params_h(const pbf_params &p);
RefConsts make_ref_consts(const pbf_params &p);
PaperConsts make_paper_consts(const pbf_params &p, uint32_t n);
// Scene descriptor of the whole box of `p` (grid origin, cell lengths,
// clamp bounds).  cell_base / particle range are left for the caller.
SceneDesc make_scene(const pbf_params &p);
// Validates a parameter set for a simulation of n particles.
int validate_params(const pbf_params &p, uint32_t n);
uint64_t grid_cells(const pbf_params &p);

// Checks a scene for a batch (grid, cell lengths against the batch's h) and
// returns the batch's solver settings with the scene's box, grid and walls,
// and the scene's cell count.  No capacity check.
int batch_check_scene(const pbf_batch *b, const pbf_params &scene, uint32_t n,
                      pbf_params *merged, uint64_t *cells);
void batch_capacity(const pbf_batch *b, uint32_t *scenes, uint32_t *particles,
                    uint32_t *cells);

// pbf_tuning <-> GatherTuning.  to_gather_tuning returns PBF_ERR_INVALID for
// a shape outside 64/128/256 threads and 4/8 loads in flight.
void to_pbf_tuning(const GatherTuning &g, const double trial_ms[kGatherKinds], pbf_tuning *out);
int to_gather_tuning(const pbf_tuning &t, GatherTuning *out);

// Device memory of the renderer, kept by the simulation or batch it draws
// (11 bytes per pixel of the largest image so far and 4 per particle):
// allocating it for every image took 160 us of a 1280 x 720 one.
struct RenderScratch {
  void *data = nullptr;
  size_t bytes = 0;
  cudaError_t reserve(size_t need) {
    if (need <= bytes) return cudaSuccess;
    release();
    const cudaError_t e = cudaMalloc(&data, need);
    if (e == cudaSuccess) bytes = need;
    else data = nullptr;
    return e;
  }
  void release() {
    if (data) cudaFree(data);
    data = nullptr;
    bytes = 0;
  }
};

// Sprites drawn in two parts, the second without what the first hides
// (k_render_splat_rest): images of many sprites that hide each other.  Frames in
// one part and in two: 152k particles at 1280 x 720 185 and 151 us, at 320 x 200
// 142 and 101, 1M at 1920 x 1080 401 and 299; with fewer sprites the two parts
// do not fill the GPU (69k at 1280 x 720 162 and 175, 33k at 640 x 360 105 and
// 143), in larger images fewer lie behind others (91k at 1920 x 1080 259 and
// 293), and small sprites take less time than placing them twice (134k of five
// pixels across 113 and 127, 160k of ten 97 and 89).  Between a quarter and a
// sixteenth of the sprites first, an eighth was best.
constexpr uint32_t kCullSprites = 81920;
constexpr uint32_t kCullPixels = 14;       // of the image per sprite, at most
constexpr float kCullDrawn = 10485760.0f;  // pixels of all sprites, at least
// (size: of a sprite at the camera's target, in pixels)
inline bool draws_in_two_parts(uint32_t n, uint32_t pixels, float size) {
  return n >= kCullSprites && (uint64_t)n * kCullPixels >= pixels &&
         (float)n * size * size >= kCullDrawn;
}

// Threads per sprite and per CTA, the CTAs of `count` sprites, and the sprite of a
// thread (eight threads per sprite number past 2^32 at 2^29 sprites).
constexpr uint32_t kSpriteThreads = 8, kSpriteCta = 128;
inline uint32_t sprite_ctas(uint32_t count) {
  return (uint32_t)(((uint64_t)count * kSpriteThreads + kSpriteCta - 1u) / kSpriteCta);
}
PBF_HOST_DEVICE inline uint32_t sprite_of_thread(uint32_t block, uint32_t thread) {
  return block * (kSpriteCta / kSpriteThreads) + thread / kSpriteThreads;
}

// Renders n particles (X: position, .w = |v|; ID: input index of each slot,
// or null when slot = input index) of the box of `prm` into rgb (host).
int render_particles(const float4 *X, const uint32_t *ID, uint32_t n, const pbf_params &prm,
                     const pbf_camera &cam, uint32_t width, uint32_t height, uint8_t *rgb,
                     RenderScratch &scratch, cudaStream_t st);

}  // namespace pbf
