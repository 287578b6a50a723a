// Parameters and buffers of the headless renderer (render_kernels.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace nbg {

constexpr int kRenderMaxTaps = 32;

struct RenderUniforms {
  float pv[16];          // proj * view, column-major
  float flare_x;         // sprite half-size in NDC
  float flare_y;
  int32_t width;         // output image
  int32_t height;
  int32_t margin;        // HDR framebuffer margin (FBO_MARGIN)
  int32_t bw, bh;        // HDR framebuffer
  int32_t pitch;         // its row in pixels, even (two pixels are one 16-byte reduction)
  int32_t ow, oh;        // blur targets (downscaled by 2)
  int32_t lw, lh;        // luminance target (half size)
  int32_t flare_n;       // flare texture is flare_n x flare_n
  float size_x, size_y;  // blur sample step (blurDownscale / width, / height)
  int32_t taps;          // Gaussian taps (centre + taps - 1 symmetric pairs)
  float offset[kRenderMaxTaps];
  float weight[kRenderMaxTaps];
};

// Light is additive in two terms: a sprite's colour is (t, 0.4 (1 - t) + 0.2 t, 1) times
// its alpha, so sums of alpha and of alpha t give all three channels (light_rgb).
struct RenderBuffers {
  float2* hdr = nullptr;     // copies x (pitch x bh); the sum of them in the first
  float2* blur1 = nullptr;   // ow x oh
  float2* blur2 = nullptr;   // ow x oh (bloom)
  double* block_sums = nullptr;
  float* mean = nullptr;
  float* flare = nullptr;    // flare_n x flare_n
  int32_t width = 0, height = 0;
  int32_t copies = 1;
};

cudaError_t launch_render(const float* pos, const float4* vel, int64_t n_pad,
                          const RenderUniforms& u, const RenderBuffers& b, float4* out,
                          cudaStream_t stream);

// Copies of the HDR buffer that pay for n particles.
int render_copies(const RenderUniforms& u, int64_t n);

// Partial luminance sums of a frame.
int64_t render_luminance_parts(const RenderUniforms& u);

// Host tables shared by the renderer and its tests.
void render_gauss_tables(float sigma, int halfwidth, float* offsets, float* weights, int* taps);
void render_flare_texture(int n, float* pixels);

}  // namespace nbg
