// Headless render math of the reference's OpenGL renderer, as CUDA kernels.
//
// The reference draws every particle as an additive, velocity-coloured point
// sprite into an HDR framebuffer with a 50-pixel margin
// (src/renderer_gl.cpp:96-111; shaders/gl/main.{vert,geom,frag}).  It then blurs
// a half-resolution copy with a separable Gaussian (renderer_gl.cpp:113-137,
// shaders/gl/blur.frag), reduces luminance over a mip chain (renderer_gl.cpp:139-146,
// shaders/gl/luminance.frag), and tonemaps HDR + bloom with an exposure and
// gamma 2.2 (renderer_gl.cpp:148-156, shaders/gl/tonemap.frag).  Here the same
// arithmetic runs on device buffers: images are row-major with row 0 at the bottom
// (the framebuffer convention), sampling is bilinear with the texture's wrap mode, and
// blending is FP32 reductions (the reference's buffer is RGBA16F).
//
// What bounds a frame: the L2's reduction units, in the splat (about 70 pixels under
// each sprite).  Everything up to the tonemap is linear in two sums per pixel, of alpha
// and of alpha t (RenderBuffers), so buffers hold a float2 per pixel, and one 16-byte
// reduction adds to two neighbouring pixels.  1,048,576 particles at 1920 x 1080: 597 us
// per frame with a float4 per pixel and a thread per particle, 269 with a lane per pair
// of pixels, 220 with the profile evaluated once per column and row (the splat is bound
// by instructions then: 2 x 2 pixels per sector, a fifth fewer sectors, gain nothing),
// 198 with the kernels as programmatic dependents and the blur's taps fixed, 185 with the
// blur's taps as pairs from shared memory and a gamma of its own (188 with the sprites'
// places rounded more finely).
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "nb_device.cuh"
#include "nb_internal.hpp"
#include "nb_render.hpp"

namespace nbg {
namespace {

constexpr int kFlareMax = 64;     // largest flare texture
constexpr int kSplatThreads = 256;

// The three channels of a pixel's sums (a: of alpha, t: of alpha t).
__device__ __forceinline__ float3 light_rgb(float a, float t) {
  return make_float3(t, 0.4f * (a - t) + 0.2f * t, a);
}

// Row of the flare texture through its centre, by linear interpolation with repeat wrap
// (its sampler never sets a wrap mode, renderer_gl.cpp:53-63).  The texture is a product
// of this profile along both axes (gen.cpp:36-51).  tab[k]: texel (k - 1) mod n.
__device__ __forceinline__ float flare_profile(const float* tab, int n, float u) {
  const float f = floorf(u);
  const int k = min(max(static_cast<int>(f) + 1, 0), n);
  return tab[k] + (tab[k + 1] - tab[k]) * (u - f);
}

// main.vert (colour), main.geom (screen-aligned quad of half-size flare * w in clip
// space), main.frag (flare alpha), additive blend.  A thread sets one particle up; then
// the warp draws its particles one after another, a lane per pair of pixels: the pairs
// of a row lie next to each other, so the reductions reach the L2 as whole sectors (a
// thread per particle sends every one on its own).
__global__ void __launch_bounds__(kSplatThreads) splat_kernel(
    const float* __restrict__ pos, const float4* __restrict__ vel, int64_t n_pad,
    RenderUniforms u, const float* __restrict__ flare, int per_warp, int copies,
    float2* __restrict__ hdr) {
  __shared__ float tab[kFlareMax + 2];
  const int n = u.flare_n;
  for (int k = threadIdx.x; k < n + 2; k += kSplatThreads)
    tab[k] = flare[(n / 2) * n + (k - 1 + n) % n];
  __syncthreads();
  hdr += static_cast<int64_t>(blockIdx.x % copies) * u.pitch * u.bh;
  const int lane = threadIdx.x & 31;
  // Texels per pixel along each axis: a sprite is flare_x * bw by flare_y * bh pixels.
  const float scale_x = n / (u.flare_x * u.bw), scale_y = n / (u.flare_y * u.bh);
  // Pixels are counted from the middle of the image, where most sprites are: there the last
  // bit of a coordinate is worth least.  (x + 1) / 2 bw - 1/2 = half x + rest + middle; the middle
  // column is even, as pairs of pixels start at even ones.
  const int mid_x = u.bw / 4 * 2, mid_y = u.bh / 2;
  const float half_x = 0.5f * u.bw, half_y = 0.5f * u.bh;
  const float rest_x = half_x - mid_x - 0.5f, rest_y = half_y - mid_y - 0.5f;
  hdr += static_cast<int64_t>(mid_y) * u.pitch + mid_x;
  constexpr int kWarps = kSplatThreads / 32;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * kWarps * per_warp;
  for (int64_t base = (static_cast<int64_t>(blockIdx.x) * kWarps + threadIdx.x / 32) * per_warp;
       base < n_pad; base += stride) {
    const int64_t g = base + lane;
    float sx = 0.f, sy = 0.f, t = 0.f;  // the quad's lower corner, the colour mix
    int kx0 = 0, kx1 = -1, ky0 = 0, ky1 = -1;
    if (lane < per_warp && g < n_pad) {
      const float px = pos[pair_index(g, 0)], py = pos[pair_index(g, 1)],
                  pz = pos[pair_index(g, 2)];
      const bool padding = pos[pair_index(g, 3)] == 0.f && px == kFarAway;
      const float* M = u.pv;  // p * mv, column-major
      const float cx = M[0] * px + M[4] * py + M[8] * pz + M[12];
      const float cy = M[1] * px + M[5] * py + M[9] * pz + M[13];
      const float cz = M[2] * px + M[6] * py + M[10] * pz + M[14];
      const float cw = M[3] * px + M[7] * py + M[11] * pz + M[15];
      const float xc = cx / cw, yc = cy / cw;
      const float x0 = xc - u.flare_x, x1 = xc + u.flare_x;
      const float y0 = yc - u.flare_y, y1 = yc + u.flare_y;
      if (!padding && cw > 0.f && !(cz < -cw || cz > cw) && x1 > -1.f && x0 < 1.f && y1 > -1.f &&
          y0 < 1.f) {
        // slow -> blue, fast -> purple; the velocity attribute carries w = 1 (renderer_gl.cpp:169)
        const float4 v = vel[g];
        t = fminf(fmaxf((v.x * v.x + v.y * v.y + v.z * v.z + 1.f) * 0.0006f, 0.f), 1.f);
        // pixel centres (k + 0.5) inside [x0, x1) in NDC
        kx0 = max(0, static_cast<int>(ceilf((x0 + 1.f) * 0.5f * u.bw - 0.5f))) - mid_x;
        kx1 = min(u.bw, static_cast<int>(ceilf((x1 + 1.f) * 0.5f * u.bw - 0.5f))) - 1 - mid_x;
        ky0 = max(0, static_cast<int>(ceilf((y0 + 1.f) * 0.5f * u.bh - 0.5f))) - mid_y;
        ky1 = min(u.bh, static_cast<int>(ceilf((y1 + 1.f) * 0.5f * u.bh - 0.5f))) - 1 - mid_y;
        sx = fmaf(xc, half_x, rest_x - u.flare_x * half_x);
        sy = fmaf(yc, half_y, rest_y - u.flare_y * half_y);
      }
    }
    unsigned todo = __ballot_sync(0xffffffffu, kx0 <= kx1 && ky0 <= ky1);
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1;
      const float qx = __shfl_sync(0xffffffffu, sx, src), qy = __shfl_sync(0xffffffffu, sy, src);
      const float qt = __shfl_sync(0xffffffffu, t, src);
      const int x_lo = __shfl_sync(0xffffffffu, kx0, src);
      const int x_hi = __shfl_sync(0xffffffffu, kx1, src);
      const int y_lo = __shfl_sync(0xffffffffu, ky0, src);
      const int y_hi = __shfl_sync(0xffffffffu, ky1, src);
      const int p0 = x_lo >> 1, np = (x_hi >> 1) - p0 + 1, rows = y_hi - y_lo + 1;
      if (np <= 8 && rows <= 16) {
        // The usual sprite: the lanes evaluate the profile once per column and row, and
        // are then 8 pairs of pixels by 4 rows.
        const int at = lane < 16 ? 2 * p0 + lane : y_lo + lane - 16;
        const bool in = lane < 16 ? at >= x_lo && at <= x_hi : at <= y_hi;
        const float w = flare_profile(
            tab, n, lane < 16 ? (at - qx) * scale_x - 0.5f : (at - qy) * scale_y - 0.5f);
        const float wi = in ? w : 0.f;
        const int p = lane & 7;
        const float a0 = __shfl_sync(0xffffffffu, wi, 2 * p);
        const float a1 = __shfl_sync(0xffffffffu, wi, 2 * p + 1);
        const float t0 = a0 * qt, t1 = a1 * qt;
        float2* to = hdr + static_cast<int64_t>(y_lo + (lane >> 3)) * u.pitch + 2 * (p0 + p);
        for (int r = 0; r < rows; r += 4, to += 4 * u.pitch) {
          const int row = r + (lane >> 3);
          const float wy = __shfl_sync(0xffffffffu, wi, 16 + min(row, 15));
          if (p < np && row < rows)
            atomicAdd(reinterpret_cast<float4*>(to),
                      make_float4(a0 * wy, t0 * wy, a1 * wy, t1 * wy));
        }
        continue;
      }
      const int total = np * rows;
      const float inv = 1.f / np;
      for (int k = lane; k < total; k += 32) {
        const int row = static_cast<int>((k + 0.5f) * inv);
        const int kx = 2 * (p0 + k - row * np), ky = y_lo + row;
        const float wy = flare_profile(tab, n, (ky - qy) * scale_y - 0.5f);
        const float ux = (kx - qx) * scale_x - 0.5f;
        const float a0 = kx >= x_lo ? wy * flare_profile(tab, n, ux) : 0.f;
        const float a1 = kx < x_hi ? wy * flare_profile(tab, n, ux + scale_x) : 0.f;
        atomicAdd(reinterpret_cast<float4*>(hdr + static_cast<int64_t>(ky) * u.pitch + kx),
                  make_float4(a0, a0 * qt, a1, a1 * qt));
      }
    }
  }
  pdl_trigger();
}

__device__ __forceinline__ float2 lerp2(float2 a, float2 b, float w) {
  return make_float2(a.x * (1.f - w) + b.x * w, a.y * (1.f - w) + b.y * w);
}

__device__ __forceinline__ void add2(float2& acc, float2 v, float w) {
  acc.x += v.x * w;
  acc.y += v.y * w;
}

// The copies of the HDR buffer into the first, two pixels per thread.
__global__ void __launch_bounds__(256) sum_copies_kernel(float4* __restrict__ hdr, int64_t count,
                                                         int copies) {
  pdl_wait();
  const int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  if (i < count) {
    float4 s = hdr[i];
#pragma unroll 4
    for (int c = 1; c < copies; ++c) {
      const float4 v = hdr[c * count + i];
      s.x += v.x, s.y += v.y, s.z += v.z, s.w += v.w;
    }
    hdr[i] = s;
  }
  pdl_trigger();
}

// Horizontal pass of the blur (blur.frag) into the half-size target, and luminance.frag
// (at half size: the pixel at (2x + 1, 2y + 1)) summed per CTA.  A CTA is kBlurX pixels of
// one target row; the two source rows it lies between are interpolated once, in shared
// memory, with the widest tap's reach on both sides.
constexpr int kBlurX = 256;

// Columns of a CTA's line (even).
__host__ __device__ constexpr int blur_cols(int reach) { return 2 * kBlurX + 2 * reach + 2; }

// A tap pair of the blur, for a pixel whose own taps start at place p of shared memory:
// the samples on both sides lie between places p + up, p + up + step and between p + down,
// p + down + step, mirrored.
struct TapPair {
  int up, down;
  float near, far;  // weights of the inner and the outer place
};

__device__ __forceinline__ void add_pair(float2& acc, const TapPair& t, float2 near0, float2 near1,
                                         float2 far0, float2 far1) {
  acc = __ffma2_rn(__fadd2_rn(near0, near1), make_float2(t.near, t.near), acc);
  acc = __ffma2_rn(__fadd2_rn(far0, far1), make_float2(t.far, t.far), acc);
}

// kEven: the source is exactly twice as wide, so a tap lies at the same place between
// two columns for every pixel: the CTA works its places and weights out once.  Two copies
// of the line, one shifted by a column, make any two neighbouring columns one 16-byte
// load.
template <bool kEven>
__global__ void __launch_bounds__(kBlurX) blur_x_kernel(const float2* __restrict__ hdr,
                                                        RenderUniforms u, int reach,
                                                        float2* __restrict__ dst,
                                                        double* __restrict__ block_sums) {
  extern __shared__ __align__(16) float2 line[];
  __shared__ double sh[kBlurX / 32];
  __shared__ TapPair taps[kRenderMaxTaps];
  // Source columns of the CTA: u of its first pixel minus the reach, and so on.
  const int c0 = 2 * static_cast<int>(blockIdx.x) * kBlurX - reach;
  const int cols = blur_cols(reach);
  if (kEven && threadIdx.x < u.taps) {
    const int i = threadIdx.x;
    const float at = 0.5f + u.offset[i] * u.size_x * u.bw;
    const int k = static_cast<int>(at);
    const float f = at - k;
    const int odd = (reach + k) & 1;
    taps[i] = TapPair{odd * (cols - 1) + reach + k, odd * (cols - 1) + reach - k,
                      u.weight[i] * (1.f - f), u.weight[i] * f};
  }
  pdl_wait();
  const int x = blockIdx.x * kBlurX + threadIdx.x, y = blockIdx.y;
  const float v = (y + 0.5f) / u.oh * u.bh - 0.5f;
  const float fv = floorf(v);
  const int y0 = min(max(static_cast<int>(fv), 0), u.bh - 1), y1 = min(y0 + 1, u.bh - 1);
  const float b = v - fv;
  // Not kEven: even and odd columns apart, as a warp's samples of one tap are two columns
  // apart.
  const int half = cols / 2;
  auto place = [half](int k) { return (k & 1) * half + (k >> 1); };
  const float2 *row0 = hdr + static_cast<int64_t>(y0) * u.pitch,
               *row1 = hdr + static_cast<int64_t>(y1) * u.pitch;
#pragma unroll 3
  for (int k = threadIdx.x; k < cols; k += kBlurX) {
    const int c = min(max(c0 + k, 0), u.bw - 1);
    const float2 l = lerp2(row0[c], row1[c], b);
    if (kEven) {
      line[k] = l;
      if (k > 0) line[cols + k - 1] = l;
    } else {
      line[place(k)] = l;
    }
  }
  __syncthreads();
  double lum = 0.0;
  if (x < u.ow) {
    const float s = (x + 0.5f) / u.ow;
    auto sample = [&](float at) {
      const float uu = at * u.bw - 0.5f;
      const float fu = floorf(uu);
      const int k = static_cast<int>(fu) - c0;
      return lerp2(line[place(k)], line[place(k + 1)], uu - fu);
    };
    float2 acc;
    if (kEven) {
      const float2* mine = line + 2 * threadIdx.x;  // the pixel lies between columns
      const float2 l = mine[reach], r = mine[reach + 1];  // reach and reach + 1
      const float w = 0.5f * u.weight[0];
      acc = make_float2((l.x + r.x) * w, (l.y + r.y) * w);
#pragma unroll 4
      for (int i = 1; i < u.taps; ++i) {
        const TapPair t = taps[i];
        const float4 p = *reinterpret_cast<const float4*>(mine + t.up);
        const float4 q = *reinterpret_cast<const float4*>(mine + t.down);
        add_pair(acc, t, make_float2(p.x, p.y), make_float2(q.z, q.w), make_float2(p.z, p.w),
                 make_float2(q.x, q.y));
      }
    } else {
      const float2 c = sample(s);
      acc = make_float2(c.x * u.weight[0], c.y * u.weight[0]);
#pragma unroll 4
      for (int i = 1; i < u.taps; ++i) {
        const float dx = u.offset[i] * u.size_x;
        const float2 p = sample(s + dx), q = sample(s - dx);
        add2(acc, make_float2(p.x + q.x, p.y + q.y), u.weight[i]);
      }
    }
    dst[static_cast<int64_t>(y) * u.ow + x] = acc;
    const float2 h = hdr[static_cast<int64_t>(2 * y + 1) * u.pitch + 2 * x + 1];
    const float3 rgb = light_rgb(h.x, h.y);
    lum = 0.2126f * rgb.x + 0.7152f * rgb.y + 0.0722f * rgb.z;
  }
  pdl_trigger();
  for (int w = 16; w > 0; w >>= 1) lum += __shfl_xor_sync(0xffffffffu, lum, w);
  if (threadIdx.x % 32 == 0) sh[threadIdx.x / 32] = lum;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kBlurX / 32; ++w) lum += sh[w];
    block_sums[static_cast<int64_t>(blockIdx.y) * gridDim.x + blockIdx.x] = lum;
  }
}

// Mean of the luminance sums: each thread adds a fixed stride of them, then a fixed tree
// (deterministic).
constexpr int kMeanThreads = 256;

__device__ void luminance_mean(const double* __restrict__ block_sums, int64_t count,
                               double inv_pixels, float* __restrict__ mean) {
  __shared__ double sh[kMeanThreads];
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  double s = 0.0;
  for (int64_t i = tid; i < count; i += kMeanThreads) s += block_sums[i];
  sh[tid] = s;
  __syncthreads();
  for (int w = kMeanThreads / 2; w > 0; w >>= 1) {
    if (tid < w) sh[tid] += sh[tid + w];
    __syncthreads();
  }
  if (tid == 0) *mean = static_cast<float>(sh[0] * inv_pixels);
}

// Vertical pass, at the target's own size: columns stay, rows are interpolated.  A CTA is
// 32 columns of kBlurRows rows, its source rows in shared memory; a thread has
// kBlurRows / 8 of them, so that a tap's places and weights are read once for all.  The
// grid's last row of CTAs takes the luminance's mean instead.
constexpr int kBlurRows = 32;

__global__ void __launch_bounds__(kMeanThreads) blur_y_kernel(
    const float2* __restrict__ src, RenderUniforms u, int reach,
    const double* __restrict__ block_sums, int64_t parts, float* __restrict__ mean,
    float2* __restrict__ dst) {
  extern __shared__ __align__(16) float2 tile[];
  __shared__ TapPair taps[kRenderMaxTaps];
  const int tid = threadIdx.y * 32 + threadIdx.x;
  if (tid < u.taps) {
    const float at = u.offset[tid] * u.size_y * u.oh;
    const int k = static_cast<int>(at);
    const float f = at - k;
    taps[tid] = TapPair{(reach + k) * 32, (reach - k) * 32, u.weight[tid] * (1.f - f),
                        u.weight[tid] * f};
  }
  pdl_wait();
  pdl_trigger();
  if (blockIdx.y + 1 == gridDim.y) {
    if (blockIdx.x == 0)
      luminance_mean(block_sums, parts, 1.0 / (static_cast<double>(u.lw) * u.lh), mean);
    return;
  }
  const int x = blockIdx.x * 32 + threadIdx.x, xc = min(x, u.ow - 1);
  const int top = blockIdx.y * kBlurRows - reach;  // row of the tile's first
#pragma unroll 4
  for (int k = threadIdx.y; k < kBlurRows + 2 * reach; k += 8)
    tile[k * 32 + threadIdx.x] =
        src[static_cast<int64_t>(min(max(top + k, 0), u.oh - 1)) * u.ow + xc];
  __syncthreads();
  constexpr int kMine = kBlurRows / 8;
  const float2* mine = tile + tid;  // row r of the thread: 8 r rows further down
  float2 acc[kMine];
#pragma unroll
  for (int r = 0; r < kMine; ++r) {
    const float2 c = mine[(reach + 8 * r) * 32];
    acc[r] = make_float2(c.x * u.weight[0], c.y * u.weight[0]);
  }
  for (int i = 1; i < u.taps; ++i) {
    const TapPair t = taps[i];
    const float2 *up = mine + t.up, *down = mine + t.down;
#pragma unroll
    for (int r = 0; r < kMine; ++r)
      add_pair(acc[r], t, up[r * 256], down[r * 256], up[r * 256 + 32], down[r * 256 - 32]);
  }
#pragma unroll
  for (int r = 0; r < kMine; ++r) {
    const int y = blockIdx.y * kBlurRows + threadIdx.y + 8 * r;
    if (x < u.ow && y < u.oh) dst[static_cast<int64_t>(y) * u.ow + x] = acc[r];
  }
}

// r^(1/2.2) = r^(5/11) for r in [0, 1], where r is 0 or at least 2^-24 (one minus a
// float): the hardware's logarithm and power of two, then one Newton step for y^11 = r^5,
// whose rounding errors the step divides by 11.  Over every such r within 1.2 ulp
// of the power in 64 bits; powf(r, 1.f / 2.2f) is within 4.1, and took most of the 375
// instructions per pixel of the tonemap.
__device__ __forceinline__ float gamma_22(float r) {
  r *= 2048.f;  // scales the result by 32: all powers below are normal numbers
  const float y = exp2f(__log2f(r) * (5.f / 11.f));
  const float r2 = r * r, r5 = r2 * r2 * r;
  const float y2 = y * y, y4 = y2 * y2, y8 = y4 * y4;
  const float z = __fdividef(fmaf(-y8 * y2, y, r5), r5) * (1.f / 11.f);
  return r == 0.f ? 0.f : fmaf(y, z, y) * (1.f / 32.f);
}

// tonemap.frag: HDR + bloom, exposure from the mean luminance, gamma 2.2.  Bound by
// instructions, of which a thread shares the exposure and the columns' places over its
// kToneRows rows.
constexpr int kToneRows = 4;

__global__ void __launch_bounds__(256) tonemap_kernel(const float2* __restrict__ hdr,
                                                      const float2* __restrict__ bloom,
                                                      const float* __restrict__ mean,
                                                      RenderUniforms u, float4* __restrict__ out) {
  const int x = blockIdx.x * 32 + threadIdx.x;
  const int y0 = blockIdx.y * 8 * kToneRows + threadIdx.y;
  if (x >= u.width) return;
  const int cx = x + u.margin;
  const float uu = static_cast<float>(cx) / u.bw * u.ow - 0.5f;
  const float per_row = static_cast<float>(u.oh) / u.bh;
  const float fu = floorf(uu), wu = uu - fu;
  const int x0 = min(max(static_cast<int>(fu), 0), u.ow - 1), x1 = min(x0 + 1, u.ow - 1);
  pdl_wait();
  const float exposure = 1.f / fminf(fmaxf(*mean * 10.f, 0.2f), 1000.f);
#pragma unroll
  for (int k = 0; k < kToneRows; ++k) {
    const int y = y0 + 8 * k;
    if (y >= u.height) return;
    const int cy = y + u.margin;
    const float2 c = hdr[static_cast<int64_t>(cy) * u.pitch + cx];
    const float vv = cy * per_row - 0.5f;
    const float fv = floorf(vv);
    const int r0 = min(max(static_cast<int>(fv), 0), u.oh - 1), r1 = min(r0 + 1, u.oh - 1);
    const float2 *b0 = bloom + static_cast<int64_t>(r0) * u.ow,
                 *b1 = bloom + static_cast<int64_t>(r1) * u.ow;
    const float2 b = lerp2(lerp2(b0[x0], b0[x1], wu), lerp2(b1[x0], b1[x1], wu), vv - fv);
    const float3 l = light_rgb(c.x + b.x, c.y + b.y);
    out[static_cast<int64_t>(y) * u.width + x] =
        make_float4(gamma_22(1.f - expf(-l.x * exposure)), gamma_22(1.f - expf(-l.y * exposure)),
                    gamma_22(1.f - expf(-l.z * exposure)), 1.f);
  }
}

// Source columns between a target pixel's centre and its widest tap, rounded up.
int blur_reach(const RenderUniforms& u) {
  return static_cast<int>(u.offset[u.taps - 1] * u.size_x * u.bw) + 3;
}

// Rows between a pixel and its widest tap, rounded up.
int blur_y_reach(const RenderUniforms& u) {
  return static_cast<int>(u.offset[u.taps - 1] * u.size_y * u.oh) + 2;
}

// Images lower than about 60 rows: taps so far apart that the rows need more shared memory
// than a kernel has by default, 48 KB with its static arrays (94 KB at 16 rows, the lowest
// image).  The limit belongs to the kernel on the device, not to a simulation: it is
// raised once and never lowered, as another thread may be about to launch a lower image.
constexpr int kBlurMaxSmem = 112 * 1024;

cudaError_t blur_y_opt_in() {
  static std::atomic<uint64_t> opted{0};  // once per device ordinal (>= 64: every call)
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = dev >= 0 && dev < 64 ? uint64_t{1} << dev : 0;
  if (bit != 0 && (opted.load(std::memory_order_acquire) & bit) != 0) return cudaSuccess;
  e = cudaFuncSetAttribute(blur_y_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kBlurMaxSmem);
  if (e == cudaSuccess && bit != 0) opted.fetch_or(bit, std::memory_order_release);
  return e;
}

}  // namespace

int64_t render_luminance_parts(const RenderUniforms& u) {
  return static_cast<int64_t>((u.ow + kBlurX - 1) / kBlurX) * u.oh;
}

// Many particles on a small image: the reductions queue up at the same sectors, so CTAs add
// to one of several copies of the buffer, and a pass adds the copies up.  1,048,576
// particles (us per frame with 1, 4, 16 and 32 copies): 381, 263, 226, 221 at 320 x 180
// (8.9 particles per pixel), 229, 185, 177, 189 at 640 x 360 (3.1), 181, 172, 208, 295 at
// 1281 x 720 (0.93), 181, 195, 315, 482 at 1920 x 1080 (0.44); 50,000 at 640 x 360 (0.15)
// 35, 35, 41, 54.
int render_copies(const RenderUniforms& u, int64_t n) {
  const double most = 4.4 * static_cast<double>(n) / (static_cast<double>(u.pitch) * u.bh);
  int copies = 1;
  while (copies < 32 && 2 * copies <= most) copies *= 2;
  return copies;
}

cudaError_t launch_render(const float* pos, const float4* vel, int64_t n_pad,
                          const RenderUniforms& u, const RenderBuffers& b, float4* out,
                          cudaStream_t stream) {
  const size_t pixels = static_cast<size_t>(u.pitch) * u.bh;
  cudaError_t e = cudaMemsetAsync(b.hdr, 0, sizeof(float2) * pixels * b.copies, stream);
  if (e != cudaSuccess) return e;
  // A warp draws its particles one after another: fewer of them where there are too few
  // for every warp the GPU holds (1,000 particles, 32 per warp: 22 us for the splat alone,
  // of 101 per frame; 67 per frame now).
  int per_warp = 32;
  while (per_warp > 4 && n_pad / per_warp < 8192) per_warp /= 2;
  const int64_t per_block = static_cast<int64_t>(per_warp) * (kSplatThreads / 32);
  const int64_t blocks = (n_pad + per_block - 1) / per_block;
  splat_kernel<<<static_cast<unsigned>(blocks < 8192 ? blocks : 8192), kSplatThreads, 0, stream>>>(
      pos, vel, n_pad, u, b.flare, per_warp, b.copies, b.hdr);
  const int reach = blur_reach(u);
  const dim3 gx((u.ow + kBlurX - 1) / kBlurX, u.oh);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if (b.copies > 1) {
    const int64_t count = static_cast<int64_t>(pixels / 2);
    e = launch_dependent(sum_copies_kernel, dim3(static_cast<unsigned>((count + 255) / 256)),
                         dim3(256), 0, stream, reinterpret_cast<float4*>(b.hdr), count, b.copies);
    if (e != cudaSuccess) return e;
  }
  const bool even = u.bw == 2 * u.ow;
  e = launch_dependent(even ? blur_x_kernel<true> : blur_x_kernel<false>, gx, dim3(kBlurX),
                       sizeof(float2) * blur_cols(reach) * (even ? 2 : 1), stream, b.hdr, u, reach,
                       b.blur1, b.block_sums);
  if (e != cudaSuccess) return e;
  const dim3 blk(32, 8);
  const int reach_y = blur_y_reach(u);
  const int smem_y = static_cast<int>(sizeof(float2)) * 32 * (kBlurRows + 2 * reach_y);
  if (smem_y > 40 * 1024 && (e = blur_y_opt_in()) != cudaSuccess) return e;
  const dim3 gy((u.ow + 31) / 32, (u.oh + kBlurRows - 1) / kBlurRows + 1);
  e = launch_dependent(blur_y_kernel, gy, blk, smem_y, stream, b.blur1, u, reach_y, b.block_sums,
                       render_luminance_parts(u), b.mean, b.blur2);
  if (e != cudaSuccess) return e;
  constexpr int kRows = 8 * kToneRows;
  return launch_dependent(tonemap_kernel,
                          dim3((u.width + 31) / 32, (u.height + kRows - 1) / kRows), blk, 0, stream,
                          b.hdr, b.blur2, b.mean, u, out);
}

}  // namespace nbg
