// Force step of small systems: one launch, no work list of blocks, no scratch.
//
// A CTA takes R i-particles against every particle of their system: each thread holds
// all R (in packed pairs) and meets its share of the j-particles, two at a time as they
// lie in memory; the threads' sums are added in a fixed tree and R threads integrate.
//
// What bounds it: below 1,000 particles the launch and one chain of latencies (positions,
// pairs, tree, state: 1.7 us per step); above, the pairs, 11 lane operations each where
// the symmetric kernel has 14 for two, and the last wave of CTAs (2,048 particles: 256 CTAs on
// 152 SMs; 1.2 us of pairs in 4.2).
#include <cuda_runtime.h>

#include "direct.cuh"
#include "nb_device.cuh"
#include "nb_kernels.hpp"

namespace nbg {
namespace {

// Loads of a thread between two foldings of its sums (two j-particles each): its chains are
// no longer than the tuned kernel's.
constexpr int kDirectChunk = 64;

template <bool kComp>
struct DirectSum {
  float s = 0.f, c = 0.f;  // s - c is the sum
  __device__ __forceinline__ void add(float t) {
    if (kComp) {
      const float y = t - c, u = s + y;
      c = (u - s) - y;
      s = u;
    } else {
      s += t;
    }
  }
};

// One j-particle (x, y, z, m) against the thread's i-particles.  kMask: leave out j == i
// by index, d = j - (first i).
template <int P, bool kMass, bool kMask>
__device__ __forceinline__ void direct_meet(const float2 (&nx)[P], const float2 (&ny)[P],
                                            const float2 (&nz)[P], float2 (&ax)[P],
                                            float2 (&ay)[P], float2 (&az)[P], float x, float y,
                                            float z, float m, float2 e2, int d) {
  const float2 xx = make_float2(x, x), yy = make_float2(y, y), zz = make_float2(z, z);
#pragma unroll
  for (int p = 0; p < P; ++p) {
    const float2 dx = __fadd2_rn(xx, nx[p]);
    const float2 dy = __fadd2_rn(yy, ny[p]);
    const float2 dz = __fadd2_rn(zz, nz[p]);
    float2 d2 = __ffma2_rn(dx, dx, e2);
    d2 = __ffma2_rn(dy, dy, d2);
    d2 = __ffma2_rn(dz, dz, d2);
    float2 t = __fmul2_rn(d2, d2);
    t = __fmul2_rn(t, d2);
    float2 s = make_float2(rsqrtf(t.x), rsqrtf(t.y));
    if (kMask) {
      if (d == 2 * p) s.x = 0.f;
      if (d == 2 * p + 1) s.y = 0.f;
    }
    if (kMass) s = __fmul2_rn(s, make_float2(m, m));
    ax[p] = __ffma2_rn(dx, s, ax[p]);
    ay[p] = __ffma2_rn(dy, s, ay[p]);
    az[p] = __ffma2_rn(dz, s, az[p]);
  }
}

// W warps per CTA, B CTAs per SM.  kXyzm: positions are a float4 (x, y, z, m) per particle, and no
// padding follows them.
template <int W, int R, int B, bool kComp, bool kMass, bool kXyzm>
__global__ void __launch_bounds__(W * 32, B) direct_kernel(const DirectArgs a) {
  constexpr int P = R / 2;
  static_assert(R == 4 || R == 8 || R == 16, "a power of two that divides kPadQuantum");
  __shared__ float part[kComp ? 6 : 3][W][R];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  int sys = a.sys, itile = blockIdx.x;
  if (a.tiles != nullptr) {
    const int2 t = a.tiles[blockIdx.x];
    sys = t.x, itile = t.y;
  }
  SystemDesc sd{};
  if (kXyzm) {
    sd.n = a.n, sd.gscale = a.gscale;
  } else {
    sd = a.f.sys[sys];
  }
  const int n = sd.n, i0 = itile * R;
  const float4* pos = reinterpret_cast<const float4*>(a.f.pos) + sd.offset;
  pdl_wait();

  // The finishing threads' state.
  const int64_t g = sd.offset + i0 + tid;
  const bool mine = tid < R && i0 + tid < n;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  float xi = 0.f, yi = 0.f, zi = 0.f;
  if (!kXyzm && mine && a.f.accel_out == nullptr) {
    v = a.f.vel[g];
    xi = a.f.pos[pair_index(g, 0)];
    yi = a.f.pos[pair_index(g, 1)];
    zi = a.f.pos[pair_index(g, 2)];
  }

  float2 nx[P], ny[P], nz[P];
#pragma unroll
  for (int p = 0; p < P; ++p) {
    const int i = i0 + 2 * p;
    float4 u = make_float4(-kFarAway, -kFarAway, -kFarAway, 0.f), q = u;
    if (kXyzm) {
      if (i < n) u = pos[i];
      if (i + 1 < n) q = pos[i + 1];
      nx[p] = make_float2(-u.x, -q.x);
      ny[p] = make_float2(-u.y, -q.y);
      nz[p] = make_float2(-u.z, -q.z);
    } else {  // R divides the padding
      u = pos[i], q = pos[i + 1];
      nx[p] = make_float2(-u.x, -u.y);
      ny[p] = make_float2(-u.z, -u.w);
      nz[p] = make_float2(-q.x, -q.y);
    }
  }
  const float2 e2 = make_float2(a.f.eps2, a.f.eps2);

  // A record is two j-particles.  Its two float4: (x0 x1 y0 y1), (z0 z1 m0 m1), or
  // (x0 y0 z0 m0), (x1 y1 z1 m1).
  const int nrec = kXyzm ? (n + 1) / 2 : ((n + kPadQuantum - 1) & -kPadQuantum) / 2;
  constexpr int kStride = W * 32;
  float4 b0, b1;
  auto fetch = [&](int rec) {
    if (kXyzm) {
      const float4 far = make_float4(kFarAway, kFarAway, kFarAway, 0.f);
      b0 = 2 * rec < n ? pos[2 * rec] : far;
      b1 = 2 * rec + 1 < n ? pos[2 * rec + 1] : far;
    } else {
      const bool in = rec < nrec;
      b0 = in ? pos[2 * rec] : make_float4(kFarAway, kFarAway, kFarAway, kFarAway);
      b1 = in ? pos[2 * rec + 1] : make_float4(kFarAway, kFarAway, 0.f, 0.f);
    }
  };
  fetch(tid);
  DirectSum<kComp> sum[3];
  for (int base = 0; base < nrec; base += kStride * kDirectChunk) {
    float2 ax[P], ay[P], az[P];
#pragma unroll
    for (int p = 0; p < P; ++p) ax[p] = ay[p] = az[p] = make_float2(0.f, 0.f);
    const int end = min(nrec, base + kStride * kDirectChunk);
#pragma unroll 1
    for (int r = base; r < end; r += kStride) {
      const float4 c0 = b0, c1 = b1;
      const int d = 2 * (r + tid) - i0;
      if (r + kStride < nrec) fetch(r + kStride + tid);
      const float x0 = c0.x, x1 = kXyzm ? c1.x : c0.y, y0 = kXyzm ? c0.y : c0.z,
                  y1 = kXyzm ? c1.y : c0.w, z0 = kXyzm ? c0.z : c1.x,
                  z1 = kXyzm ? c1.z : c1.y, m0 = kXyzm ? c0.w : c1.z, m1 = c1.w;
      if (a.f.mask_self) {
        direct_meet<P, kMass, true>(nx, ny, nz, ax, ay, az, x0, y0, z0, m0, e2, d);
        direct_meet<P, kMass, true>(nx, ny, nz, ax, ay, az, x1, y1, z1, m1, e2, d + 1);
      } else {
        direct_meet<P, kMass, false>(nx, ny, nz, ax, ay, az, x0, y0, z0, m0, e2, 0);
        direct_meet<P, kMass, false>(nx, ny, nz, ax, ay, az, x1, y1, z1, m1, e2, 0);
      }
    }
    float t[R][3];
#pragma unroll
    for (int p = 0; p < P; ++p) {
      t[2 * p][0] = ax[p].x, t[2 * p][1] = ay[p].x, t[2 * p][2] = az[p].x;
      t[2 * p + 1][0] = ax[p].y, t[2 * p + 1][1] = ay[p].y, t[2 * p + 1][2] = az[p].y;
    }
    warp_sums<R>(t);
#pragma unroll
    for (int c = 0; c < 3; ++c) sum[c].add(t[0][c]);
  }
  pdl_trigger();
  if (lane % (32 / R) == 0)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      part[c][w][lane / (32 / R)] = sum[c].s;
      if (kComp) part[3 + c][w][lane / (32 / R)] = sum[c].c;
    }
  if (W > 1)
    __syncthreads();
  else
    __syncwarp();
  if (!mine) return;
  float f[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    DirectSum<kComp> all;
    float low = 0.f;
#pragma unroll
    for (int k = 0; k < W; ++k) {
      all.add(part[c][k][tid]);
      if (kComp) low += part[3 + c][k][tid];
    }
    f[c] = kComp ? all.s - (all.c + low) : all.s;
  }
  if (kXyzm) {
    a.f.accel_out[g] = make_float4(f[0] * sd.gscale, f[1] * sd.gscale, f[2] * sd.gscale, 0.f);
  } else {
    finish_particle(a.f, sd, g, f[0], f[1], f[2], xi, yi, zi, v);
  }
}

struct DirectEntry {
  int warps, r;
  void (*kernel[2][2])(DirectArgs);  // [compensated][mass]
  void (*xyzm)(DirectArgs);          // plain, own masses
};

#define NBG_DIRECT(W, R, B)                                                                 \
  {W, R,                                                                                    \
   {{direct_kernel<W, R, B, false, false, false>, direct_kernel<W, R, B, false, true, false>}, \
    {direct_kernel<W, R, B, true, false, false>, direct_kernel<W, R, B, true, true, false>}},  \
   direct_kernel<W, R, B, false, true, true>}

const DirectEntry kShapes[] = {NBG_DIRECT(8, 8, 2), NBG_DIRECT(4, 4, 7), NBG_DIRECT(4, 8, 5),
                               NBG_DIRECT(2, 8, 10), NBG_DIRECT(1, 8, 20)};

}  // namespace

int num_direct_shapes() { return static_cast<int>(sizeof(kShapes) / sizeof(kShapes[0])); }

KernelShape direct_shape(int index) {
  const DirectEntry& e = kShapes[index];
  return KernelShape{e.warps * 32, e.r, e.warps * 64, 1};
}

// Against the symmetric kernel (its two launches take 3.8 us for 64 particles, and it needs
// thousands of particles to have a block for every warp): single systems (us per step,
// symmetric / direct) 64 3.8 / 1.7, 512 5.6 / 2.0, 2,048 7.4 / 4.2, 4,096 12.2 / 9.8, 4,500
// 12.8 / 11.7, 5,000 14.1 / 15.0; ensembles, from all pairs and i-tiles of 8 particles:
// 2.4e6 pairs in 1,091 tiles 7.8 / 4.5, 7e6 in 1,720 9.5 / 8.2, 1.1e7 in 1,270 11.9 / 9.4
// and in 4,760 11.2 / 11.3, 1.4e7 in 11,407 12.8 / 14.8, 2.2e7 in 2,792 14.7 / 16.9, 3.6e6
// in 4,830 7.8 / 7.1, 5.7e6 in 7,692 9.4 / 10.0.
//
// The shapes in the order of their warps: as many per i-tile as one wave of CTAs allows,
// and their passes over the longest system are worth (a warp meets 64 particles a pass).
// us per step with 8 x 8, 4 x 4, 4 x 8, 2 x 8, 1 x 8 warps x particles: one system of 256
// 2.0 1.7 1.7 1.9 2.9; 2,048 4.2 4.8 5.5 8.7 15.3; 4,096 10.5 9.8 10.6 16.6 29.7; 40
// systems up to 512 8.3 5.4 5.4 4.5 6.1, 16 up to 2,048 12.4 9.7 9.5 10.3 15.8, 100 up to
// 512 19.5 12.1 10.4 8.4 7.7.
int choose_direct(const SystemDesc* sys, int32_t count, int sms, double max_pairs,
                  int64_t max_tiles, bool* pays) {
  double pairs = 0;
  int64_t t4 = 0, t8 = 0;
  int32_t longest = 0;
  for (int32_t k = 0; k < count; ++k) {
    pairs += static_cast<double>(sys[k].n) * sys[k].n;
    t4 += (sys[k].n + 3) / 4;
    t8 += (sys[k].n + 7) / 8;
    longest = sys[k].n > longest ? sys[k].n : longest;
  }
  *pays = pairs <= max_pairs && t8 <= max_tiles;
  if (t8 <= 2 * sms && longest >= 512) return 0;
  if (t4 <= 7 * sms) return 1;
  if (t8 <= 5 * sms || longest > 1024) return 2;
  if (t8 <= 10 * sms || longest > 512) return 3;
  return 4;
}

cudaError_t launch_direct(int index, bool compensated, bool per_pair_mass, const DirectArgs& a,
                          int grid, cudaStream_t stream) {
  const DirectEntry& e = kShapes[index];
  return launch_dependent(e.kernel[compensated][per_pair_mass], dim3(grid), dim3(e.warps * 32), 0,
                          stream, a);
}

cudaError_t launch_direct_xyzm(int index, const DirectArgs& a, int grid, cudaStream_t stream) {
  const DirectEntry& e = kShapes[index];
  return launch_dependent(e.xyzm, dim3(grid), dim3(e.warps * 32), 0, stream, a);
}

}  // namespace nbg
