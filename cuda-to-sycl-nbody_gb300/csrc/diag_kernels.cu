// FP64 diagnostics on the GPU: kinetic and potential energy, linear and angular
// momentum, and FP64 accelerations of selected rows.  Sums are double precision, and
// so is the pair arithmetic, except the potential's of large systems, whose terms are
// sums of three floats; reductions use fixed-order trees over per-block partials, so
// results are deterministic.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <vector>

#include "nb_internal.hpp"
#include "nb_kernels.hpp"

namespace nbg {
namespace {

constexpr int kDiagThreads = 256;
constexpr int kDiagVals = 10;  // KE PE px py pz Lx Ly Lz M (unused)

__device__ __forceinline__ double block_sum(double v, double* sh) {
  // Fixed-order tree over the block.
  const int t = threadIdx.x;
  sh[t] = v;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (t < w) sh[t] += sh[t + w];
    __syncthreads();
  }
  const double r = sh[0];
  __syncthreads();
  return r;
}

// Whether a value lies where the split potential below neither overflows nor loses low
// words to underflow (NaN does not).
__device__ __forceinline__ bool splittable(float x, float y, float z, float m) {
  return fabsf(x) <= 1e6f && fabsf(y) <= 1e6f && fabsf(z) <= 1e6f &&
         (m == 0.f || (fabsf(m) >= 1e-12f && fabsf(m) <= 1e12f));
}

// Per-particle moments over the padded range [first, last): padding has zero
// mass and velocity, so it contributes nothing.  Sets *wide where a particle is not
// splittable.
__global__ void __launch_bounds__(kDiagThreads) moments_kernel(
    const float* __restrict__ pos, const float4* __restrict__ vel, int64_t first, int64_t last,
    double* __restrict__ partial, int* __restrict__ wide) {
  __shared__ double sh[kDiagThreads];
  double acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  bool far = false;
  for (int64_t g = first + blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; g < last;
       g += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float xf = pos[pair_index(g, 0)], yf = pos[pair_index(g, 1)], zf = pos[pair_index(g, 2)];
    const float mf = pos[pair_index(g, 3)];
    if (xf == kFarAway && mf == 0.f) continue;  // padding
    far = far || !splittable(xf, yf, zf, mf);
    const double m = mf;
    if (m == 0.0) continue;
    const double x = xf, y = yf, z = zf;
    const float4 v = vel[g];
    const double vx = v.x, vy = v.y, vz = v.z;
    acc[0] += 0.5 * m * (vx * vx + vy * vy + vz * vz);
    acc[2] += m * vx;
    acc[3] += m * vy;
    acc[4] += m * vz;
    acc[5] += m * (y * vz - z * vy);
    acc[6] += m * (z * vx - x * vz);
    acc[7] += m * (x * vy - y * vx);
    acc[8] += m;
  }
  if (far) atomicOr(wide, 1);
  for (int k = 0; k < 9; ++k) {
    const double s = block_sum(acc[k], sh);
    if (threadIdx.x == 0) partial[blockIdx.x * kDiagVals + k] = s;
  }
}

// ---- potential, pairs in three floats -----------------------------------------------
// The potential needs N^2 / 2 inverse square roots in double precision, about 30 FP64
// operations per pair on a pipe of 2 lanes per SM (FP32: 128; a third-order step from the
// FP32 root is no faster than rsqrt: its conversions run on that pipe too).  Here a pair's
// term is a sum of three floats (packed FP32x2, two j-particles per register pair).  The
// coordinate differences and their squares are exact (TwoSum, fused multiply-add); every
// sum is carried with its errors, so that the squared distance, the root's residual and
// the term keep more than 60 bits, and 128 terms at a time are added error-free before
// they go to FP64.  A term is then no further from exact than FP64's (over 8e6 pairs,
// emulated: 5e-19 at worst, FP64's 2.8e-16, 7e-17 RMS), whatever the distances are: where
// few distinct ones dominate nothing averages out, and terms of two floats (7.6 ms at N =
// 65,536) left errors up to 3.8e-13 of the sum (4,096 particles at two points).
// About 160 FP32 lane operations per pair, of which the FMA pipe takes 8.7 ms at N = 65,536:
// 103.5 ms with FP64 pairs, 9.6 now.
// Systems below kSplitMin particles, softenings below kSplitEps and values out of the
// split's range keep the FP64 kernel.
constexpr int kSplitMin = 4096;  // below, FP64's sums are the more exact ones
constexpr float kSplitEps = 1e-12f;
constexpr int kSplitThreads = 256;
constexpr int kSplitBI = kSplitThreads;  // i-tile (a particle per thread) and j-tile
constexpr int kSplitFlush = 64;          // j-pairs between two sums into FP64

__device__ __forceinline__ float2 both(float a) { return make_float2(a, a); }
// Signs as products: the packed operations take no negated operand, and a sign flip per lane
// costs more (9.6 ms; as flips and additions 13.7).
__device__ __forceinline__ float2 neg2(float2 a) { return __fmul2_rn(a, both(-1.f)); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, both(-1.f), a); }

// a + b = s + e exactly (Knuth's TwoSum).
__device__ __forceinline__ float2 two_sum(float2 a, float2 b, float2& e) {
  const float2 s = __fadd2_rn(a, b);
  const float2 t = sub2(s, a);
  e = __fadd2_rn(sub2(a, sub2(s, t)), sub2(b, t));
  return s;
}

// a * b = p + e exactly.
__device__ __forceinline__ float2 two_prod(float2 a, float2 b, float2& e) {
  const float2 p = __fmul2_rn(a, b);
  e = __ffma2_rn(a, b, neg2(p));
  return p;
}

// sum += t, for |t| < |sum| (Dekker's FastTwoSum): what is rounded away goes to low.  A sum
// that starts at a value well above all terms stays in its binade, so their high parts add
// without error and `sum` less that value is their sum.
__device__ __forceinline__ void add_low(float2& sum, float2& low, float2 t) {
  const float2 s = __fadd2_rn(sum, t);
  low = __fadd2_rn(low, sub2(t, sub2(s, sum)));
  sum = s;
}

// One squared difference: a - b = h + l exactly, its square p + q + r + what goes to low.
__device__ __forceinline__ float2 square_diff(float2 a, float2 nb, float2& q, float2& r,
                                              float2& low) {
  float2 l, s;
  const float2 h = two_sum(a, nb, l);
  const float2 p = two_prod(h, h, q);
  r = two_prod(__fadd2_rn(h, h), l, s);
  low = __ffma2_rn(l, l, __fadd2_rn(low, s));
  return p;
}

// The inverse square root of D = dx^2 + dy^2 + dz^2 + e2 as y + w + v.
__device__ __forceinline__ float2 split_root(float2 ax, float2 nx, float2 ay, float2 ny, float2 az,
                                             float2 nz, float2 e2, float2& w, float2& v) {
  // D = H + L + T, each below 2^-22 of the one before: the squares, then what their sum
  // and their own low parts leave (below 6 2^-24 D in all, so 2^-20 D holds them).
  float2 T = both(0.f), a, b, c, qx, qy, qz, rx, ry, rz;
  const float2 px = square_diff(ax, nx, qx, rx, T);
  const float2 py = square_diff(ay, ny, qy, ry, T);
  const float2 pz = square_diff(az, nz, qz, rz, T);
  const float2 h = two_sum(two_sum(two_sum(px, py, a), pz, b), e2, c);
  const float2 base = __fmul2_rn(h, both(0x1p-20f));
  float2 mid = base;
  add_low(mid, T, a);
  add_low(mid, T, b);
  add_low(mid, T, c);
  add_low(mid, T, qx);
  add_low(mid, T, qy);
  add_low(mid, T, qz);
  add_low(mid, T, rx);
  add_low(mid, T, ry);
  add_low(mid, T, rz);
  mid = sub2(mid, base);
  const float2 H = __fadd2_rn(h, mid);
  const float2 L = sub2(mid, sub2(H, h));
  // y is within 2^-22 of the root; e = 1 - D y^2 as E + F, from y^2 = s + t.
  const float2 y = make_float2(rsqrtf(H.x), rsqrtf(H.y));
  float2 t, pe, ce, de;
  const float2 s = two_prod(y, y, t);
  const float2 p = two_prod(H, s, pe), cp = two_prod(H, t, ce), dp = two_prod(L, s, de);
  float2 F = neg2(__ffma2_rn(T, s, __ffma2_rn(L, t, __fadd2_rn(ce, de))));
  const float2 scale = both(0x1.8p-20f);
  float2 E = __fadd2_rn(sub2(both(1.f), p), scale);
  add_low(E, F, neg2(pe));
  add_low(E, F, neg2(cp));
  add_low(E, F, neg2(dp));
  E = sub2(E, scale);
  // y (1 - e)^(-1/2) = y + y e / 2 + y 3/8 e^2, the next term below 2^-64.
  const float2 half = __fmul2_rn(y, both(0.5f));
  w = two_prod(half, E, v);
  v = __ffma2_rn(half, __ffma2_rn(__fmul2_rn(E, both(0.75f)), E, F), v);
  return y;
}

// j-pairs [p0, p1) of the shared tile against the thread's i-particle, added to s + l + k.
// kMask: leave out j == self and j >= cnt.
template <bool kMass, bool kMask>
__device__ __forceinline__ void split_pairs(const float4* tile, int p0, int p1, int cnt, float2 nx,
                                            float2 ny, float2 nz, float2 e2, int self, float2& s,
                                            float2& l, float2& k) {
#pragma unroll 2
  for (int p = p0; p < p1; ++p) {
    const float4 A = tile[2 * p], B = tile[2 * p + 1];
    float2 w, v, u, t;
    float2 y = split_root(make_float2(A.x, A.y), nx, make_float2(A.z, A.w), ny,
                          make_float2(B.x, B.y), nz, e2, w, v);
    float2 low = both(0.f);
    if (kMass) {
      const float2 m = make_float2(B.z, B.w);
      y = two_prod(m, y, low);
      w = two_prod(m, w, u);
      v = __ffma2_rn(m, v, u);
    }
    if (kMask) {
      if (2 * p == self || 2 * p >= cnt) y.x = w.x = v.x = low.x = 0.f;
      if (2 * p + 1 == self || 2 * p + 1 >= cnt) y.y = w.y = v.y = low.y = 0.f;
    }
    s = two_sum(s, y, t);
    l = two_sum(l, t, u);
    k = __fadd2_rn(k, __fadd2_rn(u, v));
    l = two_sum(l, w, u);
    k = __fadd2_rn(k, u);
    if (kMass) {
      l = two_sum(l, low, u);
      k = __fadd2_rn(k, u);
    }
  }
}

// blockIdx.x: i-tile tiles[x] = (system, tile); blockIdx.y: one of gridDim.y spans of the
// j-tiles from it to the end of the system.  Each pair of different tiles is met once;
// the i-tile itself over all ordered pairs, at half weight.  Writes its part of
// -G sum_i m_i sum_j m_j / sqrt(r^2 + eps), zero where the FP64 kernel does the system.
template <bool kMass>
__global__ void __launch_bounds__(kSplitThreads) potential_split_kernel(
    const float* __restrict__ pos, const SystemDesc* __restrict__ sys,
    const int2* __restrict__ tiles, const int* __restrict__ wide, float eps2, double G,
    double* __restrict__ partial) {
  __shared__ __align__(16) float4 tile[kSplitBI];
  __shared__ double sh[kSplitThreads];
  const int2 tl = tiles[blockIdx.x];
  const SystemDesc sd = sys[tl.x];
  const int tid = threadIdx.x;
  const int njt = (sd.n + kSplitBI - 1) / kSplitBI - tl.y;
  const int t0 = tl.y + static_cast<int>(static_cast<int64_t>(njt) * blockIdx.y / gridDim.y);
  const int t1 = tl.y + static_cast<int>(static_cast<int64_t>(njt) * (blockIdx.y + 1) / gridDim.y);
  double* out = partial + static_cast<int64_t>(blockIdx.y) * gridDim.x + blockIdx.x;
  if (*wide || sd.n < kSplitMin || t0 == t1) {
    if (tid == 0) *out = 0.0;
    return;
  }
  const float4* recs = reinterpret_cast<const float4*>(pos + 4 * sd.offset);
  const float2 e2 = both(eps2);
  const int li = tl.y * kSplitBI + tid;
  const int64_t g = sd.offset + min(li, sd.n - 1);
  const float2 nx = both(-pos[pair_index(g, 0)]), ny = both(-pos[pair_index(g, 1)]),
               nz = both(-pos[pair_index(g, 2)]);
  const double mi = li < sd.n ? static_cast<double>(pos[pair_index(g, 3)]) : 0.0;
  double acc = 0.0;
  for (int t = t0; t < t1; ++t) {
    const int cnt = min(kSplitBI, sd.n - t * kSplitBI);
    const int npairs = (cnt + 1) / 2;
    __syncthreads();
    for (int k = tid; k < 2 * npairs; k += kSplitThreads)
      tile[k] = recs[static_cast<int64_t>(t) * kSplitBI + k];
    __syncthreads();
    const bool diag = t == tl.y;
    for (int p = 0; p < npairs; p += kSplitFlush) {
      float2 s = both(0.f), l = s, k = s;
      const int p1 = min(npairs, p + kSplitFlush);
      if (diag || cnt < kSplitBI)
        split_pairs<kMass, true>(tile, p, p1, cnt, nx, ny, nz, e2, diag ? tid : -2, s, l, k);
      else
        split_pairs<kMass, false>(tile, p, p1, cnt, nx, ny, nz, e2, 0, s, l, k);
      acc += (static_cast<double>(s.x) + static_cast<double>(s.y)) +
             ((static_cast<double>(l.x) + static_cast<double>(l.y)) +
              static_cast<double>(k.x + k.y));
    }
    if (diag) acc *= 0.5;
  }
  double v = mi * acc;
  if (!kMass) v *= static_cast<double>(pos[pair_index(sd.offset, 3)]);  // the common m_j
  const double total = block_sum(-G * v, sh);
  if (tid == 0) *out = total;
}

// ---- potential, FP64 pairs ----------------------------------------------------------
// blockIdx.x: i-tile tiles[x] = (system, tile); blockIdx.y: one of gridDim.y spans of the
// j-tiles from it to the end of the system (a small system has few i-tiles: one CTA each
// left 3,000 particles at 3.6 ms).  Writes its part of -G * sum_i m_i sum_{j>i} m_j /
// sqrt(r^2 + eps), zero where the split kernel does the system (`split`: it is launched).
constexpr int kPotThreads = 128;

__global__ void __launch_bounds__(kPotThreads) potential_kernel(
    const float* __restrict__ pos, const SystemDesc* __restrict__ sys,
    const int2* __restrict__ tiles, const int* __restrict__ wide, bool split, float eps2, double G,
    double* __restrict__ partial) {
  __shared__ double sh[kPotThreads];
  __shared__ double tj[4][kPotThreads];
  const int2 tl = tiles[blockIdx.x];
  const SystemDesc sd = sys[tl.x];
  const int njt = (sd.n + kPotThreads - 1) / kPotThreads - tl.y;
  const int t0 = tl.y + static_cast<int>(static_cast<int64_t>(njt) * blockIdx.y / gridDim.y);
  const int t1 = tl.y + static_cast<int>(static_cast<int64_t>(njt) * (blockIdx.y + 1) / gridDim.y);
  double* out = partial + static_cast<int64_t>(blockIdx.y) * gridDim.x + blockIdx.x;
  if (t0 == t1 || (split && !*wide && sd.n >= kSplitMin)) {
    if (threadIdx.x == 0) *out = 0.0;
    return;
  }
  const int li = tl.y * kPotThreads + threadIdx.x;
  const bool valid = li < sd.n;
  const int64_t gi = sd.offset + (valid ? li : 0);
  const double xi = pos[pair_index(gi, 0)], yi = pos[pair_index(gi, 1)],
               zi = pos[pair_index(gi, 2)], mi = pos[pair_index(gi, 3)];
  const double e2 = eps2;
  double sum = 0.0;
  for (int t = t0; t < t1; ++t) {
    const int j0 = t * kPotThreads;
    const int cnt = min(kPotThreads, sd.n - j0);
    __syncthreads();
    if (static_cast<int>(threadIdx.x) < cnt) {
      const int64_t gj = sd.offset + j0 + threadIdx.x;
#pragma unroll
      for (int c = 0; c < 4; ++c) tj[c][threadIdx.x] = pos[pair_index(gj, c)];
    }
    __syncthreads();
    if (!valid) continue;
    for (int k = t == tl.y ? static_cast<int>(threadIdx.x) + 1 : 0; k < cnt; ++k) {
      const double dx = tj[0][k] - xi, dy = tj[1][k] - yi, dz = tj[2][k] - zi;
      const double d2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, e2)));
      sum = fma(tj[3][k], rsqrt(d2), sum);
    }
  }
  const double s = block_sum(valid ? -G * mi * sum : 0.0, sh);
  if (threadIdx.x == 0) *out = s;
}

// out[0]: the sum of the potential's parts; out[1 + c]: column c of the moments.  One
// CTA each; a thread adds a stride of the parts in order, then a fixed tree.
__global__ void __launch_bounds__(kDiagThreads) reduce_partials_kernel(
    const double* __restrict__ moments, int mblocks, const double* __restrict__ potential,
    int64_t parts, double* __restrict__ out) {
  __shared__ double sh[kDiagThreads];
  const int c = static_cast<int>(blockIdx.x) - 1;
  const double* src = c < 0 ? potential : moments + c;
  const int64_t count = c < 0 ? parts : mblocks, stride = c < 0 ? 1 : kDiagVals;
  double s = 0.0;
  for (int64_t b = threadIdx.x; b < count; b += kDiagThreads) s += src[b * stride];
  s = block_sum(s, sh);
  if (threadIdx.x == 0) out[blockIdx.x] = s;
}

// FP64 acceleration of row r: G * sum_{j != i} m_j (x_j - x_i) / (|.|^2 + eps)^(3/2).
__global__ void fp64_rows_kernel(const float* __restrict__ pos, const SystemDesc* __restrict__ sys,
                                 const int64_t* __restrict__ rows, const int32_t* __restrict__ rsys,
                                 float eps2, double G, double* __restrict__ out) {
  __shared__ double sh[kDiagThreads];
  const int64_t gi = rows[blockIdx.x];
  const SystemDesc sd = sys[rsys[blockIdx.x]];
  const double xi = pos[pair_index(gi, 0)], yi = pos[pair_index(gi, 1)],
               zi = pos[pair_index(gi, 2)];
  double ax = 0.0, ay = 0.0, az = 0.0;
  for (int j = threadIdx.x; j < sd.n; j += blockDim.x) {
    const int64_t gj = sd.offset + j;
    if (gj == gi) continue;
    const double dx = pos[pair_index(gj, 0)] - xi, dy = pos[pair_index(gj, 1)] - yi,
                 dz = pos[pair_index(gj, 2)] - zi;
    const double d2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, static_cast<double>(eps2))));
    const double inv = rsqrt(d2);
    const double s = static_cast<double>(pos[pair_index(gj, 3)]) * inv * inv * inv;
    ax = fma(dx, s, ax);
    ay = fma(dy, s, ay);
    az = fma(dz, s, az);
  }
  ax = block_sum(ax, sh);
  ay = block_sum(ay, sh);
  az = block_sum(az, sh);
  if (threadIdx.x == 0) {
    out[3 * blockIdx.x + 0] = G * ax;
    out[3 * blockIdx.x + 1] = G * ay;
    out[3 * blockIdx.x + 2] = G * az;
  }
}

}  // namespace

cudaError_t launch_diagnostics(const float* pos, const float4* vel, const SystemDesc* sys_d,
                               const SystemDesc* sys_h, int32_t first_sys, int32_t num_sys,
                               float eps2, float G, bool per_pair_mass, int sms, double* out10,
                               DiagScratch& scratch, cudaStream_t stream) {
  const int64_t first = sys_h[first_sys].offset;
  const int64_t last = sys_h[first_sys + num_sys - 1].offset + sys_h[first_sys + num_sys - 1].npad;
  const int mblocks = static_cast<int>(
      std::min<int64_t>(1024, (last - first + kDiagThreads - 1) / kDiagThreads));
  // i-tiles of the FP64 kernel, and of the split one over the systems large enough.
  if (scratch.first_sys != first_sys || scratch.num_sys != num_sys || !scratch.partial) {
    std::vector<int2> tiles;
    auto list = [&](int bi, int min_n) {
      const size_t n0 = tiles.size();
      for (int32_t s = first_sys; s < first_sys + num_sys; ++s)
        for (int t = 0; sys_h[s].n >= min_n && t < (sys_h[s].n + bi - 1) / bi; ++t)
          tiles.push_back(make_int2(s, t));
      return static_cast<int64_t>(tiles.size() - n0);
    };
    const int64_t nfp64 = list(kPotThreads, 1);
    const int64_t nsplit = list(kSplitBI, kSplitMin);
    // Spans per i-tile: enough CTAs per SM that the triangle's uneven shares even out.
    auto spans_of = [&](int64_t tiles_n, int per_sm) {
      return static_cast<int32_t>(
          std::max<int64_t>(1, std::min<int64_t>(64, per_sm * sms / std::max<int64_t>(1, tiles_n))));
    };
    scratch.spans = spans_of(nsplit, 64);
    scratch.fp64_spans = spans_of(nfp64, 16);
    const int64_t parts = nfp64 * scratch.fp64_spans + nsplit * scratch.spans;
    const int64_t need = static_cast<int64_t>(mblocks) * kDiagVals + parts + nfp64 + nsplit + 1;
    scratch.num_sys = 0;
    if (scratch.cap < need) {
      if (scratch.partial) cudaFree(scratch.partial);
      scratch.partial = nullptr;
      scratch.cap = 0;
      const cudaError_t e = cudaMalloc(&scratch.partial, need * sizeof(double));
      if (e != cudaSuccess) return e;
      scratch.cap = need;
    }
    scratch.nfp64 = nfp64;
    scratch.nsplit = nsplit;
    // The list is pageable: the copy has read it before it returns.
    const cudaError_t e =
        cudaMemcpyAsync(scratch.partial + mblocks * kDiagVals + parts, tiles.data(),
                        tiles.size() * sizeof(int2), cudaMemcpyHostToDevice, stream);
    if (e != cudaSuccess) return e;
    scratch.first_sys = first_sys;
    scratch.num_sys = num_sys;
  }
  const int64_t fp64_parts = scratch.nfp64 * scratch.fp64_spans;
  const int64_t parts = fp64_parts + scratch.nsplit * scratch.spans;
  double* mom_part = scratch.partial;
  double* pot_part = mom_part + static_cast<int64_t>(mblocks) * kDiagVals;
  const int2* tiles = reinterpret_cast<const int2*>(pot_part + parts);
  int* wide = reinterpret_cast<int*>(pot_part + parts + scratch.nfp64 + scratch.nsplit);
  const bool split = scratch.nsplit > 0 && eps2 >= kSplitEps;
  cudaError_t e = cudaMemsetAsync(wide, 0, sizeof(int), stream);
  if (e != cudaSuccess) return e;
  moments_kernel<<<mblocks, kDiagThreads, 0, stream>>>(pos, vel, first, last, mom_part, wide);
  potential_kernel<<<dim3(static_cast<unsigned>(scratch.nfp64), scratch.fp64_spans), kPotThreads, 0,
                     stream>>>(
      pos, sys_d, tiles, wide, split, eps2, G, pot_part);
  if (split) {
    const dim3 grid(static_cast<unsigned>(scratch.nsplit), scratch.spans);
    auto kernel = per_pair_mass ? potential_split_kernel<true> : potential_split_kernel<false>;
    kernel<<<grid, kSplitThreads, 0, stream>>>(pos, sys_d, tiles + scratch.nfp64, wide, eps2, G,
                                               pot_part + fp64_parts);
  }
  reduce_partials_kernel<<<10, kDiagThreads, 0, stream>>>(mom_part, mblocks, pot_part,
                                                          split ? parts : fp64_parts, out10);
  return cudaGetLastError();
}

cudaError_t launch_fp64_rows(const float* pos, const SystemDesc* sys_d, const int64_t* rows_dev,
                             const int32_t* row_sys_dev, int64_t count, float eps2, float G, bool,
                             double* out3, cudaStream_t stream) {
  if (count <= 0) return cudaSuccess;
  fp64_rows_kernel<<<static_cast<unsigned>(count), kDiagThreads, 0, stream>>>(
      pos, sys_d, rows_dev, row_sys_dev, eps2, G, out3);
  return cudaGetLastError();
}

}  // namespace nbg
