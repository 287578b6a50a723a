// Adjoint (vector-Jacobian product) of one force + integrate iteration.
//
// Forward iteration (src/simulator.cu:193-228, masses and G made explicit):
//   v' = d v + dt G F(x),  x' = x + dt v',
//   F_i(x) = sum_{j != i} m_j r_ij f(|r_ij|^2 + eps),  r_ij = x_j - x_i,  f(s) = s^(-3/2).
// Given the cotangents (lx', lv') of (x', v'):
//   mu = lv' + dt lx',   lv = d mu,   lx = lx' + dt G J(x)^T mu,
// (mu is formed where it is read; lx and lv are written by the combining pass),
// and, with K_ij = s_ij I - 3 q_ij r_ij r_ij^T (s = f, q = s / (r^2 + eps)), which is
// symmetric in i and j,
//   (J^T mu)_i = sum_{j != i} K_ij u_ij,  u_ij = m_i mu_j - m_j mu_i
//              = sum_{j != i} s_ij (u_ij + c_ij r_ij),  c_ij = -3 (r_ij . u_ij) / (r^2 + eps).
// u_ji = -u_ij, so K_ij u_ij is the term of both particles, with opposite signs, and an
// unordered pair is evaluated once.
//
// What bounds it: the FP32 FMA pipe.  A pair is 25 lane operations for both sides (22
// for one, the diagonal block's) and one MUFU rsqrt; equal masses: u = mu_j - mu_i, and
// the common mass goes into the final scale.  A backward step (this product; every
// ordered pair evaluated before) takes 118 us at N = 16,384 (207 before), 135 with
// per-particle masses (232), 18.5 at 4,690 (47.2), 1,705 at 65,536 (3,454).  Small
// systems evaluate every ordered pair in one launch (adjoint_direct_kernel).
//
// The tiling is that of the symmetric force kernel (symmetric_kernel.cuh) with one warp
// per CTA: a warp's 32 j-particles, with their cotangents and running sums, rotate
// through its lanes past 64 P i-particles held two per packed register pair; the j-side
// sums go to rows of scratch, and adjoint_add_kernel adds a particle's rows and i-side
// parts in order and applies lx = lx' + dt G (J^T mu), lv = d mu.  Lanes past the end of
// a system hold zeros and are masked by index, as j-particles: as i-particles they are
// in a system's last i-tile, whose blocks are all diagonal.
#include <cuda_runtime.h>

#include <cstdint>

#include "direct.cuh"
#include "nb_device.cuh"
#include "nb_internal.hpp"
#include "nb_kernels.hpp"
#include "symmetric.hpp"
#include "symmetric_add.cuh"

namespace nbg {
namespace {

constexpr int kAdjBJ = 32;     // j-particles a warp rotates at a time
constexpr int kAdjFold = 512;  // j-particles between two folds of the i-side sums

__device__ __forceinline__ float adj_rot(float v, int src) {
  return __shfl_sync(0xffffffffu, v, src);
}

template <int P>
struct AdjI {
  float2 nx[P], ny[P], nz[P];  // minus the positions
  float2 wx[P], wy[P], wz[P];  // minus mu
  float2 m[P];
  float2 gx[P], gy[P], gz[P];  // sums since the last fold
};

struct AdjJ {
  float x, y, z, m, ux, uy, uz;  // position, mass, mu
};

// One j-particle against the thread's i-particles.  kPair: both sides (f: the j side's
// sums of the i side's terms); kMask: leave out j == i and j >= n, where the thread's
// i-particles are li0, li0 + kStep, li0 + 2 kStep and so on.
template <int P, int kStep, bool kMass, bool kPair, bool kMask>
__device__ __forceinline__ void adj_meet(AdjI<P>& q, const AdjJ& v, float2 e2, float2& fx,
                                         float2& fy, float2& fz, int jj, int li0, int n) {
  const float2 m3c = make_float2(-3.f, -3.f);
  const float2 xx = make_float2(v.x, v.x), yy = make_float2(v.y, v.y),
               zz = make_float2(v.z, v.z), mm = make_float2(v.m, v.m);
  const float2 jx = make_float2(v.ux, v.ux), jy = make_float2(v.uy, v.uy),
               jz = make_float2(v.uz, v.uz);
#pragma unroll
  for (int r = 0; r < P; ++r) {
    const float2 dx = __fadd2_rn(xx, q.nx[r]);
    const float2 dy = __fadd2_rn(yy, q.ny[r]);
    const float2 dz = __fadd2_rn(zz, q.nz[r]);
    float2 ux, uy, uz;
    if (kMass) {
      ux = __ffma2_rn(mm, q.wx[r], __fmul2_rn(q.m[r], jx));
      uy = __ffma2_rn(mm, q.wy[r], __fmul2_rn(q.m[r], jy));
      uz = __ffma2_rn(mm, q.wz[r], __fmul2_rn(q.m[r], jz));
    } else {
      ux = __fadd2_rn(jx, q.wx[r]);
      uy = __fadd2_rn(jy, q.wy[r]);
      uz = __fadd2_rn(jz, q.wz[r]);
    }
    float2 d2 = __ffma2_rn(dx, dx, e2);
    d2 = __ffma2_rn(dy, dy, d2);
    d2 = __ffma2_rn(dz, dz, d2);
    float2 inv = make_float2(rsqrtf(d2.x), rsqrtf(d2.y));
    if (kMask) {
      if (jj == li0 + 2 * kStep * r || jj >= n) inv.x = 0.f;
      if (jj == li0 + 2 * kStep * r + kStep || jj >= n) inv.y = 0.f;
    }
    const float2 inv2 = __fmul2_rn(inv, inv);
    const float2 s = __fmul2_rn(inv2, inv);
    const float2 m3 = __fmul2_rn(inv2, m3c);
    float2 rw = __fmul2_rn(dx, ux);
    rw = __ffma2_rn(dy, uy, rw);
    rw = __ffma2_rn(dz, uz, rw);
    const float2 c = __fmul2_rn(rw, m3);
    const float2 tx = __ffma2_rn(c, dx, ux);
    const float2 ty = __ffma2_rn(c, dy, uy);
    const float2 tz = __ffma2_rn(c, dz, uz);
    q.gx[r] = __ffma2_rn(s, tx, q.gx[r]);
    q.gy[r] = __ffma2_rn(s, ty, q.gy[r]);
    q.gz[r] = __ffma2_rn(s, tz, q.gz[r]);
    if (kPair) {
      fx = __ffma2_rn(s, tx, fx);
      fy = __ffma2_rn(s, ty, fy);
      fz = __ffma2_rn(s, tz, fz);
    }
  }
}

// 32 rotations of the warp's j-particles against its i-particles (adj_meet).
template <int P, int U, bool kMass, bool kPair, bool kMask>
__device__ __forceinline__ void adj_chunk(AdjI<P>& q, AdjJ v, float2 e2, float (&out)[3], int jj,
                                          int li0, int n) {
  const int src = (threadIdx.x + 1) & 31;
  float2 fx = make_float2(0.f, 0.f), fy = fx, fz = fx;
#pragma unroll 1
  for (int k = 0; k < kAdjBJ; k += U) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      adj_meet<P, 32, kMass, kPair, kMask>(q, v, e2, fx, fy, fz, jj, li0, n);
      v.x = adj_rot(v.x, src);
      v.y = adj_rot(v.y, src);
      v.z = adj_rot(v.z, src);
      if (kMass) v.m = adj_rot(v.m, src);
      v.ux = adj_rot(v.ux, src);
      v.uy = adj_rot(v.uy, src);
      v.uz = adj_rot(v.uz, src);
      if (kMask) jj = __shfl_sync(0xffffffffu, jj, src);
      if (kPair) {
        fx.x = adj_rot(fx.x, src);
        fx.y = adj_rot(fx.y, src);
        fy.x = adj_rot(fy.x, src);
        fy.y = adj_rot(fy.y, src);
        fz.x = adj_rot(fz.x, src);
        fz.y = adj_rot(fz.y, src);
      }
    }
  }
  out[0] = fx.x + fx.y;
  out[1] = fy.x + fy.y;
  out[2] = fz.x + fz.y;
}

// mu = lv' + dt lx' of particle g.
__device__ __forceinline__ float3 adj_mu(const AdjointArgs& a, int64_t g) {
  const float4 lx = a.lam_x[g], lv = a.lam_v[g];
  return make_float3(fmaf(a.dt, lx.x, lv.x), fmaf(a.dt, lx.y, lv.y), fmaf(a.dt, lx.z, lv.z));
}

template <int P, int U, bool kMass>
__global__ void __launch_bounds__(32, 8) adjoint_pair_kernel(const AdjointArgs a) {
  constexpr int BI = 64 * P;
  __shared__ float2 sums[3 * P][32];
  const int lane = threadIdx.x;
  const float2 e2 = make_float2(a.eps2, a.eps2);
  const float2 zero = make_float2(0.f, 0.f);
  SymSegment sg = a.segs[blockIdx.x];
  pdl_wait();
  for (bool more = true; more;) {
    const int next = sg.next;
    more = next > 0;
    const int ibase = sg.itile * BI;
    const float* pos = a.pos + 4 * sg.offset;
    AdjI<P> q;
#pragma unroll
    for (int r = 0; r < P; ++r) {
      float v[2][7];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int li = min(ibase + 64 * r + 32 * h + lane, sg.n - 1);
        const float3 mu = adj_mu(a, sg.offset + li);
#pragma unroll
        for (int c = 0; c < 4; ++c) v[h][c] = pos[pair_index(li, c)];
        v[h][4] = mu.x, v[h][5] = mu.y, v[h][6] = mu.z;
      }
      q.nx[r] = make_float2(-v[0][0], -v[1][0]);
      q.ny[r] = make_float2(-v[0][1], -v[1][1]);
      q.nz[r] = make_float2(-v[0][2], -v[1][2]);
      q.m[r] = make_float2(v[0][3], v[1][3]);
      q.wx[r] = make_float2(-v[0][4], -v[1][4]);
      q.wy[r] = make_float2(-v[0][5], -v[1][5]);
      q.wz[r] = make_float2(-v[0][6], -v[1][6]);
      q.gx[r] = q.gy[r] = q.gz[r] = zero;
    }

    AdjJ nj;  // the lane's j-particle of the next chunk, loaded one chunk ahead
    auto fetch = [&](int jt) {
      const int j = jt * kAdjBJ + lane;
      nj = AdjJ{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (jt < sg.jt1 && j < sg.n) {
        const float3 mu = adj_mu(a, sg.offset + j);
        nj.x = pos[pair_index(j, 0)];
        nj.y = pos[pair_index(j, 1)];
        nj.z = pos[pair_index(j, 2)];
        if (kMass) nj.m = pos[pair_index(j, 3)];
        nj.ux = mu.x, nj.uy = mu.y, nj.uz = mu.z;
      }
    };
    fetch(sg.jt0);
    bool folded = false;
    for (int jt = sg.jt0; jt < sg.jt1; ++jt) {
      const AdjJ v = nj;
      const int j0 = jt * kAdjBJ, j = j0 + lane;
      fetch(jt + 1);
      const bool diag = j0 < ibase + BI;
      const bool ragged = j0 + kAdjBJ > sg.n;
      float out[3];
      if (!diag) {
        if (ragged)
          adj_chunk<P, 1, kMass, true, true>(q, v, e2, out, j, -BI, sg.n);
        else
          adj_chunk<P, U, kMass, true, false>(q, v, e2, out, j, 0, sg.n);
        if (j < sg.n) {
          a.rows[sg.row + j] = out[0];
          a.rows[a.plane + sg.row + j] = out[1];
          a.rows[2 * a.plane + sg.row + j] = out[2];
        }
      } else if (ragged || a.mask_self) {
        adj_chunk<P, 1, kMass, false, true>(q, v, e2, out, j,
                                            a.mask_self ? ibase + lane : -BI, sg.n);
      } else {
        adj_chunk<P, U, kMass, false, false>(q, v, e2, out, j, 0, sg.n);
      }
      if (jt + 1 == sg.jt1 ? folded : (jt + 1 - sg.jt0) % (kAdjFold / kAdjBJ) == 0) {
#pragma unroll
        for (int r = 0; r < P; ++r) {
          sums[r][lane] = folded ? __fadd2_rn(sums[r][lane], q.gx[r]) : q.gx[r];
          sums[P + r][lane] = folded ? __fadd2_rn(sums[P + r][lane], q.gy[r]) : q.gy[r];
          sums[2 * P + r][lane] = folded ? __fadd2_rn(sums[2 * P + r][lane], q.gz[r]) : q.gz[r];
          q.gx[r] = q.gy[r] = q.gz[r] = zero;
        }
        folded = true;
      }
    }
    if (!more) pdl_trigger();
    float4* part = a.partials + static_cast<int64_t>(sg.slot) * BI;
#pragma unroll
    for (int r = 0; r < P; ++r) {
      const float2 sx = folded ? sums[r][lane] : q.gx[r];
      const float2 sy = folded ? sums[P + r][lane] : q.gy[r];
      const float2 sz = folded ? sums[2 * P + r][lane] : q.gz[r];
      part[64 * r + lane] = make_float4(sx.x, sy.x, sz.x, 0.f);
      part[64 * r + 32 + lane] = make_float4(sx.y, sy.y, sz.y, 0.f);
    }
    if (more) sg = a.segs[next - 1];
  }
}

struct EarlyAdjoint {
  const AdjointArgs& a;
  float gscale;
  float4 lx, lv;
  __device__ void lists(int sys) { gscale = a.sys[sys].gscale; }
  __device__ void state(int64_t g) {
    lx = a.lam_x[g];
    lv = a.lam_v[g];
  }
};

// lx = lx' + dt G (J^T mu), lv = d mu of particle g, from its sum f and its lx', lv'.
__device__ __forceinline__ void adj_finish(const AdjointArgs& a, float gscale, int64_t g, float fx,
                                           float fy, float fz, float4 l, float4 v) {
  const float c = a.dt * gscale;
  a.lam_x_out[g] = make_float4(fmaf(c, fx, l.x), fmaf(c, fy, l.y), fmaf(c, fz, l.z), 0.f);
  a.lam_v_out[g] = make_float4(a.damping * fmaf(a.dt, l.x, v.x), a.damping * fmaf(a.dt, l.y, v.y),
                               a.damping * fmaf(a.dt, l.z, v.z), 0.f);
}

template <int kLanes, int kGroups>
__global__ void __launch_bounds__(kLanes * kGroups) adjoint_add_kernel(const AdjointArgs a,
                                                                       int bi) {
  const AddTerms t{a.tiles, a.rows, a.plane, a.carry, a.partials, a.tile0, a.tile1};
  EarlyAdjoint e{a, 0.f, {}, {}};
  AddResult r;
  if (!add_terms<kLanes, kGroups, false>(t, bi, e, r)) return;
  adj_finish(a, e.gscale, r.g, r.x, r.y, r.z, e.lx, e.lv);
}

// Small systems (n * n <= kAdjDirectPairs: a thread's chains stay below 90 terms): the
// direct force kernel's scheme (direct_kernel.cu), W warps per CTA against R i-particles,
// B CTAs per SM.
template <int W, int R, int B, bool kMass>
__global__ void __launch_bounds__(W * 32, B) adjoint_direct_kernel(const AdjointArgs a,
                                                                   const int2* tiles, int sys) {
  constexpr int P = R / 2;
  __shared__ float part[3][W][R];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  int itile = blockIdx.x;
  if (tiles != nullptr) {
    const int2 t = tiles[blockIdx.x];
    sys = t.x, itile = t.y;
  }
  const SystemDesc sd = a.sys[sys];
  const int n = sd.n, i0 = itile * R;
  const float4* pos = reinterpret_cast<const float4*>(a.pos) + sd.offset;
  pdl_wait();
  const int64_t g = sd.offset + i0 + tid;
  const bool mine = tid < R && i0 + tid < n;
  float4 l = make_float4(0.f, 0.f, 0.f, 0.f), v = l;
  if (mine) l = a.lam_x[g], v = a.lam_v[g];
  AdjI<P> q;
#pragma unroll
  for (int p = 0; p < P; ++p) {
    const int i = i0 + 2 * p;  // R divides the padding
    const float4 u = pos[i], z = pos[i + 1];
    const float3 m0 = adj_mu(a, sd.offset + i), m1 = adj_mu(a, sd.offset + i + 1);
    q.nx[p] = make_float2(-u.x, -u.y);
    q.ny[p] = make_float2(-u.z, -u.w);
    q.nz[p] = make_float2(-z.x, -z.y);
    q.m[p] = make_float2(z.z, z.w);
    q.wx[p] = make_float2(-m0.x, -m1.x);
    q.wy[p] = make_float2(-m0.y, -m1.y);
    q.wz[p] = make_float2(-m0.z, -m1.z);
    q.gx[p] = q.gy[p] = q.gz[p] = make_float2(0.f, 0.f);
  }
  const float2 e2 = make_float2(a.eps2, a.eps2), zero = make_float2(0.f, 0.f);
  constexpr int kPass = W * 64;
  AdjJ b0, b1;  // two j-particles, loaded one pass ahead
  auto fetch = [&](int j) {
    b0 = b1 = AdjJ{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (j >= n) return;
    const float4 u = pos[j], z = pos[j + 1];  // j is even: j + 1 is padding at worst
    const float3 m0 = adj_mu(a, sd.offset + j), m1 = adj_mu(a, sd.offset + j + 1);
    b0 = AdjJ{u.x, u.z, z.x, z.z, m0.x, m0.y, m0.z};
    if (j + 1 < n) b1 = AdjJ{u.y, u.w, z.y, z.w, m1.x, m1.y, m1.z};
  };
  fetch(2 * tid);
  float2 fx = zero, fy = zero, fz = zero;  // no j side
#pragma unroll 1
  for (int j0 = 0; j0 < n; j0 += kPass) {
    const AdjJ c0 = b0, c1 = b1;
    const int j = j0 + 2 * tid;
    if (j0 + kPass < n) fetch(j + kPass);
    if (a.mask_self || j0 + kPass > n) {
      const int skip = a.mask_self ? i0 : -2 * R;
      adj_meet<P, 1, kMass, false, true>(q, c0, e2, fx, fy, fz, j, skip, n);
      adj_meet<P, 1, kMass, false, true>(q, c1, e2, fx, fy, fz, j + 1, skip, n);
    } else {
      adj_meet<P, 1, kMass, false, false>(q, c0, e2, fx, fy, fz, 0, 0, 0);
      adj_meet<P, 1, kMass, false, false>(q, c1, e2, fx, fy, fz, 0, 0, 0);
    }
  }
  float t[R][3];
#pragma unroll
  for (int p = 0; p < P; ++p) {
    t[2 * p][0] = q.gx[p].x, t[2 * p][1] = q.gy[p].x, t[2 * p][2] = q.gz[p].x;
    t[2 * p + 1][0] = q.gx[p].y, t[2 * p + 1][1] = q.gy[p].y, t[2 * p + 1][2] = q.gz[p].y;
  }
  warp_sums<R>(t);
  pdl_trigger();
  if (lane % (32 / R) == 0)
#pragma unroll
    for (int c = 0; c < 3; ++c) part[c][w][lane / (32 / R)] = t[0][c];
  __syncthreads();
  if (!mine) return;
  float f[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    f[c] = part[c][0][tid];
#pragma unroll
    for (int k = 1; k < W; ++k) f[c] += part[c][k][tid];
  }
  adj_finish(a, sd.gscale, g, f[0], f[1], f[2], l, v);
}

__global__ void unpack_vec3_kernel(const float* __restrict__ in, int64_t n,
                                   const int64_t* __restrict__ map, float4* __restrict__ out) {
  for (int64_t k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; k < n;
       k += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t g = map ? map[k] : k;
    out[g] = make_float4(in[3 * k], in[3 * k + 1], in[3 * k + 2], 0.f);
  }
}

__global__ void pack_vec3_kernel(const float4* __restrict__ in, int64_t n,
                                 const int64_t* __restrict__ map, float* __restrict__ out) {
  for (int64_t k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; k < n;
       k += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t g = map ? map[k] : k;
    const float4 v = in[g];
    out[3 * k] = v.x;
    out[3 * k + 1] = v.y;
    out[3 * k + 2] = v.z;
  }
}

int grid_for(int64_t n) {
  const int64_t b = (n + 255) / 256;
  return static_cast<int>(b < 1 ? 1 : (b > 1 << 20 ? 1 << 20 : b));
}

struct AdjEntry {
  int pairs;
  void (*kernel[2])(const AdjointArgs);  // [per-particle masses]
};
#define NBG_ADJ(P, U) {P, {adjoint_pair_kernel<P, U, false>, adjoint_pair_kernel<P, U, true>}}
// By choose_direct's index.
struct AdjDirectEntry {
  int warps, r;
  void (*kernel[2])(const AdjointArgs, const int2*, int);  // [per-particle masses]
};
#define NBG_ADJ_DIRECT(W, R, B) \
  {W, R, {adjoint_direct_kernel<W, R, B, false>, adjoint_direct_kernel<W, R, B, true>}}
const AdjDirectEntry kAdjDirect[] = {NBG_ADJ_DIRECT(8, 8, 2), NBG_ADJ_DIRECT(4, 4, 5),
                                     NBG_ADJ_DIRECT(4, 8, 4), NBG_ADJ_DIRECT(2, 8, 8),
                                     NBG_ADJ_DIRECT(1, 8, 16)};

const AdjEntry kAdjShapes[] = {NBG_ADJ(6, 1), NBG_ADJ(4, 2), NBG_ADJ(1, 4)};

}  // namespace

int num_adjoint_shapes() { return static_cast<int>(sizeof(kAdjShapes) / sizeof(kAdjShapes[0])); }

KernelShape adjoint_shape(int index) {
  return KernelShape{32, 2 * kAdjShapes[index].pairs, kAdjBJ, 0};
}

cudaError_t adjoint_blocks_per_sm(int index, bool per_pair_mass, int* blocks) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(
      blocks, kAdjShapes[index].kernel[per_pair_mass], 32, 0);
}

cudaError_t launch_adjoint(int index, bool per_pair_mass, const AdjointArgs& a, int grid,
                           cudaStream_t stream) {
  return launch_dependent(kAdjShapes[index].kernel[per_pair_mass], dim3(grid), 32, 0, stream, a);
}

cudaError_t launch_adjoint_direct(int index, bool per_pair_mass, const AdjointArgs& a,
                                  const int2* tiles, int sys, int grid, cudaStream_t stream) {
  const AdjDirectEntry& e = kAdjDirect[index];
  return launch_dependent(e.kernel[per_pair_mass], dim3(grid), dim3(e.warps * 32), 0, stream, a,
                          tiles, sys);
}

template <int kLanes, int kGroups>
static cudaError_t adjoint_add_one(const AdjointArgs& a, int tiles, int bi, cudaStream_t stream) {
  return launch_dependent(adjoint_add_kernel<kLanes, kGroups>, add_grid<kLanes>(tiles, bi),
                          kLanes * kGroups, 0, stream, a, bi);
}

cudaError_t launch_adjoint_add(const AdjointArgs& a, int tiles, int bi, float terms,
                               cudaStream_t stream) {
  const AddShape sh = add_shape(static_cast<int64_t>(tiles) * bi, terms);
  return sh.groups == 1   ? adjoint_add_one<64, 1>(a, tiles, bi, stream)
         : sh.groups == 2 ? adjoint_add_one<64, 2>(a, tiles, bi, stream)
         : sh.groups == 4 ? adjoint_add_one<32, 4>(a, tiles, bi, stream)
                          : adjoint_add_one<32, 8>(a, tiles, bi, stream);
}

cudaError_t launch_unpack_vec3(const float* in, int64_t n, const int64_t* map, float4* out,
                               cudaStream_t stream) {
  unpack_vec3_kernel<<<grid_for(n), 256, 0, stream>>>(in, n, map, out);
  return cudaGetLastError();
}

cudaError_t launch_pack_vec3(const float4* in, int64_t n, const int64_t* map, float* out,
                             cudaStream_t stream) {
  pack_vec3_kernel<<<grid_for(n), 256, 0, stream>>>(in, n, map, out);
  return cudaGetLastError();
}

}  // namespace nbg
