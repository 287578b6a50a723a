// Symmetric (Newton's third law) form of the tuned force step: each unordered pair of
// particles is evaluated once and applied to both (src/simulator.cu:193-228 evaluates
// all ordered pairs; the terms are the same, r_ij rsqrt(d2^3), and d2 is the same for
// both particles, so only the order of the sums differs).
//
// What bounds it: the FP32 FMA pipe.  One side of a pair costs 11 lane operations
// (force_kernel.cuh); both sides cost 14, because only the three multiply-adds of the
// sum are repeated: 7 per interaction.  Measured, ms per step against the tuned kernel
// (compensated, equal masses): N = 1,048,576 229.0 (347.1), 262,144 14.42 (21.7), 100,003
// with per-particle masses, plain 2.52 (3.56), 25,600 0.164 (0.242); the FMA pipe is 84 %
// busy at 262,144 and 75 % at 25,600 (one-warp CTAs: two warps per scheduler, of which the
// older runs at its full rate and the younger in its gaps until it is alone).
//
//   * Each thread holds 2 P i-particles, two per packed FP32x2 register pair.  A warp
//     takes 32 j-particles at a time, one per lane, and rotates them through its lanes
//     (shuffles) together with their three running sums; after 32 steps each j has met
//     the warp's 64 P i-particles and is back in its lane with its sum.  The rotation
//     costs 9 shuffles per 2 P pairs and lane, so P is as large as the registers allow:
//     at N = 1,048,576 P = 8, 7, 6 take 239, 242, 245 ms in CTAs of 8 warps, P = 8, 4, 2
//     248, 271, 310 in CTAs of one (2 to 4 steps per unrolled block make no difference).
//     Two j-particles in the packed registers against duplicated i-particles take 12
//     shuffles for the same pairs and hold half the i-particles: 71 % of the FMA pipe in
//     the pair loop alone, against 79 to 82 %.
//   * The i-side sums stay in registers over the segment's j-range, folded every F
//     j-particles into (compensated) running sums in shared memory; the j-side sums start
//     anew every S rotations.  No chain of additions is longer than the tuned kernel's at
//     the same size (symmetric_shapes.cu has the errors).
//   * The j-side sums of a j-tile are added over the CTA's warps in shared memory, in
//     warp order (double-buffered, one barrier per j-tile), and written to the i-tile's
//     row of scratch.  symmetric_add_kernel adds a particle's rows and its i-side parts
//     in a fixed order and integrates: results do not depend on timing.
//   * j-tiles inside the i-tile (the diagonal block) run the same loop for the i side
//     only, over all ordered pairs.  The self pair is masked there when eps2^3
//     underflows, as in force_kernel.cuh.
//   * Both kernels are launched as programmatic dependents: the next one is resident, its
//     list loaded, when its predecessor ends (12,800
//     particles 57.5 -> 50.7 us per step when both were new; 49.2 now).
//   * Lanes past the end of a system hold a particle at kFarAway: its terms are zero.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "nb_device.cuh"
#include "nb_internal.hpp"
#include "nb_kernels.hpp"
#include "symmetric.hpp"

namespace nbg {

namespace {

constexpr int kSymChunk = 32;  // j-particles a warp rotates at a time

// j-tile: what several warps add up at once; one chunk where a CTA is one warp, which
// writes its rows itself (and whose work lists are cut more finely).
template <int NW>
constexpr int kSymBJ = NW == 1 ? kSymChunk : 128;

// Kahan step on both lanes: (s, c) += t, with s + c the compensated value.
__device__ __forceinline__ void sym_kahan(float2& s, float2& c, float2 t) {
  const float2 y = __fadd2_rn(t, c);
  const float2 u = __fadd2_rn(s, y);
  c = __fadd2_rn(y, __ffma2_rn(u, make_float2(-1.f, -1.f), s));
  s = u;
}

// Fold t into the running sum *s (compensation at s[comp]) and clear it; the first fold
// of a segment starts the sum.
template <bool kComp>
__device__ __forceinline__ void sym_fold(bool folded, float2* s, int comp, float2& t) {
  const float2 zero = make_float2(0.f, 0.f);
  if (kComp) {
    float2 u = zero, c = zero;
    if (folded) u = s[0], c = s[comp];
    sym_kahan(u, c, t);
    s[0] = u;
    s[comp] = c;
  } else {
    s[0] = folded ? __fadd2_rn(s[0], t) : t;
  }
  t = zero;
}

__device__ __forceinline__ float sym_rot(float v, int src) {
  return __shfl_sync(0xffffffffu, v, src);
}

template <int P>
struct SymI {
  float2 nx[P], ny[P], nz[P];  // minus the positions
  float2 ax[P], ay[P], az[P];  // sums since the last fold
};

// One chunk: 32 rotations of the warp's j-particles (x, y, z, m) against its
// i-particles.  kPair: both sides (jx, jy, jz return the sums of r * s over the i
// side, to be subtracted from j's force); else the i side only.  kMask: leave out the
// pair with j == i, by index: jj is the lane's j, li the thread's i-particles.
template <int P, int U, int S, bool kMass, bool kPair, bool kMask>
__device__ __forceinline__ void sym_chunk(SymI<P>& q, const float2* mi, float x, float y, float z,
                                          float m, float2 e2, float& jx, float& jy, float& jz,
                                          int jj, int li0, int threads) {
  const int lane = threadIdx.x & 31;
  const int src = (lane + 1) & 31;
  float2 fx = make_float2(0.f, 0.f), fy = fx, fz = fx;
  jx = jy = jz = 0.f;
#pragma unroll 1
  for (int k = 0; k < kSymChunk; k += U) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float2 xx = make_float2(x, x), yy = make_float2(y, y), zz = make_float2(z, z);
#pragma unroll
      for (int r = 0; r < P; ++r) {
        const float2 dx = __fadd2_rn(xx, q.nx[r]);
        const float2 dy = __fadd2_rn(yy, q.ny[r]);
        const float2 dz = __fadd2_rn(zz, q.nz[r]);
        float2 d2 = __ffma2_rn(dx, dx, e2);
        d2 = __ffma2_rn(dy, dy, d2);
        d2 = __ffma2_rn(dz, dz, d2);
        float2 t = __fmul2_rn(d2, d2);
        t = __fmul2_rn(t, d2);
        float2 s = make_float2(rsqrtf(t.x), rsqrtf(t.y));
        if (kMask) {
          if (jj == li0 + 2 * r * threads) s.x = 0.f;
          if (jj == li0 + (2 * r + 1) * threads) s.y = 0.f;
        }
        const float2 si = kMass ? __fmul2_rn(s, make_float2(m, m)) : s;
        q.ax[r] = __ffma2_rn(dx, si, q.ax[r]);
        q.ay[r] = __ffma2_rn(dy, si, q.ay[r]);
        q.az[r] = __ffma2_rn(dz, si, q.az[r]);
        if (kPair) {
          const float2 sj = kMass ? __fmul2_rn(s, mi[r]) : s;
          fx = __ffma2_rn(dx, sj, fx);
          fy = __ffma2_rn(dy, sj, fy);
          fz = __ffma2_rn(dz, sj, fz);
        }
      }
      x = sym_rot(x, src);
      y = sym_rot(y, src);
      z = sym_rot(z, src);
      if (kMass) m = sym_rot(m, src);
      if (kMask) jj = __shfl_sync(0xffffffffu, jj, src);
      if (kPair) {
        fx.x = sym_rot(fx.x, src);
        fx.y = sym_rot(fx.y, src);
        fy.x = sym_rot(fy.x, src);
        fy.y = sym_rot(fy.y, src);
        fz.x = sym_rot(fz.x, src);
        fz.y = sym_rot(fz.y, src);
      }
    }
    if (kPair && S < kSymChunk && (S == U || (k + U) % S == 0)) {
      const int by = (lane + S) & 31;
      jx = sym_rot(jx, by) + (fx.x + fx.y);
      jy = sym_rot(jy, by) + (fy.x + fy.y);
      jz = sym_rot(jz, by) + (fz.x + fz.y);
      fx = fy = fz = make_float2(0.f, 0.f);
    }
  }
  if (kPair && S == kSymChunk) {
    jx = fx.x + fx.y;
    jy = fy.x + fy.y;
    jz = fz.x + fz.y;
  }
}

}  // namespace

// NW warps, P i-pairs per thread (i-tiles of 64 P NW particles), U rotations per unrolled
// block, S per sum of the j side (every one of them moves with its j-particle), F j-particles
// per fold of the i side.
// kXyzm: positions are a float4 (x, y, z, m) per particle, and no padding follows them.
template <int NW, int P, int U, int S, int F, bool kComp, bool kMass, bool kXyzm>
__global__ void __launch_bounds__(NW * 32, 8 / NW) symmetric_kernel(const SymArgs a) {
  constexpr int T = NW * 32;
  constexpr int BI = T * 2 * P;
  constexpr int BJ = kSymBJ<NW>;
  constexpr int kFoldTiles = F / BJ;
  static_assert(BI % BJ == 0 && F % BJ == 0, "i-tiles and folds hold whole j-tiles");
  extern __shared__ __align__(16) float sym_smem[];
  // Running i-side sums: [kComp ? 6 : 3][P] float2 per thread, and the j-side sums of
  // the warps: [2][NW][3][BJ] (one warp writes its row of scratch directly).
  constexpr int kSums = kComp ? 6 : 3;
  float2* sums = reinterpret_cast<float2*>(sym_smem) + threadIdx.x;
  float* jbuf = sym_smem + 2 * kSums * P * T;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const float2 e2 = make_float2(a.f.eps2, a.f.eps2);
  const float2 zero = make_float2(0.f, 0.f);
  int par = 0;  // buffer of the next j-tile's j-side sums

  // The lists are older than the predecessor's launch; the state is not.
  SymSegment sg = a.segs[blockIdx.x];
  pdl_wait();
  // Where the next segment is loaded makes no difference to what runs, but ptxas
  // schedules the pair loop differently (N = 1,048,576: 8 warps 229 ms at the top of the
  // loop, 239 at its end; one warp 252 and 244).
  constexpr bool kTop = NW == 8;
  for (int next = blockIdx.x + 1; next > 0;) {
    if (kTop && next != static_cast<int>(blockIdx.x) + 1) sg = a.segs[next - 1];
    next = sg.next;
    const int ibase = sg.itile * BI;
    const float* pos = a.f.pos + 4 * sg.offset;  // offsets are even: whole pair records

    auto at = [](int i, int c) -> int64_t {
      return kXyzm ? 4 * static_cast<int64_t>(i) + c : pair_index(i, c);
    };

    SymI<P> q;
    float2 mi[P];
#pragma unroll
    for (int r = 0; r < P; ++r) {
      float v[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int li = ibase + (2 * r + h) * T + tid;
        const bool real = li < sg.n;
#pragma unroll
        for (int c = 0; c < 4; ++c)
          v[h][c] = real ? pos[at(li, c)] : (c < 3 ? kFarAway : 0.f);
      }
      q.nx[r] = make_float2(-v[0][0], -v[1][0]);
      q.ny[r] = make_float2(-v[0][1], -v[1][1]);
      q.nz[r] = make_float2(-v[0][2], -v[1][2]);
      mi[r] = make_float2(v[0][3], v[1][3]);
      q.ax[r] = q.ay[r] = q.az[r] = zero;
    }

    // The lane's j-particle of the next chunk, loaded one chunk ahead.
    const int jend = min(kXyzm ? sg.n : (sg.n + kPadQuantum - 1) & -kPadQuantum, sg.jt1 * BJ);
    float nx = kFarAway, ny = kFarAway, nz = kFarAway, nm = 0.f;
    auto fetch = [&](int j0) {
      const int j = j0 + lane;
      const bool in = j < jend;
      nx = in ? pos[at(j, 0)] : kFarAway;
      ny = in ? pos[at(j, 1)] : kFarAway;
      nz = in ? pos[at(j, 2)] : kFarAway;
      if (kMass) nm = in ? pos[at(j, 3)] : 0.f;
    };
    fetch(sg.jt0 * BJ);

    bool folded = false;  // sums in shared memory
    for (int jt = sg.jt0; jt < sg.jt1; ++jt) {
      const int j0 = jt * BJ;
      const bool diag = j0 < ibase + BI;
      const int nch = min(BJ / kSymChunk, (jend - j0 + kSymChunk - 1) / kSymChunk);
      float* jb = jbuf + (par * NW + w) * 3 * BJ;
#pragma unroll 1
      for (int c = 0; c < nch; ++c) {
        const float x = nx, y = ny, z = nz, m = nm;
        const int j = j0 + c * kSymChunk + lane;
        fetch(j0 + (c + 1) * kSymChunk);
        float jx, jy, jz;
        if (!diag) {
          sym_chunk<P, U, S, kMass, true, false>(q, mi, x, y, z, m, e2, jx, jy, jz, j, 0, T);
          if (NW == 1) {
            if (j < sg.n) {
              a.rows[sg.row + j] = jx;
              a.rows[a.plane + sg.row + j] = jy;
              a.rows[2 * a.plane + sg.row + j] = jz;
            }
          } else {
            jb[c * kSymChunk + lane] = jx;
            jb[BJ + c * kSymChunk + lane] = jy;
            jb[2 * BJ + c * kSymChunk + lane] = jz;
          }
        } else if (a.f.mask_self) {
          sym_chunk<P, 1, S, kMass, false, true>(q, mi, x, y, z, m, e2, jx, jy, jz, j, ibase + tid,
                                                 T);
        } else {
          sym_chunk<P, U, S, kMass, false, false>(q, mi, x, y, z, m, e2, jx, jy, jz, j, 0, T);
        }
      }
      // Fold the i-side sums (never where the segment is short: they stay in registers).
      const int done = jt + 1 - sg.jt0;
      if (jt + 1 == sg.jt1 ? folded : done % kFoldTiles == 0) {
#pragma unroll
        for (int r = 0; r < P; ++r) {
          sym_fold<kComp>(folded, sums + r * T, 3 * P * T, q.ax[r]);
          sym_fold<kComp>(folded, sums + (P + r) * T, 3 * P * T, q.ay[r]);
          sym_fold<kComp>(folded, sums + (2 * P + r) * T, 3 * P * T, q.az[r]);
        }
        folded = true;
      }
      if (NW > 1 && !diag) {
        // Every warp has stored its part of this j-tile (and, one barrier earlier, had
        // read the other buffer): add them in warp order.
        __syncthreads();
        const float* src = jbuf + par * NW * 3 * BJ;
        const int cnt = min(BJ, sg.n - j0);
#pragma unroll
        for (int e = tid; e < 3 * BJ; e += T) {
          const int comp = e / BJ, j = e % BJ;
          float s = src[e];
#pragma unroll
          for (int v = 1; v < NW; ++v) s += src[v * 3 * BJ + e];
          if (j < cnt) a.rows[comp * a.plane + sg.row + j0 + j] = s;
        }
        par ^= 1;
      }
    }

    if (next <= 0) pdl_trigger();
    // The segment's i-side sums: (hi, lo) records, or the plain sums.
    constexpr int kRec = kComp ? 2 : 1;
    float4* part = a.f.partials + static_cast<int64_t>(sg.slot) * BI * kRec;
#pragma unroll
    for (int r = 0; r < P; ++r) {
      float2 sx = q.ax[r], sy = q.ay[r], sz = q.az[r], cx = zero, cy = zero, cz = zero;
      if (folded) {
        sx = sums[r * T], sy = sums[(P + r) * T], sz = sums[(2 * P + r) * T];
        if (kComp)
          cx = sums[(3 * P + r) * T], cy = sums[(4 * P + r) * T], cz = sums[(5 * P + r) * T];
      }
      const int i0 = 2 * r * T + tid, i1 = i0 + T;
      part[i0 * kRec] = make_float4(sx.x, sy.x, sz.x, 0.f);
      part[i1 * kRec] = make_float4(sx.y, sy.y, sz.y, 0.f);
      if (kComp) {
        part[i0 * kRec + 1] = make_float4(cx.x, cy.x, cz.x, 0.f);
        part[i1 * kRec + 1] = make_float4(cx.y, cy.y, cz.y, 0.f);
      }
    }
    if (!kTop && next > 0) sg = a.segs[next - 1];
  }
}

template <int NW, int P, bool kComp>
constexpr int symmetric_smem() {
  return 8 * (kComp ? 6 : 3) * P * NW * 32 + (NW > 1 ? 4 * 2 * NW * 3 * kSymBJ<NW> : 0);
}

}  // namespace nbg
