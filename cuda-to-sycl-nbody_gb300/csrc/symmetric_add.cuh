// The adding pass of the symmetric kernels (symmetric_kernel.cuh, adjoint_kernel.cu): a
// particle's sum over its i-tile's parts (the CTAs that shared it) minus the rows of the
// i-tiles before its own, in a fixed order, compensated or plain.  With several bands
// the running sum is carried from band to band.
//
// What bounds it: load latency (a particle of a 4,096-particle system has up to 130
// terms of 12 to 32 bytes, a few MB in all, from L2), not bandwidth.  So a CTA is 32
// particles by 8 groups, each group adding a contiguous range of the terms, eight loads
// in flight, and the groups' sums are added in order: 4,096 particles took 45 us per
// step with one thread per particle, 18 with 8 groups.  With more particles or fewer terms
// the latency is hidden without so many groups (add_shape).
#pragma once

#include <cuda_runtime.h>

#include "nb_device.cuh"
#include "nb_internal.hpp"
#include "symmetric.hpp"

namespace nbg {

constexpr int kAddBatch = 8;
// Particles by groups of a CTA, for bands of `padded` particles (tiles times bi) with
// `terms` rows and parts per particle on average.  us per step, 32 x 8, 32 x 4, 64 x 2 and
// 64 x 1: ensembles of 4,096 systems of up to 1,024 particles (1.6 terms) 515 384 338 303,
// 640 of up to 4,096 (3.0) 452 400 381 369, 100 of up to 1,024 (7.2) 19.1 16.1 15.1 15.1, 40
// of up to 4,096 (11) 32.9 29.4 28.2 29.0; single systems of 5,000 particles (70) 14.7
// 15.5 18.3 24.2, 8,192 (54) 25.0 25.3 26.5 30.2, 10,000 35.0 34.8 36.2 39.1, 20,000 105.5
// 103.5 104.3 107.0, 40,000 380.0 376.6 375.8 378.3, 100,000 (18) 2,173 2,164 2,161 2,160.
struct AddShape {
  int lanes, groups;
};
inline AddShape add_shape(int64_t padded, float terms) {
  if (terms < 8.f) return {64, 1};
  if (terms < 32.f || padded >= 32768) return {64, 2};
  return padded >= 10000 ? AddShape{32, 4} : AddShape{32, 8};
}

// What the pass reads: the band [tile0, tile1) of i-tiles, its rows and parts.
struct AddTerms {
  const SymTile* tiles;
  const float* rows;
  int64_t plane;
  float4* carry;  // running sums, with their low words if compensated
  const float4* partials;
  int tile0, tile1;
};

struct AddResult {
  int64_t g;      // particle
  float x, y, z;  // its sum
};

namespace {

template <bool kComp>
struct Sum3 {
  float s[3] = {0.f, 0.f, 0.f}, c[3] = {0.f, 0.f, 0.f};
  __device__ __forceinline__ void add(int k, float t) {
    if (kComp) {
      const float y = t - c[k], u = s[k] + y;
      c[k] = (u - s[k]) - y;
      s[k] = u;
    } else {
      s[k] += t;
    }
  }
};

// blockIdx.x: i-tile tile0 + x of the band's systems; blockIdx.y: kAddLanes of its
// particles.  True in the one thread per particle that holds its complete sum (in `out`).
// early.lists(sys) runs before the predecessor's results are waited for, early.state(g)
// after that and before the sums, in the thread that will finish particle g.
template <int kAddLanes, int kAddGroups, bool kComp, class Early>
__device__ __forceinline__ bool add_terms(const AddTerms& a, int bi, Early& early,
                                          AddResult& out) {
  __shared__ float group_sum[kAddGroups][6][kAddLanes];
  const int t = a.tile0 + blockIdx.x;
  const SymTile tile = a.tiles[t];
  const int sys0 = t - tile.itile;  // the system's first i-tile
  const int64_t row_first = a.tiles[max(sys0, a.tile0)].row;
  early.lists(tile.sys);
  pdl_wait();
  const int lane = threadIdx.x % kAddLanes, group = threadIdx.x / kAddLanes;
  const int idx = blockIdx.y * kAddLanes + lane;
  const int j = tile.itile * bi + idx;
  if (j - lane >= tile.n) return false;
  const bool real = j < tile.n;
  const int64_t g = tile.offset + j;
  const int i0 = max(0, a.tile0 - sys0);  // the band's first i-tile in the system
  const bool mine = t < a.tile1;          // the particle's i-tile is in the band
  const int nrows = (mine ? tile.itile : a.tile1 - sys0) - i0;
  const int nparts = mine ? tile.nslots : 0;

  if (group == 0 && real) early.state(g);

  Sum3<kComp> sum;
  float q[3] = {0.f, 0.f, 0.f};  // low words of the parts
  // The group's rows.  The row of each i-tile is bi values shorter than the one before.
  const int k1 = real ? nrows * (group + 1) / kAddGroups : 0;
  int k = nrows * group / kAddGroups;
  const int64_t npad = (tile.n + kPadQuantum - 1) & -kPadQuantum;
  int64_t step = npad - static_cast<int64_t>(i0 + 2 + k) * bi;  // from row k to row k + 1
  const float* row = a.rows + (row_first + j + k * (npad - static_cast<int64_t>(i0 + 2) * bi) -
                               bi * (static_cast<int64_t>(k) * (k - 1) / 2));
  for (; k < k1; k += kAddBatch) {
    float v[kAddBatch][3];
#pragma unroll
    for (int u = 0; u < kAddBatch; ++u) {
      const bool in = k + u < k1;
      v[u][0] = in ? -row[0] : 0.f;
      v[u][1] = in ? -row[a.plane] : 0.f;
      v[u][2] = in ? -row[2 * a.plane] : 0.f;
      row += step;
      step -= bi;
    }
#pragma unroll
    for (int u = 0; u < kAddBatch; ++u)
#pragma unroll
      for (int c = 0; c < 3; ++c) sum.add(c, v[u][c]);
  }
  // The group's parts.
  constexpr int kRec = kComp ? 2 : 1;
  const int p1 = real ? nparts * (group + 1) / kAddGroups : 0;
  int p = nparts * group / kAddGroups;
  const float4* part =
      a.partials + (static_cast<int64_t>(tile.slot0 + p) * bi + idx) * kRec;
  for (; p < p1; p += kAddBatch / 2) {
    float4 h[kAddBatch / 2], l[kAddBatch / 2];
#pragma unroll
    for (int u = 0; u < kAddBatch / 2; ++u) {
      const bool in = p + u < p1;
      h[u] = in ? part[0] : make_float4(0.f, 0.f, 0.f, 0.f);
      if (kComp) l[u] = in ? part[1] : make_float4(0.f, 0.f, 0.f, 0.f);
      part += static_cast<int64_t>(bi) * kRec;
    }
#pragma unroll
    for (int u = 0; u < kAddBatch / 2; ++u) {
      sum.add(0, h[u].x);
      sum.add(1, h[u].y);
      sum.add(2, h[u].z);
      if (kComp) q[0] += l[u].x, q[1] += l[u].y, q[2] += l[u].z;
    }
  }
  pdl_trigger();
  // Group sums in order, each as its sum and what is still to be added to it.
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    group_sum[group][c][lane] = sum.s[c];
    group_sum[group][3 + c][lane] = kComp ? q[c] - sum.c[c] : 0.f;
  }
  __syncthreads();
  if (group > 0 || !real) return false;
  Sum3<kComp> all;
  float low[3] = {0.f, 0.f, 0.f};
  if (sys0 < a.tile0) {  // earlier bands
    const float4 s = a.carry[kRec * g];
    all.s[0] = s.x, all.s[1] = s.y, all.s[2] = s.z;
    if (kComp) {
      const float4 l = a.carry[kRec * g + 1];
      low[0] = l.x, low[1] = l.y, low[2] = l.z;
    }
  }
#pragma unroll
  for (int u = 0; u < kAddGroups; ++u)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      all.add(c, group_sum[u][c][lane]);
      if (kComp) low[c] += group_sum[u][3 + c][lane];
    }
  if (kComp)
#pragma unroll
    for (int c = 0; c < 3; ++c) low[c] -= all.c[c];
  if (!mine) {  // later bands add the rest
    a.carry[kRec * g] = make_float4(all.s[0], all.s[1], all.s[2], 0.f);
    if (kComp) a.carry[kRec * g + 1] = make_float4(low[0], low[1], low[2], 0.f);
    return false;
  }
  out = AddResult{g, all.s[0] + low[0], all.s[1] + low[1], all.s[2] + low[2]};
  return true;
}

template <int kLanes>
dim3 add_grid(int tiles, int bi) {
  return dim3(tiles, bi / kLanes);
}

}  // namespace

}  // namespace nbg
