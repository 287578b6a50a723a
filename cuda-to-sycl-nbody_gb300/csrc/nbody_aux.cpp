// C ABI: FP64 diagnostics and the adjoint of the step (host side).
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <vector>

#include "nb_internal.hpp"
#include "nb_kernels.hpp"
#include "nb_runtime.hpp"
#include "nbody_gb300.h"

using namespace nbg;

namespace nbg {

void release_aux(nb_sim* s) {
  if (s->diag.partial) cudaFree(s->diag.partial);
  s->diag = DiagScratch{};
  dev_free(s->diag_out_d);
  AdjointState& a = s->adj;
  for (auto* p : a.ckpt_pos) cudaFree(p);
  for (auto* p : a.ckpt_vel) cudaFree(p);
  for (auto* p : a.seg_pos) cudaFree(p);
  dev_free(a.lam_x);
  dev_free(a.lam_v);
  dev_free(a.mu);
  dev_free(a.tmp);
  dev_free(a.vel);
  free_worklist(a.wl);
  a = AdjointState{};
}

}  // namespace nbg

namespace {

// The pair kernel's shape, and its largest grid.  The shapes' rates are measured at
// N = 65,536 (1.73, 1.83 and 2.30 ms per backward step); the blocks per CTA, where two
// neighbouring shapes meet (us per backward step with the larger / the smaller
// i-tiles): 16,384 133 / 131 and 65,536 1,730 / 1,830 for 768 against 256 particles;
// 4,690 30.6 / 28.7 and 16,384 131 / 159 for 256 against 64.
int adjoint_shape_for(const nb_sim* s, int* grid) {
  static constexpr double kRates[][2] = {{1.0, 6.0}, {0.945, 1.7}, {0.751, 0.0}};
  constexpr int kCount = sizeof(kRates) / sizeof(kRates[0]);
  SymCandidate c[kCount];
  for (int k = 0; k < kCount; ++k) {
    int per_sm = 0;
    if (adjoint_blocks_per_sm(k, s->per_pair_mass, &per_sm) != cudaSuccess || per_sm < 1)
      per_sm = 1;
    c[k] = SymCandidate{adjoint_shape(k), kRates[k][0], kRates[k][1], per_sm * s->sms};
  }
  const int shape =
      choose_symmetric(s->sys_h.data(), 0, static_cast<int32_t>(s->sys_h.size()), c, kCount,
                       kAdjDiagCost, kAdjPairCost);
  *grid = c[shape].max_grid;
  return shape;
}

int ensure_adjoint_buffers(nb_sim* s, int32_t ncp, int32_t every) {
  AdjointState& a = s->adj;
  const size_t np = static_cast<size_t>(s->n_pad);
  // Each buffer by itself: a call that failed between two of them leaves the first.
  while (static_cast<int32_t>(a.ckpt_pos.size()) < ncp) {
    float* p = nullptr;
    NB_TRY(dev_alloc(&p, 4 * np));
    a.ckpt_pos.push_back(p);
  }
  while (static_cast<int32_t>(a.ckpt_vel.size()) < ncp) {
    float4* v = nullptr;
    NB_TRY(dev_alloc(&v, np));
    a.ckpt_vel.push_back(v);
  }
  if (!a.vel) NB_TRY(dev_alloc(&a.vel, np));
  while (static_cast<int32_t>(a.seg_pos.size()) < every - 1) {
    float* p = nullptr;
    NB_TRY(dev_alloc(&p, 4 * np));
    // Padding particles must sit far away with zero mass in every buffer the
    // force kernel reads; the kernel writes only real particles.
    NB_CUDA(launch_fill_padding(p, a.vel, s->n_pad, s->stream));
    a.seg_pos.push_back(p);
  }
  for (float4** p : {&a.lam_x, &a.lam_v, &a.mu, &a.tmp})
    if (!*p) NB_TRY(dev_alloc(p, np));
  if (a.wl.grid == 0) {
    const int32_t nsys = static_cast<int32_t>(s->sys_h.size());
    bool pays = false;
    // A pair of the adjoint is twice the work of a force's, so the line lies lower (us per
    // backward step, symmetric / direct): 512 particles 6.9 / 3.7, 1,024 7.1 / 4.7, 2,048
    // 9.0 / 8.0, 2,432 10.2 / 9.0, 3,000 11.9 / 12.6; ensembles of 2.4e6 pairs in
    // 1,091 i-tiles of 8 10.0 / 8.8, in 3,129 10.2 / 9.4, 3.6e6 in 414 10.5 / 9.5 and in 4,830
    // 11.0 / 11.4, 4.1e6 in 1,808 10.6 / 10.8, 7e6 in 1,720 12.4 / 16.1.
    a.shape = choose_direct(s->sys_h.data(), nsys, s->sms,
                            nsys == 1 ? kAdjDirectPairs : kAdjDirectEnsemblePairs,
                            kAdjDirectTiles, &pays);
    a.direct = pays;
    if (a.direct) return plan_direct(s, direct_shape(a.shape).r, 0, nsys, &a.wl);
    int grid = 0;
    a.shape = adjoint_shape_for(s, &grid);
    const KernelShape sh = adjoint_shape(a.shape);
    // In as few bands as the device has room for, down to one i-tile's row.
    for (int64_t values = kSymScratchBytes / kSymRowBytes;;) {
      const SymPlanHost h = plan_symmetric(s->sys_h.data(), 0, nsys, sh.bi(), sh.bj, grid, values,
                                           kAdjDiagCost, kAdjPairCost);
      const int st = upload_symmetric(s, h, sh, 1, kAdjDiagCost, kAdjPairCost, &a.wl);
      if (st != NB_ERR_OUT_OF_MEMORY || values == 0) {
        NB_TRY(st);
        break;
      }
      values = std::min(values, h.row_values) / 2;
    }
  }
  return NB_OK;
}

}  // namespace

extern "C" {

int nb_sim_diagnostics(nb_sim* s, int32_t system, nb_diagnostics* out) {
  if (!s || !out) return set_error(NB_ERR_INVALID_ARGUMENT, "NULL argument");
  DeviceGuard dg_(s->device);
  const int32_t nsys = static_cast<int32_t>(s->sys_h.size());
  if (system < -1 || system >= nsys) return set_error(NB_ERR_INVALID_ARGUMENT, "bad system");
  if (!s->diag_out_d) NB_TRY(dev_alloc(&s->diag_out_d, 10));
  const int32_t first = system < 0 ? 0 : system;
  const int32_t count = system < 0 ? nsys : 1;
  NB_CUDA(launch_diagnostics(s->pos_d[s->cur], s->vel_d, s->sys_d, s->sys_h.data(), first, count,
                             s->params.dist_eps, s->params.G, s->per_pair_mass, s->sms,
                             s->diag_out_d, s->diag, s->stream));
  double h[10];
  NB_CUDA(cudaMemcpyAsync(h, s->diag_out_d, sizeof(h), cudaMemcpyDeviceToHost, s->stream));
  NB_CUDA(cudaStreamSynchronize(s->stream));
  out->potential = h[0];
  out->kinetic = h[1];
  out->total = h[0] + h[1];
  out->momentum[0] = h[3];
  out->momentum[1] = h[4];
  out->momentum[2] = h[5];
  out->angular_momentum[0] = h[6];
  out->angular_momentum[1] = h[7];
  out->angular_momentum[2] = h[8];
  out->mass = h[9];
  return NB_OK;
}

int nb_sim_fp64_accelerations(nb_sim* s, const uint64_t* rows, uint64_t count, double* ax,
                              double* ay, double* az) {
  if (!s || (count && (!rows || !ax || !ay || !az)))
    return set_error(NB_ERR_INVALID_ARGUMENT, "NULL argument");
  DeviceGuard dg_(s->device);
  if (count == 0) return NB_OK;
  if (count > (1u << 24)) return set_error(NB_ERR_INVALID_ARGUMENT, "too many rows");
  std::vector<int64_t> g(count);
  std::vector<int32_t> sy(count);
  for (uint64_t k = 0; k < count; ++k) {
    if (rows[k] >= s->n_real) return set_error(NB_ERR_INVALID_ARGUMENT, "row out of range");
    const auto it = std::upper_bound(s->user_offset.begin(), s->user_offset.end(),
                                     static_cast<int64_t>(rows[k]));
    const int32_t sys = static_cast<int32_t>(it - s->user_offset.begin()) - 1;
    sy[k] = sys;
    g[k] = s->sys_h[sys].offset + (static_cast<int64_t>(rows[k]) - s->user_offset[sys]);
  }
  int64_t* g_d = nullptr;
  int32_t* s_d = nullptr;
  double* o_d = nullptr;
  int st = dev_alloc(&g_d, count);
  if (st == NB_OK) st = dev_alloc(&s_d, count);
  if (st == NB_OK) st = dev_alloc(&o_d, 3 * count);
  std::vector<double> o(3 * count);
  cudaError_t e = cudaSuccess;
  if (st == NB_OK) {
    e = cudaMemcpyAsync(g_d, g.data(), count * sizeof(int64_t), cudaMemcpyHostToDevice, s->stream);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(s_d, sy.data(), count * sizeof(int32_t), cudaMemcpyHostToDevice,
                          s->stream);
    if (e == cudaSuccess)
      e = launch_fp64_rows(s->pos_d[s->cur], s->sys_d, g_d, s_d, static_cast<int64_t>(count),
                           s->params.dist_eps, s->params.G, s->per_pair_mass, o_d, s->stream);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(o.data(), o_d, 3 * count * sizeof(double), cudaMemcpyDeviceToHost,
                          s->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
  }
  dev_free(g_d);
  dev_free(s_d);
  dev_free(o_d);
  if (st != NB_OK) return st;
  if (e != cudaSuccess) return cuda_error(e, "fp64 accelerations");
  for (uint64_t k = 0; k < count; ++k) {
    ax[k] = o[3 * k];
    ay[k] = o[3 * k + 1];
    az[k] = o[3 * k + 2];
  }
  return NB_OK;
}

int nb_sim_adjoint_forward(nb_sim* s, int32_t T, int32_t checkpoint_every) {
  if (!s) return set_error(NB_ERR_INVALID_ARGUMENT, "sim is NULL");
  DeviceGuard dg_(s->device);
  if (T < 1 || checkpoint_every < 1)
    return set_error(NB_ERR_INVALID_ARGUMENT, "T and checkpoint_every must be >= 1");
  if (s->params.calc_method != NB_BRANCH)
    return set_error(NB_ERR_STATE, "the adjoint is defined for the BRANCH method only");
  for (const SystemDesc& d : s->sys_h)
    if (d.shard_first != 0 || d.shard_count != 0)
      return set_error(NB_ERR_STATE, "the adjoint needs the whole system, not a shard");
  const int32_t every = std::min(checkpoint_every, T);
  const int32_t ncp = (T + every - 1) / every;
  s->adj.valid = false;
  NB_TRY(ensure_adjoint_buffers(s, ncp, every));
  const size_t np = static_cast<size_t>(s->n_pad);
  for (int32_t k = 0; k < ncp; ++k) {
    NB_CUDA(cudaMemcpyAsync(s->adj.ckpt_pos[k], s->pos_d[s->cur], 4 * np * sizeof(float),
                            cudaMemcpyDeviceToDevice, s->stream));
    NB_CUDA(cudaMemcpyAsync(s->adj.ckpt_vel[k], s->vel_d, np * sizeof(float4),
                            cudaMemcpyDeviceToDevice, s->stream));
    NB_TRY(nb_sim_advance(s, std::min(every, T - k * every)));
  }
  NB_TRY(nb_sim_synchronize(s));
  s->adj.T = T;
  s->adj.every = every;
  s->adj.count = ncp;
  s->adj.valid = true;
  return NB_OK;
}

// The backward sweep, stream-ordered on the simulation's stream, from device
// gradients dL/dx_T, dL/dv_T (n x 3, xyz-interleaved; gv_T may be NULL) to device
// dL/dx_0, dL/dv_0.  The outputs may alias the inputs: the inputs are read first.
static int adjoint_backward_stream(nb_sim* s, const float* gx_T, const float* gv_T, float* gx_0,
                                   float* gv_0) {
  AdjointState& a = s->adj;
  const size_t n = s->n_real;
  const size_t np = static_cast<size_t>(s->n_pad);
  NB_CUDA(cudaMemsetAsync(a.lam_x, 0, np * sizeof(float4), s->stream));
  NB_CUDA(cudaMemsetAsync(a.lam_v, 0, np * sizeof(float4), s->stream));
  NB_CUDA(cudaMemsetAsync(a.tmp, 0, np * sizeof(float4), s->stream));
  NB_CUDA(cudaMemsetAsync(a.mu, 0, np * sizeof(float4), s->stream));
  NB_CUDA(launch_unpack_vec3(gx_T, n, s->map_d, a.lam_x, s->stream));
  if (gv_T) NB_CUDA(launch_unpack_vec3(gv_T, n, s->map_d, a.lam_v, s->stream));
  const float dt = s->params.dt;
  for (int32_t k = a.count - 1; k >= 0; --k) {
    const int32_t t0 = k * a.every;
    const int32_t L = std::min(a.every, a.T - t0);
    // Recompute the positions x_{t0+1} .. x_{t0+L-1} from the checkpoint's, which are
    // x_{t0}; each step of the recomputation replaces the velocities.
    if (L > 1)
      NB_CUDA(cudaMemcpyAsync(a.vel, a.ckpt_vel[k], np * sizeof(float4), cudaMemcpyDeviceToDevice,
                              s->stream));
    auto at = [&](int32_t t) { return t == 0 ? a.ckpt_pos[k] : a.seg_pos[t - 1]; };
    for (int32_t t = 0; t + 1 < L; ++t) {
      ForceArgs fa = base_args(s);
      fa.pos = at(t);
      fa.pos_next = at(t + 1);
      fa.vel = a.vel;
      NB_TRY(launch_with(s, fa, s->wl));
    }
    // Reverse through the segment.
    for (int32_t t = L - 1; t >= 0; --t) {
      AdjointArgs aa{};
      aa.pos = at(t);
      aa.lam_x = a.lam_x;
      aa.lam_v = a.lam_v;
      aa.lam_x_out = a.tmp;
      aa.lam_v_out = a.mu;  // second buffer pair: (tmp, mu) <- (lam_x, lam_v)
      aa.sys = s->sys_d;
      aa.tiles = a.wl.sym_tiles;
      aa.rows = s->rows_d;
      aa.plane = a.wl.row_values;
      aa.carry = s->carry_d;
      aa.partials = s->partials_d;
      aa.eps2 = s->params.dist_eps;
      aa.dt = dt;
      aa.damping = s->params.damping;
      aa.mask_self = s->mask_self;
      if (a.direct)
        NB_CUDA(launch_adjoint_direct(a.shape, s->per_pair_mass, aa, a.wl.direct_tiles,
                                      a.wl.direct_sys, a.wl.grid, s->stream));
      for (const SymBand& b : a.wl.bands) {
        aa.segs = a.wl.sym_segs + b.seg0;
        aa.tile0 = b.tile0;
        aa.tile1 = b.tile1;
        NB_CUDA(launch_adjoint(a.shape, s->per_pair_mass, aa, b.grid, s->stream));
        NB_CUDA(launch_adjoint_add(aa, b.end - b.tile0, adjoint_shape(a.shape).bi(), a.wl.terms,
                                   s->stream));
      }
      std::swap(a.lam_x, a.tmp);
      std::swap(a.lam_v, a.mu);
    }
  }
  NB_CUDA(launch_pack_vec3(a.lam_x, n, s->map_d, gx_0, s->stream));
  NB_CUDA(launch_pack_vec3(a.lam_v, n, s->map_d, gv_0, s->stream));
  return NB_OK;
}

int nb_sim_adjoint_backward(nb_sim* s, const float* gx_T, const float* gv_T, float* gx_0,
                            float* gv_0) {
  if (!s || !gx_T || !gx_0 || !gv_0) return set_error(NB_ERR_INVALID_ARGUMENT, "NULL argument");
  DeviceGuard dg_(s->device);
  AdjointState& a = s->adj;
  if (!a.valid) return set_error(NB_ERR_STATE, "call nb_sim_adjoint_forward first");
  NB_TRY(ensure_staging(s));
  const size_t n = s->n_real;
  float* stage = s->staging_d;  // 7n floats: the two n x 3 arrays in and out
  NB_CUDA(cudaMemcpyAsync(stage, gx_T, 3 * n * sizeof(float), cudaMemcpyHostToDevice, s->stream));
  if (gv_T)
    NB_CUDA(cudaMemcpyAsync(stage + 3 * n, gv_T, 3 * n * sizeof(float), cudaMemcpyHostToDevice,
                            s->stream));
  NB_TRY(adjoint_backward_stream(s, stage, gv_T ? stage + 3 * n : nullptr, stage, stage + 3 * n));
  NB_CUDA(cudaMemcpyAsync(gx_0, stage, 3 * n * sizeof(float), cudaMemcpyDeviceToHost, s->stream));
  NB_CUDA(cudaMemcpyAsync(gv_0, stage + 3 * n, 3 * n * sizeof(float), cudaMemcpyDeviceToHost,
                          s->stream));
  NB_CUDA(cudaStreamSynchronize(s->stream));
  return check_error_word(s);
}

int nb_sim_adjoint_backward_device(nb_sim* s, const float* gx_T_device, const float* gv_T_device,
                                   float* gx_0_device, float* gv_0_device) {
  if (!s || !gx_T_device || !gx_0_device || !gv_0_device)
    return set_error(NB_ERR_INVALID_ARGUMENT, "NULL argument");
  DeviceGuard dg_(s->device);
  if (!s->adj.valid) return set_error(NB_ERR_STATE, "call nb_sim_adjoint_forward first");
  return adjoint_backward_stream(s, gx_T_device, gv_T_device, gx_0_device, gv_0_device);
}

}  // extern "C"
