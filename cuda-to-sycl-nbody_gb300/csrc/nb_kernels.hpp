// Host-callable launchers of the device kernels (implemented in the .cu files).
#pragma once

#include <cuda_runtime.h>

#include "nb_internal.hpp"

namespace nbg {

// ---- force + integrate (force_kernel.cu) ----------------------------------------
int num_force_configs();
KernelShape force_config_shape(int index);
// Launch the tuned force kernel of shape `index`.  `compensated` selects the Kahan
// accumulator, `per_pair_mass` multiplies each pair term by m_j, `live` the variant
// that skips the register slots past the end of a system (its work list is planned
// with live-slot weights, live_slots_pay in worklist.hpp).
cudaError_t launch_force(int index, bool compensated, bool per_pair_mass, bool live,
                         const ForceArgs& a, int grid, cudaStream_t stream);
cudaError_t force_blocks_per_sm(int index, bool compensated, bool per_pair_mass, bool live,
                                int* blocks);

// ---- symmetric force step (symmetric_kernel.cuh, symmetric_add.cu) -------------------
struct SymSegment;
struct SymTile;
struct SymArgs {
  ForceArgs f;               // pos, pos_next, vel, accel_out, sys, partials, eps2, dt, ...
  const SymSegment* segs;    // the band's, linked (link_segments)
  const SymTile* tiles;      // every i-tile
  float* rows;               // [3][plane] j-side sums
  int64_t plane;
  float4* carry;             // running sums between bands, [n_pad] (compensated: [n_pad][2])
  int32_t tile0, tile1;      // the band's i-tiles
};
int num_symmetric_shapes();
KernelShape symmetric_shape(int index);  // threads, i-particles per thread, j-tile, 0 stages
// Compiled with compensated sums only for these masses (the faster kernel).
bool symmetric_always_compensates(int index, bool per_pair_mass);
cudaError_t symmetric_blocks_per_sm(int index, bool compensated, bool per_pair_mass, int* blocks);
cudaError_t launch_symmetric(int index, bool compensated, bool per_pair_mass, const SymArgs& a,
                             int grid, cudaStream_t stream);
// The same over positions in the caller's layout, a float4 (x, y, z, m) per particle
// (plain sums, per-particle masses; accelerations only).
cudaError_t symmetric_xyzm_blocks_per_sm(int index, int* blocks);
cudaError_t launch_symmetric_xyzm(int index, const SymArgs& a, int grid, cudaStream_t stream);
// Add the rows and parts of the band's i-tiles and integrate; `tiles` i-tiles from a.tile0,
// `terms` rows and parts per particle on average.
cudaError_t launch_symmetric_add(bool compensated, const SymArgs& a, int tiles, int bi,
                                 float terms, cudaStream_t stream);

// ---- direct force step of small systems (direct_kernel.cu) ----------------------------
struct DirectArgs {
  ForceArgs f;        // pos, pos_next, vel, accel_out, sys, eps2, dt, ...
  const int2* tiles;  // (system, i-tile) of each CTA; NULL: CTA b is i-tile b of `sys`
  int32_t sys;
  int32_t n;          // launch_direct_xyzm: particles, and what their sums are times
  float gscale;
};
int num_direct_shapes();
// Threads, i-particles of a CTA (every thread holds them all), j-particles per pass, 1.
KernelShape direct_shape(int index);
// The shape for `count` systems; *pays: they have at most max_pairs pairs and max_tiles
// i-tiles of 8 particles.  Up to these the direct kernel beats the symmetric one:
constexpr double kDirectPairs = 2.2e7;          // one system
constexpr double kDirectEnsemblePairs = 1.2e7;  // several
constexpr int64_t kDirectTiles = 6000;
constexpr double kAdjDirectPairs = 6.5e6;  // the same of the adjoint
constexpr double kAdjDirectEnsemblePairs = 3.5e6;
constexpr int64_t kAdjDirectTiles = 3000;
int choose_direct(const SystemDesc* sys, int32_t count, int sms, double max_pairs,
                  int64_t max_tiles, bool* pays);
cudaError_t launch_direct(int index, bool compensated, bool per_pair_mass, const DirectArgs& a,
                          int grid, cudaStream_t stream);
// Positions as for launch_symmetric_xyzm, one system.
cudaError_t launch_direct_xyzm(int index, const DirectArgs& a, int grid, cudaStream_t stream);

// ---- compatibility kernel (aux_kernels.cu) ------------------------------------------
// The reference's PREDICATED variant as shipped, one thread per i-particle over one
// system (simulator.cu:186-229 with the (i == id) mask of :208-209).
cudaError_t launch_predicated(const ForceArgs& a, const SystemDesc& sd, int32_t sys_index,
                              cudaStream_t stream);

// ---- reference-order force + integrate (reference_order_kernel.cu) -------------------
// particle_interaction<BRANCH> with the reference's per-particle summation order
// and arithmetic (bit-identical results on the same GPU), equal masses per system;
// `predicated` selects particle_interaction<PREDICATED>'s pair term instead.
// Shapes are indexed largest i-tile first.  The kernel walks a stream-K work list
// (ForceArgs segs / seg_begin / fix) of reference_order_shape(index) tiles; split
// i-tiles hand their running sums over through `partials` and `counters`.  `dup` is
// the duplicated j-layout of a.pos (2 float4 per padded particle) written by
// launch_reference_order_dup, for the shapes that need it.  With split i-tiles the
// launch is cooperative: grid <= blocks per SM x SMs.
int reference_order_num_shapes();
KernelShape reference_order_shape(int index);  // threads, i-particles per thread, j-tile, stages
cudaError_t reference_order_blocks_per_sm(int index, bool predicated, int* blocks);
cudaError_t launch_reference_order_dup(const float* pos, int64_t n_pad_total, float4* dup,
                                       cudaStream_t stream);
cudaError_t launch_reference_order(int index, bool predicated, const ForceArgs& a,
                                   const float4* dup, int grid, bool split,
                                   cudaStream_t stream);
bool reference_order_needs_dup(int index);

// ---- measured FP32 throughput (peak_probe.cu) ----------------------------------------
// Time `repeats` launches (after one warm-up) of an FFMA2 loop over sms x blocks_per_sm
// CTAs; `scratch` holds sms * blocks_per_sm * fp32_peak_threads() float2.
cudaError_t measure_fp32_peak(int sms, float2* scratch, int blocks_per_sm, int iters,
                              int repeats, cudaStream_t stream, double* tflops, float* best_ms);
int fp32_peak_threads();

// ---- state movement (aux_kernels.cu) ------------------------------------------------
// Device SoA staging <-> simulation layout.  `map` holds, for each of the n real
// particles in user order, its padded device index.
cudaError_t launch_unpack_state(const float* soa /*[7][n]: x y z vx vy vz m*/, int64_t n,
                                const int64_t* map, float* pos, float4* vel, bool with_mass,
                                cudaStream_t stream);
cudaError_t launch_pack_state(const float* pos, const float4* vel, int64_t n, const int64_t* map,
                              float* soa /*[6][n]*/, cudaStream_t stream);
// The device error word into pinned host memory.
cudaError_t launch_read_error(const int32_t* err, int32_t* host, cudaStream_t stream);
cudaError_t launch_pack_accel(const float4* acc, int64_t n, const int64_t* map,
                              float* soa /*[3][n]*/, cudaStream_t stream);
cudaError_t launch_export(const float* pos, const float4* vel, int64_t n, const int64_t* map,
                          float4* pos_out, float4* vel_out, cudaStream_t stream);
cudaError_t launch_fill_padding(float* pos, float4* vel, int64_t n_pad_total, cudaStream_t stream);

// ---- FP64 diagnostics (diag_kernels.cu) ---------------------------------------------
struct DiagScratch {
  double* partial = nullptr;  // moments, potential parts, tile lists, range flag
  int64_t cap = 0;            // doubles
  int32_t first_sys = 0, num_sys = 0;  // the systems the tile lists are for
  int64_t nfp64 = 0, nsplit = 0;       // tiles of the FP64 and of the split kernel
  int32_t spans = 1, fp64_spans = 1;   // parts their j-tiles are cut into
};
cudaError_t launch_diagnostics(const float* pos, const float4* vel, const SystemDesc* sys_d,
                               const SystemDesc* sys_h, int32_t first_sys, int32_t num_sys,
                               float eps2, float G, bool per_pair_mass, int sms, double* out10,
                               DiagScratch& scratch, cudaStream_t stream);
cudaError_t launch_fp64_rows(const float* pos, const SystemDesc* sys_d, const int64_t* rows_dev,
                             const int32_t* row_sys_dev, int64_t count, float eps2, float G,
                             bool per_pair_mass, double* out3, cudaStream_t stream);

// ---- adjoint (adjoint_kernel.cu) ----------------------------------------------------
struct AdjointArgs {
  const float* pos;       // pair layout, positions x_t at which the Jacobian is taken
  const float4* lam_x;    // [n_pad] lam_x' (cotangent of x')
  const float4* lam_v;    // [n_pad] lam_v' (cotangent of v')
  float4* lam_x_out;      // [n_pad] lam_x = lam_x' + dt * G * J^T mu, mu = lam_v' + dt lam_x'
  float4* lam_v_out;      // [n_pad] lam_v = damping * mu
  const SystemDesc* sys;
  const SymSegment* segs;  // work list, i-tiles, row scratch and parts: as in SymArgs
  const SymTile* tiles;
  float* rows;
  int64_t plane;
  float4* carry;
  float4* partials;
  int32_t tile0, tile1;
  float eps2;
  float dt;
  float damping;
  int32_t mask_self;
};
int num_adjoint_shapes();
KernelShape adjoint_shape(int index);  // threads, i-particles per thread, j-tile, 0 stages
cudaError_t adjoint_blocks_per_sm(int index, bool per_pair_mass, int* blocks);
cudaError_t launch_adjoint(int index, bool per_pair_mass, const AdjointArgs& a, int grid,
                           cudaStream_t stream);
// Small systems: shape `index` of choose_direct, its i-tiles as in DirectArgs.
cudaError_t launch_adjoint_direct(int index, bool per_pair_mass, const AdjointArgs& a,
                                  const int2* tiles, int sys, int grid, cudaStream_t stream);
// Add the rows and parts of the band's i-tiles and write lam_x_out and lam_v_out.
cudaError_t launch_adjoint_add(const AdjointArgs& a, int tiles, int bi, float terms,
                               cudaStream_t stream);
// n x 3 interleaved (user order) <-> padded float4.
cudaError_t launch_unpack_vec3(const float* in, int64_t n, const int64_t* map, float4* out,
                               cudaStream_t stream);
cudaError_t launch_pack_vec3(const float4* in, int64_t n, const int64_t* map, float* out,
                             cudaStream_t stream);

// ---- initial conditions on the device (initgen.cu) ------------------------------------
// kind 1: thin disks, 2: Plummer (needs raw [6 * total] and mean [6 * nsys] FP64
// scratch), 3: two-disk collisions.  first_d[k] = first user index of system k.
cudaError_t launch_generate(int kind, float* pos, float4* vel, const SystemDesc* sys_d,
                            const int64_t* first_d, int32_t nsys, int64_t total, uint64_t seed,
                            double eps, double* raw, double* mean, cudaStream_t stream);

}  // namespace nbg
