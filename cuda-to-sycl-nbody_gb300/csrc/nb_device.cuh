// Device helpers shared by the kernels.
#pragma once

#include <cuda_runtime.h>

#include "nb_internal.hpp"

namespace nbg {

// Programmatic dependent launch: a kernel launched with launch_dependent may start
// while its predecessor in the stream still runs.  pdl_wait returns when the
// predecessor has finished and its writes are visible; pdl_trigger lets the successor
// start (once every CTA has called it or left).  Kernels trigger near their end: a
// successor whose CTAs become resident earlier finds free places only on the SMs that
// have little or no work, and its CTAs crowd there (reference order, 16,384 particles on
// 128 CTAs: 192 us per step triggered at the start, 153 near the end; symmetric, 2,048
// particles: 8.5 and 7.4).
__device__ __forceinline__ void pdl_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void pdl_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... Params, class... Args>
cudaError_t launch_dependent(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem,
                             cudaStream_t stream, Args... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Integrate (or write accelerations for) one real particle at (xi, yi, zi) of velocity v.
__device__ __forceinline__ void finish_particle(const ForceArgs& a, const SystemDesc& sd,
                                                int64_t gi, float fx, float fy, float fz,
                                                float xi, float yi, float zi, float4 v) {
  const float g = sd.gscale;
  if (a.accel_out != nullptr) {
    a.accel_out[gi] = make_float4(fx * g, fy * g, fz * g, 0.f);
    return;
  }
  // v = v * damping; v += (F * dt) * G   (simulator.cu:214-216)
  v.x = fmaf(fx * a.dt, g, v.x * a.damping);
  v.y = fmaf(fy * a.dt, g, v.y * a.damping);
  v.z = fmaf(fz * a.dt, g, v.z * a.damping);
  a.vel[gi] = v;
  // x' = x + v * dt   (simulator.cu:223-228)
  a.pos_next[pair_index(gi, 0)] = fmaf(v.x, a.dt, xi);
  a.pos_next[pair_index(gi, 1)] = fmaf(v.y, a.dt, yi);
  a.pos_next[pair_index(gi, 2)] = fmaf(v.z, a.dt, zi);
  a.pos_next[pair_index(gi, 3)] = a.pos[pair_index(gi, 3)];
}
__device__ __forceinline__ void finish_particle(const ForceArgs& a, const SystemDesc& sd,
                                                int64_t gi, float fx, float fy, float fz,
                                                float xi, float yi, float zi) {
  const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
  finish_particle(a, sd, gi, fx, fy, fz, xi, yi, zi, a.accel_out ? none : a.vel[gi]);
}

}  // namespace nbg
