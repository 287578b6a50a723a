// Accelerations for callers that cannot allocate GPU memory.
//
// Some callers of a physics step own every byte of GPU memory themselves: a
// render engine or plugin host that hands out pre-sized buffers from its own
// pools, a real-time loop that must not hit cudaMalloc's implicit device-wide
// synchronization in the middle of a frame, or a process that reserves its whole
// memory budget up front.  nb_accelerations_noalloc serves them.  They pass
// their own input and output buffers; the library allocates nothing on the
// device and, on success, nothing on the host.
//
// The work the symmetric force kernel needs beyond its input and output -- the work
// list, the partial sums and the rows of j-side sums -- lives in one file-scope device
// array, kNaScratchBytes long; larger systems run in bands of i-tiles that take turns in
// it (20,000 particles 216 us per call with the tuned kernel and its list uploaded on
// every call, 126 now).  Small systems run the direct kernel, which needs
// none of it.  Every GPU that loads this module keeps that array
// until the process exits.  All calls share it and it keeps the last call's contents:
// the work list stays for the next call of the same size, unless a call fails on the way.
// Two calls whose work overlapped on the GPU would race on it, so each call holds a
// process-wide lock until its stream has drained: the calls of one process run one after
// another, whatever streams and threads they come from.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <mutex>

#include "nb_internal.hpp"
#include "nb_kernels.hpp"
#include "nb_runtime.hpp"
#include "nbody_gb300.h"
#include "noalloc_plan.hpp"

namespace nbg {

namespace {

constexpr int kNaMaxDevices = 64;

}  // namespace

// The scratch array.  In host code this name is only a host-side stand-in:
// host code must take the device address with cudaGetSymbolAddress (below).
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaScratchBytes];

namespace {

struct DeviceSetup {
  bool ready = false;
  unsigned char* scratch = nullptr;  // device address of g_noalloc_scratch
  int grid[kNaCount] = {};           // largest grid of each shape
  int sms = 0;
  // The plan in the scratch: for `n` particles; n = 0: none.
  uint64_t n = 0;
  float G = 0.f;
  bool copied = false;
  int shape = 0;
  int64_t plane = 0;
  float terms = 0.f;
  int nbands = 0;
  SymBand bands[kNaMaxBands];
  NaLayout at;
};

std::mutex g_na_mutex;            // guards the host-side tables below
DeviceSetup g_na_setup[kNaMaxDevices];
NaPlan g_na_plan;
alignas(256) unsigned char g_na_image[kNaMaxImage];

// What a call does when it ends early, by an error after its first enqueue: nothing may be
// left in flight when the lock goes, and the plan may not be in the scratch.  (A call on a
// stream that is being captured fails so: its uploads were recorded, not made.)
struct Drain {
  DeviceSetup& d;
  cudaStream_t stream;
  bool done = false;
  ~Drain() {
    if (done) return;
    d.n = 0;
    cudaStreamSynchronize(stream);
    cudaGetLastError();
  }
};

// Once per device, with that device current: the scratch's device address and the
// shapes' grids.
int na_setup(int dev) {
  DeviceSetup& d = g_na_setup[dev];
  if (d.ready) return NB_OK;
  int sms = 0;
  cudaDeviceProp prop;
  NB_TRY(check_device(&sms, &prop));
  void* p = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e != cudaSuccess) return cuda_error(e, "cudaGetSymbolAddress(no-allocation scratch)");
  for (int k = 0; k < kNaCount; ++k) {
    int blocks = 0;
    NB_CUDA(symmetric_xyzm_blocks_per_sm(kNaShapes[k], &blocks));
    d.grid[k] = std::max(1, std::min(blocks * sms, kNaMaxGrid));
  }
  d.sms = sms;
  d.scratch = static_cast<unsigned char*>(p);
  d.ready = true;
  return NB_OK;
}

// The system record in the scratch, which alone depends on G.
int na_upload_system(DeviceSetup& d, uint64_t n, float G, cudaStream_t st) {
  const SystemDesc sd = na_system(n, G);
  // The host source is pageable: the copy has read it before it returns.
  NB_CUDA(cudaMemcpyAsync(d.scratch + d.at.sys, &sd, sizeof(sd), cudaMemcpyHostToDevice, st));
  d.G = G;
  return NB_OK;
}

// Plan n particles and put the plan into the scratch, in one copy.  A call of another size
// than the last takes that much longer (us per call, the same size / sizes in turn: 5,000
// particles 24 / 51, 20,000 126 / 158, 25,000 193 / 253; planned by trial, with 128-bit
// divisions and four copies, 84, 296 and 538; the tuned kernel with its list uploaded on
// every call 55, 216 and 284).
int na_upload(DeviceSetup& d, uint64_t n, float G, bool copied, cudaStream_t st) {
  d.n = 0;  // nothing until all of it is there
  SymCandidate c[kNaCount];
  for (int k = 0; k < kNaCount; ++k)
    c[k] = SymCandidate{symmetric_shape(kNaShapes[k]), kNaRates[k][0], kNaRates[k][1], d.grid[k]};
  const int k = na_plan(na_system(n, G), c, d.sms, copied, g_na_plan, g_na_image);
  if (k < 0)
    return set_error(NB_ERR_INVALID_ARGUMENT, "work list exceeds the no-allocation scratch");
  // As na_upload_system's.
  NB_CUDA(cudaMemcpyAsync(d.scratch, g_na_image, g_na_plan.at.partials, cudaMemcpyHostToDevice,
                          st));
  d.G = G;
  d.copied = copied;
  d.shape = kNaShapes[k];
  d.plane = g_na_plan.row_values;
  d.terms = terms_per_particle(g_na_plan, c[k].shape.bi());
  d.nbands = static_cast<int>(g_na_plan.bands.size());
  for (int b = 0; b < d.nbands; ++b) d.bands[b] = g_na_plan.bands[b];
  d.at = g_na_plan.at;
  d.n = n;
  return NB_OK;
}

}  // namespace

}  // namespace nbg

using namespace nbg;

extern "C" int nb_accelerations_noalloc(const float* pos_xyzm_device, uint64_t n, float G,
                                        float dist_eps, float* accel_xyzw_device,
                                        void* stream) {
  if (!pos_xyzm_device || !accel_xyzw_device)
    return set_error(NB_ERR_INVALID_ARGUMENT, "NULL device buffer");
  if ((reinterpret_cast<uintptr_t>(pos_xyzm_device) & 15) ||
      (reinterpret_cast<uintptr_t>(accel_xyzw_device) & 15))
    return set_error(NB_ERR_INVALID_ARGUMENT, "device buffers must be 16-byte aligned");
  if (n == 0 || n > static_cast<uint64_t>(kNaMaxParticles))
    return set_error(NB_ERR_INVALID_ARGUMENT,
                     "nb_accelerations_noalloc takes 1 to 262144 particles (its fixed "
                     "18 MiB device scratch); use nb_sim_accelerations for more");
  if (!std::isfinite(G) || !std::isfinite(dist_eps) || dist_eps < 0.f)
    return set_error(NB_ERR_INVALID_ARGUMENT, "G and dist_eps must be finite, dist_eps >= 0");
  int dev = 0;
  NB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNaMaxDevices) return set_error(NB_ERR_NO_DEVICE, "device ordinal");
  cudaStream_t st = static_cast<cudaStream_t>(stream);

  std::lock_guard<std::mutex> lock(g_na_mutex);
  NB_TRY(na_setup(dev));
  DeviceSetup& d = g_na_setup[dev];
  // A caller may pass one buffer for both: bands would read positions that earlier bands
  // have replaced, so overlapping buffers are copied first.
  const uintptr_t in = reinterpret_cast<uintptr_t>(pos_xyzm_device);
  const uintptr_t out = reinterpret_cast<uintptr_t>(accel_xyzw_device);
  const bool copied = in < out + 16 * n && out < in + 16 * n;
  SystemDesc whole{};
  whole.n = static_cast<int32_t>(n);
  bool direct = false;
  const int small = choose_direct(&whole, 1, d.sms, kDirectPairs, kDirectTiles, &direct);
  Drain drain{d, st};
  if (direct) {
    // One launch without a plan.
    DirectArgs a{};
    a.f.pos = pos_xyzm_device;
    if (copied) {
      d.n = 0;  // the copy takes the plan's place
      NB_CUDA(cudaMemcpyAsync(d.scratch, pos_xyzm_device, 16 * n, cudaMemcpyDeviceToDevice, st));
      a.f.pos = reinterpret_cast<const float*>(d.scratch);
    }
    a.f.accel_out = reinterpret_cast<float4*>(accel_xyzw_device);
    a.f.eps2 = dist_eps;
    a.f.mask_self = dist_eps * dist_eps * dist_eps >= FLT_MIN ? 0 : 1;
    a.n = whole.n;
    a.gscale = G;
    const int r = direct_shape(small).r;
    NB_CUDA(launch_direct_xyzm(small, a, (whole.n + r - 1) / r, st));
    NB_CUDA(cudaStreamSynchronize(st));
    drain.done = true;
    return NB_OK;
  }
  if (d.n != n || d.copied != copied)
    NB_TRY(na_upload(d, n, G, copied, st));
  else if (d.G != G)
    NB_TRY(na_upload_system(d, n, G, st));
  unsigned char* base = d.scratch;
  SymArgs a{};
  a.f.pos = pos_xyzm_device;
  if (copied) {
    NB_CUDA(cudaMemcpyAsync(base + d.at.copy, pos_xyzm_device, 16 * n, cudaMemcpyDeviceToDevice,
                            st));
    a.f.pos = reinterpret_cast<const float*>(base + d.at.copy);
  }
  a.f.accel_out = reinterpret_cast<float4*>(accel_xyzw_device);
  a.f.sys = reinterpret_cast<const SystemDesc*>(base + d.at.sys);
  a.f.partials = reinterpret_cast<float4*>(base + d.at.partials);
  a.f.eps2 = dist_eps;
  const float e3 = dist_eps * dist_eps * dist_eps;
  a.f.mask_self = (e3 >= FLT_MIN) ? 0 : 1;
  a.tiles = reinterpret_cast<const SymTile*>(base + d.at.tiles);
  a.rows = reinterpret_cast<float*>(base + d.at.rows);
  a.plane = d.plane;
  a.carry = a.f.accel_out;  // a particle's place is free until its last band
  const int bi = symmetric_shape(d.shape).bi();
  for (int b = 0; b < d.nbands; ++b) {
    const SymBand& band = d.bands[b];
    a.segs = reinterpret_cast<const SymSegment*>(base + d.at.segs) + band.seg0;
    a.tile0 = band.tile0;
    a.tile1 = band.tile1;
    NB_CUDA(launch_symmetric_xyzm(d.shape, a, band.grid, st));
    NB_CUDA(launch_symmetric_add(false, a, band.end - band.tile0, bi, d.terms, st));
  }
  NB_CUDA(cudaStreamSynchronize(st));
  drain.done = true;
  return NB_OK;
}
