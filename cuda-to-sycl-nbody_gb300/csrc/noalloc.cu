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
// array, kScratchBytes (13 MiB) long; larger systems run in bands of i-tiles that take
// turns in it (20,000 particles 223 us per call with the tuned kernel and its list
// uploaded on every call, 146 now).  Small systems run the direct kernel, which needs
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
#include "symmetric_plan.hpp"

namespace nbg {

namespace {

constexpr int64_t kNaMaxParticles = 1 << 18;  // 262,144
constexpr int kNaMaxDevices = 64;
constexpr size_t kScratchBytes = 13u << 20;

// Candidate shapes by index of the symmetric kernel (i-tiles of 4,096, 256 and 64
// particles), largest first, and choose_symmetric's rates for them.  512-particle
// i-tiles would need 10 MB for the parts and as much for the rows at their sizes.
constexpr int kNaShapes[] = {0, 2, 3};
constexpr double kNaRates[][2] = {{1.0, 6.0}, {0.86, 0.8}, {0.617, 0.0}};
constexpr int kNaCount = 3;

// A table of fixed size with the vector operations the planner uses; what does not fit
// is dropped and remembered.
template <class T, int N>
struct FixedTable {
  T data[N];
  int n = 0;
  bool full = false;
  void push_back(const T& v) {
    if (n < N)
      data[n++] = v;
    else
      full = true;
  }
  void clear() {
    n = 0;
    full = false;
  }
  void assign(size_t count, const T& v) {
    clear();
    for (size_t k = 0; k < count; ++k) push_back(v);
  }
  void erase(T* from, T* to) {
    (void)to;  // the planner erases the tail
    n = static_cast<int>(from - data);
  }
  size_t size() const { return n; }
  bool empty() const { return n == 0; }
  T& operator[](size_t i) { return data[i]; }
  const T& operator[](size_t i) const { return data[i]; }
  T& back() { return data[n - 1]; }
  T* begin() { return data; }
  T* end() { return data + n; }
  const T* begin() const { return data; }
  const T* end() const { return data + n; }
};

// Bounds: at most 64 i-tiles of 4,096 particles, each a band of its own on up to 152
// CTAs; the smaller shapes are chosen for at most about 128 i-tiles, in a few bands on
// at most kNaMaxGrid CTAs.  A plan that passes them is refused for the next shape.
constexpr int kNaMaxGrid = 2432;
constexpr int kNaMaxTiles = 512;
constexpr int kNaMaxSegments = 10240;
constexpr int kNaMaxBands = 64;

struct FixedPlan {
  FixedTable<SymSegment, kNaMaxSegments> segs;
  FixedTable<int32_t, kNaMaxSegments + kNaMaxBands + 1> seg_begin;
  FixedTable<SymTile, kNaMaxTiles> tiles;
  FixedTable<int32_t, 2> sys_tile0;
  FixedTable<SymBand, kNaMaxBands> bands;
  int64_t row_values = 0;
  int32_t slots = 0;
  int32_t split_tiles = 0;
  void clear() {
    segs.clear();
    seg_begin.clear();
    tiles.clear();
    sys_tile0.clear();
    bands.clear();
    row_values = 0;
    slots = split_tiles = 0;
  }
  bool fits() const {
    return !segs.full && !seg_begin.full && !tiles.full && !bands.full;
  }
};

}  // namespace

// The scratch array.  In host code this name is only a host-side stand-in:
// host code must take the device address with cudaGetSymbolAddress (below).
static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

namespace {

constexpr size_t align256(size_t x) { return (x + 255) / 256 * 256; }

// Where the current plan's parts lie in the scratch; `copy`: of the caller's positions,
// 0 where they are read in place.
struct Layout {
  size_t sys = 0, segs = 256, tiles = 0, partials = 0, rows = 0, copy = 0;
};

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
  Layout at;
};

std::mutex g_na_mutex;            // guards the host-side tables below
DeviceSetup g_na_setup[kNaMaxDevices];
FixedPlan g_na_plan;
FixedTable<SymSegment, kNaMaxSegments> g_na_linked;

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

// Plan shape k for the system: as large bands as the scratch holds, on the shape's
// full grid, or a smaller one where even one i-tile's row and parts are too much.  False
// if it does not fit.
bool na_plan(const SystemDesc& sd, const DeviceSetup& d, int k, bool copied, Layout* at) {
  const KernelShape sh = symmetric_shape(kNaShapes[k]);
  const int64_t tiles = (sd.n + sh.bi() - 1) / sh.bi();
  if (tiles > kNaMaxTiles) return false;
  const int64_t part = static_cast<int64_t>(sh.bi()) * sizeof(float4);  // bytes of one slot
  const int64_t longest = std::max<int64_t>(0, sd.npad - sh.bi());      // values of the first row
  const int64_t copy = copied ? static_cast<int64_t>(sd.n) * 16 : 0;
  int64_t grid = d.grid[k];
  for (int64_t per = tiles; grid >= 1;) {
    // A plan of `per` i-tiles per band: its row values at most, and whether the parts and
    // the rows of the largest band fit beside its tables.
    const int64_t values = std::max<int64_t>(1, per * longest);
    g_na_plan.clear();
    plan_symmetric_into(&sd, 0, 1, sh.bi(), sh.bj, static_cast<int32_t>(grid), values, per,
                        kSymDiagCost, kSymPairCost, g_na_plan);
    if (g_na_plan.fits()) {
      at->tiles = align256(at->segs + g_na_plan.segs.size() * sizeof(SymSegment));
      at->partials = align256(at->tiles + g_na_plan.tiles.size() * sizeof(SymTile));
      at->rows = align256(at->partials + g_na_plan.slots * static_cast<size_t>(part));
      const size_t end =
          align256(at->rows + 3 * sizeof(float) * static_cast<size_t>(g_na_plan.row_values));
      at->copy = copied ? end : 0;
      if (end + static_cast<size_t>(copy) <= kScratchBytes) {
        g_na_linked.n = static_cast<int>(g_na_plan.segs.size());
        link_segments_into(g_na_plan, sh.bi() / sh.bj, sh.threads == 32 ? 4 * d.sms : 0,
                           kSymDiagCost, kSymPairCost, g_na_linked);
        return true;
      }
    }
    if (per > 1)
      per = (per + 1) / 2;
    else
      grid -= 8;
  }
  return false;
}

// Plan n particles and put the plan into the scratch.
int na_upload(DeviceSetup& d, uint64_t n, float G, bool copied, cudaStream_t st) {
  d.n = 0;  // nothing until all of it is there
  SystemDesc sd{};
  sd.offset = 0;
  sd.n = static_cast<int32_t>(n);
  sd.npad = (sd.n + kPadQuantum - 1) / kPadQuantum * kPadQuantum;
  sd.gscale = G;  // per-pair masses: each pair term carries m_j
  SymCandidate c[kNaCount];
  for (int k = 0; k < kNaCount; ++k)
    c[k] = SymCandidate{symmetric_shape(kNaShapes[k]), kNaRates[k][0], kNaRates[k][1], d.grid[k]};
  int k = choose_symmetric(&sd, 0, 1, c, kNaCount, kSymDiagCost, kSymPairCost);
  Layout at;
  if (!na_plan(sd, d, k, copied, &at) && !na_plan(sd, d, k = 0, copied, &at))
    return set_error(NB_ERR_INVALID_ARGUMENT, "work list exceeds the no-allocation scratch");
  unsigned char* base = d.scratch;
  // Host sources are pageable: each copy has read them before it returns.
  NB_CUDA(cudaMemcpyAsync(base + at.segs, g_na_linked.data, g_na_linked.n * sizeof(SymSegment),
                          cudaMemcpyHostToDevice, st));
  NB_CUDA(cudaMemcpyAsync(base + at.tiles, g_na_plan.tiles.data,
                          g_na_plan.tiles.size() * sizeof(SymTile), cudaMemcpyHostToDevice, st));
  NB_CUDA(cudaMemcpyAsync(base + at.sys, &sd, sizeof(sd), cudaMemcpyHostToDevice, st));
  d.G = G;
  d.copied = copied;
  d.shape = kNaShapes[k];
  d.plane = g_na_plan.row_values;
  d.terms = terms_per_particle(g_na_plan, symmetric_shape(kNaShapes[k]).bi());
  d.nbands = static_cast<int>(g_na_plan.bands.size());
  for (int b = 0; b < d.nbands; ++b) d.bands[b] = g_na_plan.bands[b];
  d.at = at;
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
                     "13 MiB device scratch); use nb_sim_accelerations for more");
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
  if (d.n != n || d.G != G || d.copied != copied) NB_TRY(na_upload(d, n, G, copied, st));
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
