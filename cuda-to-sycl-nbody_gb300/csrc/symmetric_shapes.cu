// Compiled shapes of the symmetric force kernel (symmetric_kernel.cuh): warps per CTA,
// i-pairs per thread, rotations per unrolled block, per sum of the j side, j-particles per
// fold of the i side.
#include <atomic>

#include "symmetric_kernel.cuh"

namespace nbg {
namespace {

template <int NW, int P, int U, int S, int F, bool C, bool M, bool X>
cudaError_t smem_opt_in() {
  static std::atomic<uint64_t> opted{0};  // once per device ordinal (>= 64: every call)
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = dev >= 0 && dev < 64 ? uint64_t{1} << dev : 0;
  if (bit != 0 && (opted.load(std::memory_order_acquire) & bit) != 0) return cudaSuccess;
  e = cudaFuncSetAttribute(symmetric_kernel<NW, P, U, S, F, C, M, X>,
                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                           symmetric_smem<NW, P, C>());
  if (e == cudaSuccess && bit != 0) opted.fetch_or(bit, std::memory_order_release);
  return e;
}

template <int NW, int P, int U, int S, int F, bool C, bool M, bool X>
cudaError_t launch_one(const SymArgs& a, int grid, cudaStream_t st) {
  const cudaError_t e = smem_opt_in<NW, P, U, S, F, C, M, X>();
  if (e != cudaSuccess) return e;
  return launch_dependent(symmetric_kernel<NW, P, U, S, F, C, M, X>, dim3(grid), NW * 32,
                          symmetric_smem<NW, P, C>(), st, a);
}

template <int NW, int P, int U, int S, int F, bool C, bool M, bool X>
cudaError_t occ_one(int* blocks) {
  const cudaError_t e = smem_opt_in<NW, P, U, S, F, C, M, X>();
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(
      blocks, symmetric_kernel<NW, P, U, S, F, C, M, X>, NW * 32, symmetric_smem<NW, P, C>());
}

struct SymEntry {
  int warps, pairs, bj;
  cudaError_t (*launch[2][2])(const SymArgs&, int, cudaStream_t);  // [compensated][mass]
  cudaError_t (*occ[2][2])(int*);
  cudaError_t (*launch_xyzm)(const SymArgs&, int, cudaStream_t);   // plain, own masses
  cudaError_t (*occ_xyzm)(int*);
};

// S and F with compensated sums; plain ones are more exact than the tuned kernel's with
// whole chunks and longer folds already (25,600 particles 3.7e-7 / 6.6e-8).
#define NBG_SYM(NW, P, U, S, F) NBG_SYM2(NW, P, U, S, F, kSymChunk, (NW == 8 ? 512 : 128))
#define NBG_SYM2(NW, P, U, S, F, S0, F0)                                                        \
  {NW, P, kSymBJ<NW>,                                                                           \
   {{launch_one<NW, P, U, S0, F0, NW == 8, false, false>,                                       \
     launch_one<NW, P, U, S0, F0, false, true, false>},                                         \
    {launch_one<NW, P, U, S, F, true, false, false>,                                            \
     launch_one<NW, P, U, S, F, true, true, false>}},                                           \
   {{occ_one<NW, P, U, S0, F0, NW == 8, false, false>,                                          \
     occ_one<NW, P, U, S0, F0, false, true, false>},                                            \
    {occ_one<NW, P, U, S, F, true, false, false>, occ_one<NW, P, U, S, F, true, true, false>}}, \
   launch_one<NW, P, U, S0, F0, false, true, true>,                                             \
   occ_one<NW, P, U, S0, F0, false, true, true>}

// How often the j-side sums (S rotations) and the i-side sums (F j-particles) start anew
// decides the error: relative RMS error of the force against 64 bits, disks and spheres
// with equal masses, 1e-8, tuned kernel / whole chunks and folds of 128 / these:
// 8,192 4.30 3.53 / 5.32 4.31 / 4.04 3.40; 12,800 4.60 4.15 / 5.29 4.65 / 4.46 4.10; 25,600
// 4.65 4.25 / 5.07 4.58 / 4.45 4.13.  They cost 4, 3 and 2 % of the time.
const SymEntry kShapes[] = {NBG_SYM(8, 8, 2, 32, 512), NBG_SYM(1, 8, 2, 8, 128),
                            NBG_SYM(1, 4, 4, 4, 64), NBG_SYM(1, 1, 4, 32, 128)};

}  // namespace

int num_symmetric_shapes() { return static_cast<int>(sizeof(kShapes) / sizeof(kShapes[0])); }

KernelShape symmetric_shape(int index) {
  const SymEntry& e = kShapes[index];
  return KernelShape{e.warps * 32, 2 * e.pairs, e.bj, 0};
}

// 8 warps with equal masses: plain sums take longer than compensated ones, whose pair loop
// ptxas schedules better (us per step, plain / compensated: 65,536 particles 977 / 954,
// 262,144 14,925 / 14,420, 1,048,576 237,354 / 229,182).  With masses of their own, and
// in the shapes of one warp, plain is as fast or faster.
bool symmetric_always_compensates(int index, bool per_pair_mass) {
  return kShapes[index].warps == 8 && !per_pair_mass;
}

cudaError_t symmetric_blocks_per_sm(int index, bool compensated, bool per_pair_mass, int* blocks) {
  return kShapes[index].occ[compensated][per_pair_mass](blocks);
}

cudaError_t launch_symmetric(int index, bool compensated, bool per_pair_mass, const SymArgs& a,
                             int grid, cudaStream_t stream) {
  return kShapes[index].launch[compensated][per_pair_mass](a, grid, stream);
}

cudaError_t symmetric_xyzm_blocks_per_sm(int index, int* blocks) {
  return kShapes[index].occ_xyzm(blocks);
}

cudaError_t launch_symmetric_xyzm(int index, const SymArgs& a, int grid, cudaStream_t stream) {
  return kShapes[index].launch_xyzm(a, grid, stream);
}

}  // namespace nbg
