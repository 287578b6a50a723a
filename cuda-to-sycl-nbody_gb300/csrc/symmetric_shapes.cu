// Compiled shapes of the symmetric force kernel (symmetric_kernel.cuh): warps per CTA,
// i-pairs per thread.
#include <atomic>

#include "symmetric_kernel.cuh"

namespace nbg {
namespace {

template <int NW, int P, int U, bool C, bool M, bool X>
cudaError_t smem_opt_in() {
  static std::atomic<uint64_t> opted{0};  // once per device ordinal (>= 64: every call)
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = dev >= 0 && dev < 64 ? uint64_t{1} << dev : 0;
  if (bit != 0 && (opted.load(std::memory_order_acquire) & bit) != 0) return cudaSuccess;
  e = cudaFuncSetAttribute(symmetric_kernel<NW, P, U, C, M, X>,
                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                           symmetric_smem<NW, P, C>());
  if (e == cudaSuccess && bit != 0) opted.fetch_or(bit, std::memory_order_release);
  return e;
}

template <int NW, int P, int U, bool C, bool M, bool X>
cudaError_t launch_one(const SymArgs& a, int grid, cudaStream_t st) {
  const cudaError_t e = smem_opt_in<NW, P, U, C, M, X>();
  if (e != cudaSuccess) return e;
  return launch_dependent(symmetric_kernel<NW, P, U, C, M, X>, dim3(grid), NW * 32,
                          symmetric_smem<NW, P, C>(), st, a);
}

template <int NW, int P, int U, bool C, bool M, bool X>
cudaError_t occ_one(int* blocks) {
  const cudaError_t e = smem_opt_in<NW, P, U, C, M, X>();
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(
      blocks, symmetric_kernel<NW, P, U, C, M, X>, NW * 32, symmetric_smem<NW, P, C>());
}

struct SymEntry {
  int warps, pairs, bj;
  cudaError_t (*launch[2][2])(const SymArgs&, int, cudaStream_t);  // [compensated][mass]
  cudaError_t (*occ[2][2])(int*);
  cudaError_t (*launch_xyzm)(const SymArgs&, int, cudaStream_t);   // plain, own masses
  cudaError_t (*occ_xyzm)(int*);
};

#define NBG_SYM(NW, P, U)                                                                         \
  {NW, P, kSymBJ<NW>,                                                                             \
   {{launch_one<NW, P, U, NW == 8, false, false>, launch_one<NW, P, U, false, true, false>},      \
    {launch_one<NW, P, U, true, false, false>, launch_one<NW, P, U, true, true, false>}},         \
   {{occ_one<NW, P, U, NW == 8, false, false>, occ_one<NW, P, U, false, true, false>},            \
    {occ_one<NW, P, U, true, false, false>, occ_one<NW, P, U, true, true, false>}},               \
   launch_one<NW, P, U, false, true, true>, occ_one<NW, P, U, false, true, true>}

const SymEntry kShapes[] = {NBG_SYM(8, 8, 2), NBG_SYM(1, 8, 2), NBG_SYM(1, 4, 4),
                            NBG_SYM(1, 1, 4)};

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
