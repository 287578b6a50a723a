// The adding pass of the symmetric force step, with the integrate epilogue.
#include <cuda_runtime.h>

#include "nb_device.cuh"
#include "nb_kernels.hpp"
#include "symmetric_add.cuh"

namespace nbg {
namespace {

struct EarlyForce {
  const ForceArgs& f;
  SystemDesc sd;
  float x, y, z;
  __device__ void lists(int sys) { sd = f.sys[sys]; }
  __device__ void state(int64_t g) {
    if (f.accel_out != nullptr) return;
    x = f.pos[pair_index(g, 0)];
    y = f.pos[pair_index(g, 1)];
    z = f.pos[pair_index(g, 2)];
  }
};

template <int kLanes, int kGroups, bool kComp>
__global__ void __launch_bounds__(kLanes * kGroups) symmetric_add_kernel(const SymArgs a, int bi) {
  const AddTerms t{a.tiles, a.rows, a.plane, a.carry, a.f.partials, a.tile0, a.tile1};
  EarlyForce e{a.f, {}, 0.f, 0.f, 0.f};
  AddResult r;
  if (add_terms<kLanes, kGroups, kComp>(t, bi, e, r))
    finish_particle(a.f, e.sd, r.g, r.x, r.y, r.z, e.x, e.y, e.z);
}

template <int kLanes, int kGroups>
cudaError_t add_one(bool compensated, const SymArgs& a, int tiles, int bi, cudaStream_t stream) {
  return launch_dependent(compensated ? symmetric_add_kernel<kLanes, kGroups, true>
                                      : symmetric_add_kernel<kLanes, kGroups, false>,
                          add_grid<kLanes>(tiles, bi), kLanes * kGroups, 0, stream, a, bi);
}

}  // namespace

cudaError_t launch_symmetric_add(bool compensated, const SymArgs& a, int tiles, int bi,
                                 float terms, cudaStream_t stream) {
  const AddShape sh = add_shape(static_cast<int64_t>(tiles) * bi, terms);
  return sh.groups == 1   ? add_one<64, 1>(compensated, a, tiles, bi, stream)
         : sh.groups == 2 ? add_one<64, 2>(compensated, a, tiles, bi, stream)
         : sh.groups == 4 ? add_one<32, 4>(compensated, a, tiles, bi, stream)
                          : add_one<32, 8>(compensated, a, tiles, bi, stream);
}

}  // namespace nbg
