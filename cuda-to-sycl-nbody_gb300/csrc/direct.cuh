// The tree of the direct kernels (direct_kernel.cu, adjoint_kernel.cu).
#pragma once

#include <cuda_runtime.h>

namespace nbg {

// The warp's sums of R particles that every lane holds a part of: halve the particles a
// lane holds while it adds its partner's, then add over the lanes that hold the same one.
// Particle lane / (32 / R) is then in t[0].
template <int R>
__device__ __forceinline__ void warp_sums(float (&t)[R][3]) {
  const int lane = threadIdx.x & 31;
  int cnt = R;
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) {
    const bool upper = (lane & m) != 0;
    if (cnt > 1) {
      cnt /= 2;
#pragma unroll
      for (int k = 0; k < R / 2; ++k)
        if (k < cnt)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const float give = upper ? t[k][c] : t[k + cnt][c];
            const float keep = upper ? t[k + cnt][c] : t[k][c];
            t[k][c] = keep + __shfl_xor_sync(0xffffffffu, give, m);
          }
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) t[0][c] += __shfl_xor_sync(0xffffffffu, t[0][c], m);
    }
  }
}

}  // namespace nbg
