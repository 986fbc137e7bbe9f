// The single-GPU n-way reduction kernels as reduce_nway.cu launches them (reduce_nway_wide.cu, reduce_nway_shift.cu,
// reduce_nway_scaled.cu), and the part they share.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../api/ft_types.h"
#include "nway_layout.h"

namespace ftk {

// Kernels for pointers that agree modulo 32 (reduce_nway_wide.cu).  `code` selects a configuration (0: by size;
// see launch_cfg there); returns cudaErrorInvalidValue when (policy, fan-in, code) has no instantiation.
cudaError_t launch_wide(int pol, const NwayArgs& a, int code, int sms, cudaStream_t st);
// Kernels for pointers that do not agree modulo 32 (reduce_nway_shift.cu); `realign`: the sources do, the result does not.
cudaError_t launch_shift(int pol, const NwayArgs& a, bool realign, cudaStream_t st);
// out = a.scale * sum over `len` elements of whole vectors in `a` (reduce_nway_scaled.cu).
cudaError_t launch_scaled(bool in_bf16, bool out_bf16, const NwayArgs& a, unsigned long long len, int sms, cudaStream_t st);

#ifdef __CUDACC__
// The edges of the vector, by the CTA the launch adds for them, or the first one (less than 160 bytes: one or two units a thread).
template <int POL, template <int> class Scalar>
__device__ __forceinline__ void reduce_edges(const NwayArgs& a) {
  using S = Scalar<POL>;
  using T = typename S::elem;
  for (int e = threadIdx.x; e < a.edge; e += blockDim.x) {
    const long long i = e < a.head ? (long long)e - a.head : (long long)(a.nbody + (e - a.head));
    typename S::acc acc{};
    for (int k0 = 0; k0 < a.n; k0 += 8) {   // eight loads in flight, like the body: a small vector waits for this CTA
      T v[8];
#pragma unroll
      for (int g = 0; g < 8; ++g)
        if (k0 + g < a.n) v[g] = ((const T*)a.src[k0 + g])[i];
#pragma unroll
      for (int g = 0; g < 8; ++g)
        if (k0 + g < a.n) acc = k0 + g == 0 ? S::load(v[g]) : S::comb(acc, S::load(v[g]));
    }
    ((T*)a.dst)[i] = S::store(acc);
  }
}
#endif

}  // namespace ftk
