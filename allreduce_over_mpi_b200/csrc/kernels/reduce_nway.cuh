// Argument block of the single-GPU n-way reduction kernels (reduce_nway.cu, reduce_nway_wide.cu,
// reduce_nway_shift.cu, reduce_nway_scaled.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../api/ft_types.h"

namespace ftk {

// One launch covers a whole vector: the body in 32- or 16-byte vectors, and the elements in front of and behind it
// (the edges) one by one in a CTA of their own (the last one), so that neither a ragged length nor a slice that starts
// off a vector boundary costs a second launch or takes the rest of the vector off the vector loads.
struct NwayArgs {
  const void* src[FT_MAX_FANIN];  // start of the body in every source
  void* dst;
  unsigned long long nvec;    // body length, in the kernel's vectors
  unsigned long long nbody;   // ... and in scalar units (see ScalarOp)
  int n;
  uint16_t head, edge;        // scalar units in front of the body; in front of and behind it together
  uint8_t shift[FT_MAX_FANIN];  // shifted kernels: bytes by which source k's body lies behind a 16-byte (realign: 32-byte) boundary
};

// Kernels for pointers that agree modulo 32 (reduce_nway_wide.cu).  `code` selects a configuration (0: by size;
// see launch_cfg there); returns cudaErrorInvalidValue when (policy, fan-in, code) has no instantiation.
cudaError_t launch_wide(int pol, const NwayArgs& a, int code, int sms, cudaStream_t st);
// Kernels for pointers that do not agree modulo 32 (reduce_nway_shift.cu); `realign`: the sources do, the result does not.
cudaError_t launch_shift(int pol, const NwayArgs& a, bool realign, cudaStream_t st);
// out = scale * sum over `len` elements of whole vectors in `a` (reduce_nway_scaled.cu).
cudaError_t launch_scaled(bool in_bf16, bool out_bf16, const NwayArgs& a, unsigned long long len, float scale, int sms, cudaStream_t st);

#ifdef __CUDACC__
// The edges of the vector, by the CTA the launch adds for them (less than 160 bytes: one or two units a thread).
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
