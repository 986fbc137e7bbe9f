// Prefix reductions straight from and to pinned host memory: out[j] = in[0] (op) ... (op) in[fanin[j] - 1].
//
// PCIe bounds it.  One kernel reads every input over the link once and posts every result back as it arises, so both
// directions of the link are busy from the first microseconds on, there are no device buffers to pass through, and a
// call is one launch.  The copy engines have to finish a chunk of inputs before its sums can start, and pay a few
// microseconds per copy: 8 fp32 inputs of 1 Mi elements and 4 results took 1002 us through them in one chunk and take
// 684 us here (33.6 MB in at 49 GB/s, 16.8 MB out at the same time; the copy engines alone, both ways at once without
// a reduction: 720 us); 20 000 elements 59 -> 20 us, 1000 elements of two inputs 20 -> 4 us.
//
// A handful of CTAs fills the link, so the rest of the GPU stays free: 1 MB of loads in flight.  Where the host memory is
// near, 256 KB do (8 CTAs with eight inputs, 681 us), but from a farther socket they reach 41 GB/s only (809 us; 683 us
// with 32 CTAs on either box).  Many more make reads and writes collide (592 CTAs 771 us).
#include "pdl.cuh"
#include "vec.cuh"
#include "host_prefix.h"

namespace ftk {

template <int POL>
__global__ void __launch_bounds__(256) host_prefix_kernel(const __grid_constant__ HostPrefixArgs a) {
  using P = typename PolById<POL>::type;
  pdl_begin();
  const uint64_t nvec = a.bytes / 16, items = nvec + a.bytes % 16 / a.es;   // whole vectors, then single elements
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < items; i += stride) {
    const bool full = i < nvec;
    const uint64_t off = full ? i * 16 : nvec * 16 + (i - nvec) * a.es;
    typename P::Acc acc;
    constexpr int G = 8;
    for (int k0 = 0; k0 < a.n_in; k0 += G) {
      uint4 v[G];
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (k0 + g < a.n_in) {
          const unsigned char* p = (const unsigned char*)a.in[k0 + g] + off;
          v[g] = full ? ld_stream(p) : ld_element(p, a.es);
        }
#pragma unroll
      for (int g = 0; g < G; ++g) {
        if (k0 + g >= a.n_in) break;
        if (k0 + g == 0) P::init(acc, v[g]);
        else P::add(acc, v[g]);
        for (int j = a.first[k0 + g]; j < a.first[k0 + g + 1]; ++j) {   // the results that end with this input
          unsigned char* q = (unsigned char*)a.out[j] + off;
          if (full) st_vec(q, P::fin(acc));
          else st_element(q, P::fin(acc), a.es);
        }
      }
    }
  }
}

template <int POL>
static cudaError_t launch_t(const HostPrefixArgs& a, cudaStream_t st) {
  const uint64_t items = a.bytes / 16 + a.bytes % 16 / a.es;
  // 32 CTAs of 256 threads with eight inputs, more with fewer
  uint64_t grid = 256 / (a.n_in < 8 ? a.n_in : 8), want = (items + 255) / 256;
  if (grid > want) grid = want;
  return launch_pdl(host_prefix_kernel<POL>, (unsigned)grid, 256, 0, st, a);
}

cudaError_t launch_host_prefix(int pol, const HostPrefixArgs& a, cudaStream_t st) {
  switch (pol) {
    case POL_ADD8: return launch_t<POL_ADD8>(a, st);
    case POL_ADD16: return launch_t<POL_ADD16>(a, st);
    case POL_ADD32: return launch_t<POL_ADD32>(a, st);
    case POL_ADD64: return launch_t<POL_ADD64>(a, st);
    case POL_OR: return launch_t<POL_OR>(a, st);
    case POL_AND: return launch_t<POL_AND>(a, st);
    case POL_F32: return launch_t<POL_F32>(a, st);
    case POL_F64: return launch_t<POL_F64>(a, st);
    case POL_BF16: return launch_t<POL_BF16>(a, st);
    case POL_F16: return launch_t<POL_F16>(a, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace ftk
