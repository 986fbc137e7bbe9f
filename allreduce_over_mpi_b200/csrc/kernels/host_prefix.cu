// Prefix reductions straight from and to pinned host memory: out[j] = in[0] (op) ... (op) in[fanin[j] - 1].
//
// PCIe bounds it.  One kernel reads every input over the link once and posts every result back as it arises, so both
// directions of the link are busy from the first microseconds on, there are no device buffers to pass through, and a
// call is one launch.  The copy engines have to finish a chunk of inputs before its sums can start, and pay a few
// microseconds per copy: 8 fp32 inputs of 1 Mi elements and 4 results took 1002 us through them in one chunk and take
// 681 us here (33.6 MB in at 49 GB/s, 16.8 MB out at the same time; reading alone 657 us, the copy engines both ways at
// once without a reduction 720 us).
//
// Each SM that takes part costs a call a few tenths of a microsecond, so a CTA has 1024 threads and a call at most six of
// them, with the same number of turns each.  Two inputs of 16 KB took 4.8 us with four CTAs of 256 threads and take 3.9 with
// one; of 64 KB 8.8 -> 6.9, of 256 KB 16.9 -> 14.8 (16.1 with two vectors a thread); eight of 8 KB 5.8 -> 4.8, of 64 KB
// 17.3 -> 15.2, of 1 MB 173.2 -> 171.0.
// The second CTA costs 1.1 us, so up to 32 KB of two to four inputs one CTA takes two vectors a thread: two inputs of 20 KB 4.8
// us (5.4 with two CTAs of 1024, 5.4 with five of 256), of 32 KB 5.2 (5.9 and 5.9), four of 24 KB 6.4 (6.9 and 7.0).  More inputs
// would need twice the registers.
// Where the host memory is near, 100 KB of loads in flight fill the link; from a farther socket 256 KB reach 41 GB/s only
// (49 with 1 MB).  So from three turns up a thread takes two vectors at a time of two or three inputs: 384 KB in flight at
// least.  Many CTAs make reads and writes collide (592 of 256 threads 771 us).
//
// The elements behind the last whole vector go a thread each, in a warp of their own: sharing one with vectors their loads
// waited for those one by one (eight inputs of 1027 fp32 elements 11.5 us, 4.0 now).
#include "pdl.cuh"
#include "vec.cuh"
#include "host_prefix.h"

namespace ftk {

constexpr int kHostThreads = 1024, kHostCtas = 6;

// 16 bytes, or one element in the low bytes of the vector, at p; without a branch, so that all loads of a thread are issued
// back to back.
__device__ __forceinline__ void host_load(const unsigned char* p, bool ok, uint4& v) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\t@q ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n\t}"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p), "r"((uint32_t)ok) : "memory");
}
// Items of a call: its whole vectors, counted up to a multiple of 32, then the single elements behind them.
__host__ __device__ __forceinline__ uint64_t host_vectors(uint64_t bytes) { return (bytes / 16 + 31) / 32 * 32; }
template <class T>
__host__ __device__ __forceinline__ uint64_t host_items(uint64_t bytes) { return host_vectors(bytes) + bytes % 16 / sizeof(T); }

// U: vectors a thread takes at a time, of 8 / U inputs; two only where all inputs are one group.
template <int POL, int U>
__global__ void __launch_bounds__(kHostThreads) host_prefix_kernel(const __grid_constant__ HostPrefixArgs a) {
  using P = typename PolById<POL>::type;
  using T = typename ScalarOp<POL>::elem;
  constexpr int G = 8 / U;
  pdl_begin();
  const uint64_t nvec = a.bytes / 16, padded = host_vectors(a.bytes), items = host_items<T>(a.bytes);
  const uint64_t stride = (uint64_t)gridDim.x * kHostThreads;
  for (uint64_t i = (uint64_t)blockIdx.x * kHostThreads + threadIdx.x; i < items; i += stride * U) {
    typename P::Acc acc;
    for (int k0 = 0; k0 < a.n_in; k0 += G) {
      uint4 v[U][G];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint64_t item = i + u * stride;
        if (item < padded) {   // all of a warp
#pragma unroll
          for (int g = 0; g < G; ++g)
            if (k0 + g < a.n_in) host_load((const unsigned char*)a.in[k0 + g] + item * 16, item < nvec, v[u][g]);
        } else if (item < items) {
#pragma unroll
          for (int g = 0; g < G; ++g)
            if (k0 + g < a.n_in) v[u][g] = ld_element((const T*)((const unsigned char*)a.in[k0 + g] + nvec * 16) + (item - padded), sizeof(T));
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint64_t item = i + u * stride;
        const bool full = item < nvec;
        if (!full && (item < padded || item >= items)) continue;
        const uint64_t off = full ? item * 16 : nvec * 16 + (item - padded) * sizeof(T);
#pragma unroll
        for (int g = 0; g < G; ++g) {
          if (k0 + g >= a.n_in) break;
          if (k0 + g == 0) P::init(acc, v[u][g]);
          else P::add(acc, v[u][g]);
          for (int j = a.first[k0 + g]; j < a.first[k0 + g + 1]; ++j) {   // the results that end with this input
            unsigned char* q = (unsigned char*)a.out[j] + off;
            if (full) st_vec(q, P::fin(acc));
            else st_element(q, P::fin(acc), sizeof(T));
          }
        }
      }
    }
  }
}

template <int POL, int U>
static cudaError_t launch_u(const HostPrefixArgs& a, cudaStream_t st) {
  // CTAs with the same number of turns each
  const uint64_t want = (host_items<typename ScalarOp<POL>::elem>(a.bytes) + kHostThreads * U - 1) / (kHostThreads * U);
  const uint64_t turns = (want + kHostCtas - 1) / kHostCtas;
  return launch_pdl(host_prefix_kernel<POL, U>, (unsigned)((want + turns - 1) / turns), kHostThreads, 0, st, a);
}
template <int POL>
static cudaError_t launch_t(const HostPrefixArgs& a, cudaStream_t st) {
  constexpr uint64_t turn = kHostThreads * 16;   // bytes of a vector that a CTA takes at a time
  const bool one_cta = a.n_in <= 4 && a.bytes > turn && a.bytes <= 2 * turn;   // instead of two
  return one_cta || (a.n_in <= 3 && a.bytes > 3 * kHostCtas * turn) ? launch_u<POL, 2>(a, st) : launch_u<POL, 1>(a, st);
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
