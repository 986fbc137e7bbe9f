// Launching: what every launch does afterwards, and programmatic dependent launch for the short kernels.
//
// Between two kernels of a stream lie about 2 us in which nothing runs: the second one is set up only when the first
// has completed.  A kernel launched with launch_pdl() is set up when the CTAs of the one before it have left; it calls
// pdl_begin() before it touches memory, which returns when that one has completed and its writes are visible, so
// stream order holds as before.  Every kernel launched this way calls pdl_begin().
// fp32 x2 of 64 Ki elements, launches back to back: 4.1 -> 2.0 us each; bf16 x8 of 4 Mi: 14.4 -> 11.7.
//
// Where data comes from HBM, some 1.7 us of the memory's time were still lost between two calls: the last CTAs of one drain,
// the first of the next wait for their data.  So a call that moves 50 MB or more
//   * lets its successor be set up once all its CTAs have issued their loads (pdl_next()), and
//   * has its first CTAs fetch their sources into L2 while they wait in pdl_begin() (l2_ahead()): 12 MB, what HBM delivers in
//     that time.  More, or all CTAs, cost L2 what they give HBM.
// us a call, calls in a row on fresh tensors, without and with both: fp32 x2 of 5 M 10.1 -> 8.8, x3 views 12.9 -> 11.4, x8 of 2.5 M
// 14.5 -> 12.9, of 6.5 M 34.3 -> 33.2; bf16 x8 of 4 M 12.0 -> 10.6, its views 11.2 -> 10.1, averaged 12.0 -> 10.6; eight ranks'
// all-reduce of 6 MB 16.6 -> 15.3, of 25 MB 63.5 -> 62.2.  The request alone gives nothing.
// Smaller calls neither ask nor fetch: in L2 the waiting CTAs hold slots that the running kernel's own next CTAs want, and the
// fetches are in the way (fp32 x3 of 1 M in L2 2.2 us, 2.7 with both; x4 of 1 M with the request at the start 4.0 instead of
// 2.3).  Above 50 MB that is so only for calls in a row on one set of tensors that L2 holds whole, up to 100 MB (x2 of 5 M 5.0 ->
// 6.0, x3 5.9 -> 6.4, x8 of 2.5 M 6.2 -> 7.0); with two sets in turn x2 has 7.1 -> 7.4, x3 12.7 -> 11.4, x8 14.5 -> 13.0.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

extern "C" void ft_count_launch(uint64_t n);   // see ft_launch_count()

namespace ftk {

// Behind every launch, with what it answered.  Counts it if it went out; if not, takes the error away from the runtime,
// which would hand it to the next caller that asks whether ITS launch went well.
inline cudaError_t launched(cudaError_t e) {
  if (e == cudaSuccess) ft_count_launch(1);
  else cudaGetLastError();
  return e;
}

__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The successor may be set up from here on; it still waits in its pdl_begin().
__device__ __forceinline__ void pdl_next(uint32_t early) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t@q griddepcontrol.launch_dependents;\n\t}" ::"r"(early) : "memory");
}
// Fetch the line at p into L2.  In front of pdl_begin() too: L2 is where all SMs meet, so a line that the kernel before
// this one still writes is the written one afterwards.
__device__ __forceinline__ void l2_ahead(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p) : "memory"); }

// What the host pays for a launch depends on the size of the kernel's parameters, but not as one would think: 1.62 us with
// 24 or 32 bytes modulo 64, 1.85 to 2.15 with any other number (8 to 1280 in steps of 8; driver 580.159, PDL attribute).
constexpr bool cheap_to_launch(size_t bytes) { return bytes % 64 == 24 || bytes % 64 == 32; }

template <class Params>
cudaError_t launch_pdl(void (*kernel)(Params), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, const std::remove_cv_t<Params>& args) {
  static_assert(cheap_to_launch(sizeof(Params)), "fill the parameters up");
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return launched(cudaLaunchKernelEx(&cfg, kernel, args));
}

}  // namespace ftk
