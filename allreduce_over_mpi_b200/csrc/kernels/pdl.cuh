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
//   * lets its successor be set up before it ends, once each of its CTAs has asked for that (pdl_next(), where its loads are
//     issued) or has left, and
//   * has its first CTAs fetch their sources into L2 while they wait in pdl_begin() (l2_ahead()): 12 MB, what HBM delivers in
//     that time.  More, or all CTAs, cost L2 what they give HBM.
// us a call, calls in a row on fresh tensors, without and with both: fp32 x2 of 5 M 10.1 -> 8.7, x3 views 12.9 -> 11.4, x8 of 2.5 M
// 14.5 -> 12.9, of 6.5 M 34.3 -> 33.2; bf16 x8 of 4 M 12.0 -> 10.5, its views 11.1 -> 10.1, averaged 11.9 -> 10.4; eight ranks'
// all-reduce of 6 MB 16.4 -> 15.4, of 25 MB 63.5 -> 62.5.  The request alone gives nothing, and only a call of this library in
// front of another gives anything: behind a kernel that does not ask, and in front of one, a call is as fast as without.
// Smaller calls neither ask nor fetch: in L2 the waiting CTAs hold slots that the running kernel's own next CTAs want, and the
// fetches are in the way (fp32 x3 of 1 M in L2 2.2 us, 2.7 with both; x4 of 1 M with the request at the start 4.0 instead of
// 2.3).
//
// Only the last CTAs ask: those before them have left by the time it matters, and asking costs.  It is a message of each CTA
// to what starts CTAs, and where data lies in L2 a call of two sources is bound by just that (8000 CTAs in 8 us).  So
// 16 of 128 threads an SM ask, as many as the chip holds; from 100 MB on, which no longer lie in L2, 20, since CTAs that wait
// for HBM leave in less order (fp32 x2 of 20 M 33.9 us if all ask, 34.4 with 16 an SM, 34.0 with 20; of 40 M 68.7, 68.1, 67.8).
// One set of tensors over and over, which L2 holds whole up to 100 MB, us with neither / all asking / this: fp32 x2 of 5 M 5.0 /
// 6.0 / 5.6, of 8 M 7.6 / 9.2 / 7.9, uint8 x2 of 30 M 7.3 / 8.6 / 7.5, fp32 x3 of 5 M 5.9 / 6.2 / 6.2, bf16 x8 of 4 M 5.7 / 5.9 /
// 5.9, fp32 x8 of 2.5 M 6.3 / 7.0 / 7.0, x2 averaged to bf16 of 10 M 7.9 / 11.1 / 8.6.  What is left is the fetching.  It is paid as
// well, 0.1 to 0.8 us, where kernels that do not ask have just written all the sources and left them in L2.  A sum in
// place to which one fresh tensor is added gains (x2 of 5 M 7.4 -> 7.1).
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

// This CTA asks: once all have, or have left, the successor is set up.  It still waits in its pdl_begin().
__device__ __forceinline__ void pdl_next(bool ask) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t@q griddepcontrol.launch_dependents;\n\t}" ::"r"((uint32_t)ask) : "memory");
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
