// Launching: what every launch does afterwards, and programmatic dependent launch for the short kernels.
//
// Between two kernels of a stream lie about 2 us in which nothing runs: the second one is set up only when the first
// has completed.  A kernel launched with launch_pdl() is set up when the CTAs of the one before it have left; it calls
// pdl_begin() before it touches memory, which returns when that one has completed and its writes are visible, so
// stream order holds as before.  Every kernel launched this way calls pdl_begin().
// fp32 x2 of 64 Ki elements, launches back to back: 4.1 -> 2.0 us each; bf16 x8 of 4 Mi: 14.4 -> 11.7.
//
// No kernel here asks for its successor earlier (griddepcontrol.launch_dependents): waiting CTAs then hold registers
// and slots that the running kernel's own next CTAs want.  fp32 x4 of 1 M: 4.0 us with the request at the start, 2.6
// with it behind the loads, 2.3 without.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

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

template <class... Params, class... Args>
cudaError_t launch_pdl(void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, const Args&... args) {
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
  return launched(cudaLaunchKernelEx(&cfg, kernel, args...));
}

}  // namespace ftk
