// Argument block of host_prefix_kernel (host_prefix.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../api/ft_types.h"

namespace ftk {

struct HostPrefixArgs {
  const void* in[FT_MAX_FANIN];     // device addresses of pinned host memory, 16-byte aligned
  void* out[FT_MAX_FANIN];          // ordered by fan-in
  uint8_t first[FT_MAX_FANIN + 1];  // results first[k] .. first[k + 1] - 1 end with input k
  uint64_t bytes;                   // of each vector
  int n_in;
  uint64_t fill[4];                 // to a size that is cheap to launch with (pdl.cuh)
};

cudaError_t launch_host_prefix(int pol, const HostPrefixArgs& a, cudaStream_t st);

}  // namespace ftk
