// An all-reduce (or one half of it) over the copies of ALL ranks of a world that lives on one device, in one launch.
//
// Run stage by stage, the 2*4 tree over eight ranks moves 31 times a rank's bytes and takes 40 launches; the data
// itself is 16 times a rank's bytes (every input read once, every result written once), and that is what this kernel
// moves.  HBM bounds it from a few MB up, the launch below.  A thread takes 16 or 32 bytes of one block from every
// rank, eight loads in flight, evaluates the block's program (planner/world_program.hpp: the plan's own order of
// additions and roundings) in registers and stores the copies that change.  The program is looked up in the kernel's
// parameters, in chains of a few constant-cache misses before the first load (which is why the programs of up to eight ranks
// are compiled in, world_tree.cu); all its branches are uniform across a CTA.
#include <algorithm>

#include "../api/flextree.h"
#include "pdl.cuh"
#include "vec.cuh"
#include "world_dev.h"

namespace ftk {

constexpr int kWorldThreads = 128;

// Predicated accesses (no branch, so that the loads of all steps are issued back to back): V 16-byte vectors at p.
template <int V>
__device__ __forceinline__ void world_load(const unsigned char* p, bool ok, uint4 (&v)[V]) {
  if constexpr (V == 2)
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %9, 0;\n\t"
                 "@q ld.global.L1::no_allocate.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\t}"
                 : "=r"(v[0].x), "=r"(v[0].y), "=r"(v[0].z), "=r"(v[0].w), "=r"(v[1].x), "=r"(v[1].y), "=r"(v[1].z), "=r"(v[1].w)
                 : "l"(p), "r"((uint32_t)ok) : "memory");
  else
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\t"
                 "@q ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n\t}"
                 : "=r"(v[0].x), "=r"(v[0].y), "=r"(v[0].z), "=r"(v[0].w) : "l"(p), "r"((uint32_t)ok) : "memory");
}
template <int V>
__device__ __forceinline__ void world_store(unsigned char* p, bool ok, const uint4 (&v)[V]) {
  if constexpr (V == 2)
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %9, 0;\n\t@q st.global.v8.u32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n\t}"
                 ::"l"(p), "r"(v[0].x), "r"(v[0].y), "r"(v[0].z), "r"(v[0].w), "r"(v[1].x), "r"(v[1].y), "r"(v[1].z), "r"(v[1].w),
                   "r"((uint32_t)ok) : "memory");
  else
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\t@q st.global.v4.u32 [%0], {%1,%2,%3,%4};\n\t}"
                 ::"l"(p), "r"(v[0].x), "r"(v[0].y), "r"(v[0].z), "r"(v[0].w), "r"((uint32_t)ok) : "memory");
}
// blockIdx.y: the program entry.  V: 16-byte vectors per thread and rank; DEPTH: accumulators the program may put aside; G: steps whose loads are in flight together; RANKS: size
// of the parameters.  At most 128 registers, so that four CTAs of 128 threads fit an SM: with 144 and CTAs of 256 only
// one did, and the 2*4 tree over eight bf16 buckets of 25 MB took 87 us instead of 66 (6.4 TB/s).
template <int POL, int V, int DEPTH, int G, int RANKS>
__global__ void __launch_bounds__(kWorldThreads, 4) world_reduce_kernel(const __grid_constant__ WorldArgs<RANKS> a) {
  using P = typename PolById<POL>::type;
  static_assert(G <= kWorldGroup, "the parameters are filled for this many");
  const void* const* out = a.ptr + a.kSteps;
  pdl_begin();
  const int first = a.entry[blockIdx.y].first, nsteps = a.entry[blockIdx.y].nsteps;
  const uint32_t mask = (uint32_t)a.entry[blockIdx.y].mask;
  const uint64_t lo = (uint64_t)a.entry[blockIdx.y].block * a.block_bytes;
  const uint64_t end = lo + a.block_bytes < a.total_bytes ? lo + a.block_bytes : a.total_bytes;
  if (lo >= end) return;
  // whole vectors first, then the elements behind the last one, a thread each
  const uint64_t i = (uint64_t)blockIdx.x * kWorldThreads + threadIdx.x, whole = (end - lo) / (V * 16);
  const bool full = i < whole;
  const uint64_t off = lo + (full ? i * (V * 16) : whole * (V * 16) + (i - whole) * a.es);
  if (off >= end) return;
  typename P::Acc acc[V], aside[DEPTH][V];
  for (int k0 = 0; k0 < nsteps; k0 += G) {
    uint4 v[G][V];
#pragma unroll
    for (int g = 0; g < G; ++g) world_load<V>((const unsigned char*)a.ptr[first + k0 + g] + off, full && k0 + g < nsteps, v[g]);
    if (!full) {
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (k0 + g < nsteps) v[g][0] = ld_element((const unsigned char*)a.ptr[first + k0 + g] + off, a.es);
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      if (k0 + g >= nsteps) break;
      const uint32_t code = a.code[first + k0 + g];
      if (code & 1) {
#pragma unroll
        for (int h = 0; h < V; ++h) {
#pragma unroll
          for (int d = DEPTH - 1; d > 0; --d) aside[d][h] = aside[d - 1][h];
          aside[0][h] = acc[h];   // (the first step puts aside a value nothing takes back)
          P::init(acc[h], v[g][h]);
        }
      } else {
#pragma unroll
        for (int h = 0; h < V; ++h) P::add(acc[h], v[g][h]);
      }
      const int rounds = (int)(code >> 2);
      for (int r = 0; r < rounds; ++r) {
        uint4 w[V];
#pragma unroll
        for (int h = 0; h < V; ++h) w[h] = P::fin(acc[h]);
        const uint32_t to = a.store[first + k0 + g][r];
        if (to != kNoStore) {
          if (full) world_store<V>((unsigned char*)out[to] + off, true, w);
          else st_element((unsigned char*)out[to] + off, w[0], a.es);
        }
        const bool pop = r + 1 < rounds || (code & 2);
#pragma unroll
        for (int h = 0; h < V; ++h) {
          if (pop) {
            acc[h] = aside[0][h];
#pragma unroll
            for (int d = 0; d + 1 < DEPTH; ++d) aside[d][h] = aside[d + 1][h];
            P::add(acc[h], w[h]);
          } else {
            P::init(acc[h], w[h]);
          }
        }
      }
    }
  }
  uint4 w[V];
#pragma unroll
  for (int h = 0; h < V; ++h) w[h] = a.entry[blockIdx.y].scaled ? P::fins(acc[h], a.scale) : P::fin(acc[h]);
#pragma unroll
  for (int r = 0; r < RANKS; ++r) world_store<V>((unsigned char*)out[r] + off, full && (mask >> r & 1), w);
  if (!full)
    for (int r = 0; r < RANKS; ++r)
      if (mask >> r & 1) st_element((unsigned char*)out[r] + off, w[0], a.es);
}

template <int POL, int V, int DEPTH, int G, int RANKS>
static cudaError_t launch_t(const WorldArgs<RANKS>& a, int entries, cudaStream_t st) {
  // threads of the longest block: the first one's vectors, or the last one's vectors and elements
  const uint64_t last = (a.total_bytes - 1) % a.block_bytes + 1;
  const uint64_t most = std::max(a.total_bytes > a.block_bytes ? a.block_bytes / (V * 16) : 0, last / (V * 16) + last % (V * 16) / a.es);
  const uint64_t per = (most + kWorldThreads - 1) / kWorldThreads;
  if (per == 0 || per > 0x7fffffffull) return cudaErrorInvalidValue;
  return launch_pdl(world_reduce_kernel<POL, V, DEPTH, G, RANKS>, dim3((unsigned)per, (unsigned)entries), kWorldThreads, 0, st, a);
}

// Of up to eight ranks only the integers' reduce-scatters of trees come here (one word a value, so the deepest form costs
// nothing: eight int32 buckets of 25 MB flat 63.8 us, 2*4 64.3).  From nine ranks up every program runs the deepest form: sixteen fp32 buckets flat 130 us (6.5 TB/s), 4*4
// 132, 2*2*2*2 141 (6.0 TB/s), in bf16 139, 151 and 166 us.
template <int POL, int RANKS>
static cudaError_t launch_r(const WorldArgs<RANKS>& a, int entries, bool wide, cudaStream_t st) {
  if constexpr (RANKS <= 8) {
    return wide ? launch_t<POL, 2, 2, 8, RANKS>(a, entries, st) : launch_t<POL, 1, 2, 8, RANKS>(a, entries, st);
  } else {
    return launch_t<POL, 1, 3, 8, RANKS>(a, entries, st);
  }
}

template <int RANKS>
cudaError_t launch_world(int pol, const WorldArgs<RANKS>& a, int entries, bool wide, cudaStream_t st) {
  switch (pol) {
    case POL_ADD8: return launch_r<POL_ADD8>(a, entries, wide, st);
    case POL_ADD16: return launch_r<POL_ADD16>(a, entries, wide, st);
    case POL_ADD32: return launch_r<POL_ADD32>(a, entries, wide, st);
    case POL_ADD64: return launch_r<POL_ADD64>(a, entries, wide, st);
    case POL_OR: return launch_r<POL_OR>(a, entries, wide, st);
    case POL_AND: return launch_r<POL_AND>(a, entries, wide, st);
    default: break;
  }
  if constexpr (RANKS > 8) {
    switch (pol) {
      case POL_F32: return launch_r<POL_F32>(a, entries, wide, st);
      case POL_F64: return launch_r<POL_F64>(a, entries, wide, st);
      case POL_BF16: return launch_r<POL_BF16>(a, entries, wide, st);
      case POL_F16: return launch_r<POL_F16>(a, entries, wide, st);
      default: break;
    }
  }
  return cudaErrorInvalidValue;
}
template cudaError_t launch_world<8>(int, const WorldArgs<8>&, int, bool, cudaStream_t);
template cudaError_t launch_world<16>(int, const WorldArgs<16>&, int, bool, cudaStream_t);

}  // namespace ftk
