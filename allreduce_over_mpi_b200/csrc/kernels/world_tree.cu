// One pass over the copies of all ranks of a world that lives on one device, for up to eight ranks: sums whose program is
// compiled in, and copies.
//
// The data is read once and written once, so HBM bounds a large call and L2 one that fits there; a small one is bounded by
// what happens before its first load.  Against world_reduce_kernel, which looks each step up in a kilobyte of parameters
// (one miss of the constant cache after the other, branches, moves of the values put aside, up to 126 registers), calls
// captured in a graph, three sets of tensors in turn, eight ranks in place, us:
//                      fp32 2 KB    fp32 400 KB    fp32 2 MB     bf16 6 MB      bf16 25 MB      fp16 25 MB
//     flat            2.95 -> 1.34  3.78 -> 1.78  5.75 -> 3.70  19.6 -> 16.1  64.4 -> 63.9    64.4 -> 63.9
//     2*4             3.90 -> 1.38  4.79 -> 1.81  7.79 -> 3.74  20.3 -> 16.2  65.0 -> 63.9    66.5 -> 64.0
//     2*2*2           3.83 -> 1.38  4.72 -> 1.85  8.06 -> 3.77  22.5 -> 16.3  72.1 -> 64.0    74.0 -> 64.1
//     ring            4.11 -> 1.38  5.06 -> 1.85  8.24 -> 3.78  20.4 -> 16.2  65.1 -> 64.0    68.7 -> 64.1
// (64 us is 6.55 TB/s, the rate of a copy.  With fetching ahead, pdl.cuh, calls in a row on the stream: fp32 6 MB 15.3, bf16 25
// MB 2*4 62.6, fp16 12 MB 2*2*2 34.9 at first and 29.7 now.)  Integers, flat of eight: 3.36 -> 2.20, 4.25 -> 2.40 us at 2 and 400 KB.
#include <algorithm>
#include <utility>

#include "../api/flextree.h"
#include "pdl.cuh"
#include "vec.cuh"
#include "world_dev.h"

namespace ftk {

constexpr bool floating(int pol) { return pol == POL_F32 || pol == POL_F64 || pol == POL_BF16 || pol == POL_F16; }

// L2's choice of what leaves first, for accesses of 32 bytes (narrower ones have none): before the rest, or as usual.
__device__ __forceinline__ uint64_t l2_policy(bool first) {
  uint64_t normal, early;
  asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(normal));
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(early));
  return first ? early : normal;
}
// Predicated accesses (no branch, so that all of them are issued back to back): V 16-byte vectors at p.
template <int V>
__device__ __forceinline__ void tree_load(const unsigned char* p, bool ok, uint4 (&v)[V], uint64_t policy) {
  if constexpr (V == 2)
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %9, 0;\n\t"
                 "@q ld.global.L1::no_allocate.L2::cache_hint.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8], %10;\n\t}"
                 : "=r"(v[0].x), "=r"(v[0].y), "=r"(v[0].z), "=r"(v[0].w), "=r"(v[1].x), "=r"(v[1].y), "=r"(v[1].z), "=r"(v[1].w)
                 : "l"(p), "r"((uint32_t)ok), "l"(policy) : "memory");
  else
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\t"
                 "@q ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n\t}"
                 : "=r"(v[0].x), "=r"(v[0].y), "=r"(v[0].z), "=r"(v[0].w) : "l"(p), "r"((uint32_t)ok) : "memory");
}
template <int V>
__device__ __forceinline__ void tree_store(unsigned char* p, bool ok, const uint4 (&v)[V]) {
  if constexpr (V == 2)
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %9, 0;\n\t@q st.global.v8.u32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n\t}"
                 ::"l"(p), "r"(v[0].x), "r"(v[0].y), "r"(v[0].z), "r"(v[0].w), "r"(v[1].x), "r"(v[1].y), "r"(v[1].z), "r"(v[1].w),
                   "r"((uint32_t)ok) : "memory");
  else
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\t@q st.global.v4.u32 [%0], {%1,%2,%3,%4};\n\t}"
                 ::"l"(p), "r"(v[0].x), "r"(v[0].y), "r"(v[0].z), "r"(v[0].w), "r"((uint32_t)ok) : "memory");
}
template <int V>
__device__ __forceinline__ void tree_store(unsigned char* p, bool ok, const uint4 (&v)[V], uint64_t policy) {
  if constexpr (V == 2)
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %9, 0;\n\t"
                 "@q st.global.L2::cache_hint.v8.u32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8}, %10;\n\t}"
                 ::"l"(p), "r"(v[0].x), "r"(v[0].y), "r"(v[0].z), "r"(v[0].w), "r"(v[1].x), "r"(v[1].y), "r"(v[1].z), "r"(v[1].w),
                   "r"((uint32_t)ok), "l"(policy) : "memory");
  else
    tree_store<V>(p, ok, v);
}

// Where a thread works: whole vectors of V x 16 bytes first, then the elements behind the last one, a thread each.
struct TreePlace {
  uint64_t off;
  bool full, any;
};
template <int V>
__device__ __forceinline__ TreePlace tree_place(const WorldTreeArgs& a, uint32_t block, uint32_t es) {
  const uint64_t lo = block * a.block_bytes, end = lo + a.block_bytes < a.total_bytes ? lo + a.block_bytes : a.total_bytes;
  if (lo >= end) return {0, false, false};
  const uint64_t i = (uint64_t)blockIdx.x * kTreeThreads + threadIdx.x, whole = (end - lo) / (V * 16);
  const bool full = i < whole;
  const uint64_t off = lo + (full ? i * (V * 16) : whole * (V * 16) + (i - whole) * es);
  return {off, full, off < end};
}

__device__ __forceinline__ uint32_t tree_cta() { return blockIdx.y * gridDim.x + blockIdx.x; }

// A step's code and a round's place are constants here: with all loops unrolled nothing is left of them but the additions,
// the roundings and, of the values put aside, their registers.  A value that was just rounded is put aside in the element
// type.
template <class P, int V, int N, uint32_t CODE, class Round>
__device__ __forceinline__ void tree_sum(const uint4 (&v)[N][V], typename P::Acc (&acc)[V], Round&& round) {
  typename P::Acc aside[2][V];
  uint4 w[V], packed[2][V];
  bool in_w = false, is_packed[2] = {false, false};
  int sp = 0, t = 0;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const uint32_t code = CODE >> (4 * k) & 15;
    if (code & 1) {
      if (k > 0) {
        is_packed[sp] = in_w;
#pragma unroll
        for (int h = 0; h < V; ++h) {
          if (in_w) packed[sp][h] = w[h];
          else aside[sp][h] = acc[h];
        }
        ++sp;
      }
#pragma unroll
      for (int h = 0; h < V; ++h) P::init(acc[h], v[k][h]);
    } else {
#pragma unroll
      for (int h = 0; h < V; ++h) {
        if (in_w) P::init(acc[h], w[h]);
        P::add(acc[h], v[k][h]);
      }
    }
    in_w = false;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      if (r >= (int)(code >> 2)) continue;
#pragma unroll
      for (int h = 0; h < V; ++h) w[h] = P::fin(acc[h]);
      round(t++, w);
      if (r + 1 < (int)(code >> 2) || (code & 2)) {
        --sp;
#pragma unroll
        for (int h = 0; h < V; ++h) {
          if (is_packed[sp]) P::init(acc[h], packed[sp][h]);
          else acc[h] = aside[sp][h];
          P::add(acc[h], w[h]);
        }
      } else {
        in_w = true;
      }
    }
  }
}

// blockIdx.y: the entry.  All N loads of a thread are in flight together, whatever the program.  The parameters are looked up
// in front of pdl_begin(), while the kernel before this one ends.  At most 128 registers, for four CTAs on an SM (32 bytes
// of eight ranks take 88 in fp32 and 120 in bf16, 16 bytes 56 to 71).
template <int POL, int V, int TREE>
__global__ void __launch_bounds__(kTreeThreads, 4) world_tree_kernel(const __grid_constant__ WorldTreeArgs a) {
  using P = typename PolById<POL>::type;
  constexpr WorldTree T = kWorldTrees[TREE];
  constexpr int N = T.ranks;
  const uint32_t ES = floating(POL) ? (uint32_t)sizeof(typename ScalarOp<POL>::elem) : a.es;   // (the integers' policies serve several widths)
  const uint64_t word = a.entry[blockIdx.y];
  const uint32_t lo = (uint32_t)word, hi = (uint32_t)(word >> 32);
  const TreePlace at = tree_place<V>(a, hi & 7, ES);
  const unsigned char* src[N];
#pragma unroll
  for (int k = 0; k < N; ++k) src[k] = (const unsigned char*)a.in[lo >> (3 * k) & 7] + at.off;
  if (tree_cta() < a.seam.ahead && at.full && !(threadIdx.x & 3)) {
#pragma unroll
    for (int k = 0; k < N; ++k) l2_ahead(src[k]);
  }
  pdl_begin();
  if (!at.any) return;
  uint4 v[N][V];
  const uint64_t policy = l2_policy(a.streams);
#pragma unroll
  for (int k = 0; k < N; ++k) tree_load<V>(src[k], at.full, v[k], policy);
  pdl_next(tree_cta() >= a.seam.ask);
  if (!at.full) {
#pragma unroll
    for (int k = 0; k < N; ++k) v[k][0] = ld_element(src[k], ES);
  }
  typename P::Acc acc[V];
  const auto round = [&](int t, const uint4 (&w)[V]) {
    const uint32_t to = (uint32_t)(word >> (kTreeStore + 4 * t)) & 15;
    if (to != 15) {
      if (at.full) tree_store<V>((unsigned char*)a.out[to] + at.off, true, w);
      else st_element((unsigned char*)a.out[to] + at.off, w[0], ES);
    }
  };
  if (T.code[0] == T.code[1] || !(hi >> (kTreeWhich - 32) & 1)) tree_sum<P, V, N, T.code[0]>(v, acc, round);
  else tree_sum<P, V, N, T.code[1]>(v, acc, round);
  uint4 w[V];
#pragma unroll
  for (int h = 0; h < V; ++h) w[h] = P::fins(acc[h], a.scale);
  const uint32_t mask = lo >> kTreeMask;
#pragma unroll
  for (int r = 0; r < N; ++r) tree_store<V>((unsigned char*)a.out[r] + at.off, at.full && (mask >> r & 1), w);
  if (!at.full) {
#pragma unroll
    for (int r = 0; r < N; ++r)
      if (mask >> r & 1) st_element((unsigned char*)a.out[r] + at.off, w[0], ES);
  }
}

// Copies of one rank's block to others.
template <int V>
__global__ void __launch_bounds__(kTreeThreads) world_copy_kernel(const __grid_constant__ WorldTreeArgs a) {
  const uint64_t word = a.entry[blockIdx.y];
  const uint32_t lo = (uint32_t)word;
  const TreePlace at = tree_place<V>(a, (uint32_t)(word >> 32) & 7, a.es);
  const unsigned char* src = (const unsigned char*)a.in[lo & 7] + at.off;
  pdl_begin();
  if (!at.any) return;
  uint4 v[V];
  const uint64_t policy = l2_policy(a.streams);
  tree_load<V>(src, at.full, v, policy);
  pdl_next(tree_cta() >= a.seam.ask);
  if (!at.full) v[0] = ld_element(src, a.es);
  const uint32_t mask = lo >> kTreeMask;
#pragma unroll
  for (int r = 0; r < kTreeRanks; ++r) tree_store<V>((unsigned char*)a.out[r] + at.off, at.full && (mask >> r & 1), v, policy);
  if (!at.full)
    for (int r = 0; r < kTreeRanks; ++r)
      if (mask >> r & 1) st_element((unsigned char*)a.out[r] + at.off, v[0], a.es);
}

// CTAs that cover the longest block: the first one's vectors, or the last one's vectors and elements.
template <int V>
static dim3 tree_grid(const WorldTreeArgs& a, int entries) {
  const uint64_t last = (a.total_bytes - 1) % a.block_bytes + 1;
  const uint64_t most = std::max(a.total_bytes > a.block_bytes ? a.block_bytes / (V * 16) : 0, last / (V * 16) + last % (V * 16) / a.es);
  const uint64_t per = (most + kTreeThreads - 1) / kTreeThreads;
  return per > 0x7fffffffull ? dim3(0) : dim3((unsigned)per, (unsigned)entries);
}
template <int POL, int V, int TREE>
static cudaError_t launch_t(const WorldTreeArgs& a, int entries, cudaStream_t st) {
  const dim3 grid = tree_grid<V>(a, entries);
  return grid.x ? launch_pdl(world_tree_kernel<POL, V, TREE>, grid, kTreeThreads, 0, st, a) : cudaErrorInvalidValue;
}
template <int POL, int... TREE>
static cudaError_t launch_p(const WorldTreeArgs& a, int tree, int entries, bool wide, cudaStream_t st, std::integer_sequence<int, TREE...>) {
  using Fn = cudaError_t (*)(const WorldTreeArgs&, int, cudaStream_t);
  static constexpr Fn wide_fn[] = {launch_t<POL, 2, TREE>...}, narrow_fn[] = {launch_t<POL, 1, TREE>...};
  return (wide ? wide_fn : narrow_fn)[tree](a, entries, st);
}

// `tree`: index into kWorldTrees; integers have the flat ones only (is_flat_tree).
cudaError_t launch_world_tree(int pol, const WorldTreeArgs& a, int tree, int entries, bool wide, cudaStream_t st) {
  constexpr std::make_integer_sequence<int, kWorldTreeCount> all{};
  constexpr std::make_integer_sequence<int, kFlatTrees> flat{};
  switch (pol) {
    case POL_F32: return launch_p<POL_F32>(a, tree, entries, wide, st, all);
    case POL_F64: return launch_p<POL_F64>(a, tree, entries, wide, st, all);
    case POL_BF16: return launch_p<POL_BF16>(a, tree, entries, wide, st, all);
    case POL_F16: return launch_p<POL_F16>(a, tree, entries, wide, st, all);
    default: break;
  }
  if (tree >= kFlatTrees) return cudaErrorInvalidValue;
  switch (pol) {
    case POL_ADD8: return launch_p<POL_ADD8>(a, tree, entries, wide, st, flat);
    case POL_ADD16: return launch_p<POL_ADD16>(a, tree, entries, wide, st, flat);
    case POL_ADD32: return launch_p<POL_ADD32>(a, tree, entries, wide, st, flat);
    case POL_ADD64: return launch_p<POL_ADD64>(a, tree, entries, wide, st, flat);
    case POL_OR: return launch_p<POL_OR>(a, tree, entries, wide, st, flat);
    case POL_AND: return launch_p<POL_AND>(a, tree, entries, wide, st, flat);
    default: return cudaErrorInvalidValue;
  }
}
cudaError_t launch_world_copy(const WorldTreeArgs& a, int entries, bool wide, cudaStream_t st) {
  const dim3 grid = wide ? tree_grid<2>(a, entries) : tree_grid<1>(a, entries);
  if (!grid.x) return cudaErrorInvalidValue;
  return wide ? launch_pdl(world_copy_kernel<2>, grid, kTreeThreads, 0, st, a) : launch_pdl(world_copy_kernel<1>, grid, kTreeThreads, 0, st, a);
}

}  // namespace ftk
