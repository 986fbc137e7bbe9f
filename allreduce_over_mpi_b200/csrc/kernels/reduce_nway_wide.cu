// Single-GPU n-way reduction with 256-bit global accesses (sm_100a).
//
// Blackwell adds 32-byte vector loads and stores (ld/st.global.v8.b32) and, on them only,
// the per-instruction L2 eviction priority.  For a pure streaming sum that halves the
// number of memory instructions per byte against the 16-byte kernels of reduce_nway.cu
// and lets both the inputs (read once) and the result (written once) leave L2 first.
// The fan-in is a template parameter for the common cases, so every load of a step is
// issued before the first add and nothing is indexed at run time.
//
// Same job as the reference's reduce_sum_2 .. reduce_sum_8 kernels
// (vector_add/reduce_sum_gpu.h:13-69), which move 4 bytes per thread.
#include <type_traits>

#include "pdl.cuh"
#include "reduce_nway.cuh"
#include "vec.cuh"

namespace ftk {

// LD: 0 = L1::no_allocate, 1 = L1::no_allocate + L2::evict_first, 2 = non-coherent + L2::evict_first
template <int LD>
__device__ __forceinline__ void ld32(const void* p, uint4& a, uint4& b) {
  if (LD == 0)
    asm volatile("ld.global.L1::no_allocate.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w) : "l"(p) : "memory");
  else if (LD == 1)
    asm volatile("ld.global.L1::no_allocate.L2::evict_first.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w) : "l"(p) : "memory");
  else
    asm volatile("ld.global.nc.L1::no_allocate.L2::evict_first.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w) : "l"(p));
}
// ST: 0 = default (write-back), 1 = L2::evict_first, 2 = L1::no_allocate only
template <int ST>
__device__ __forceinline__ void st32(void* p, const uint4& a, const uint4& b) {
  if (ST == 0)
    asm volatile("st.global.v8.u32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w) : "memory");
  else if (ST == 1)
    asm volatile("st.global.L1::no_allocate.L2::evict_first.v8.u32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w) : "memory");
  else
    asm volatile("st.global.L1::no_allocate.v8.u32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w) : "memory");
}

// The default: one 32-byte unit per thread, 128 threads, the grid covers the vector once, evict-first stores.  NSRC > 0:
// the fan-in is known at compile time; NSRC == 0: it is a.n (any value up to FT_MAX_FANIN).  Sources are taken GROUP at
// a time: all loads of a group are issued before its first add.  How a thread
// behind the end is kept from loading decides how many the compiler leaves in flight: a predicate on each load keeps a
// group and more (72 registers, bf16 x8 of 4 M 11.7 us), leaving early 50 registers and 12.2 us, loading zeros instead
// 40 registers and 14.1 us.
//
// What bounds it is HBM, or L2 below about 100 MB.
// Calls below 50 MB: groups of four (eight from nine sources up).  Over 2, 4, 8 and 16 sources of 16 KB to 256 MB in fp32,
// bf16 and fp16 that is 0.8 % from the best of 12 configurations on average and 8 % at most (128-512 threads, groups of 4
// and 8, three places for the dependent launch); 256 threads lose up to 26 % where the grid fills the chip only once or
// twice.  The edges are the job of a CTA of their own, the last one, behind the body: a branch in front of the loads cost 3
// to 5 %.  fp32 x8 of 1 M: 4.8 us.
// Larger ones (EARLY) fetch ahead and ask for their successor (pdl.cuh).  Where they ask decides what it is worth: behind
// the first load of the last group, with the edges between the loads and the additions, it works; with code behind the
// store it worked no better than asking at the very end.  All of up to eight sources in flight together pay then, and the
// edges are the first CTA's: the last one starts when the call is nearly over (fp32 x3 views of 5 M 12.2 us with the last
// one, 11.4 with the first).  us, calls in a row on fresh tensors, neither / this: fp32 x2 of 5 M 10.1 / 8.7, x3 views 12.9
// / 11.4, x4 of 2.7 M 9.2 / 7.9, x8 of 1.5 M 9.4 / 8.0, of 2.5 M 14.5 / 12.9, of 6.5 M 34.3 / 33.2 (7.1 TB/s), of 64 Mi
// 335.1 / 334.2 (7.2); bf16 x8 of 4 M 12.0 / 10.6; int32 masks x6 of 3 M 13.6 / 12.1; fp64 x2 of 4 M 15.4 / 14.1.  From nine
// sources up they ask behind the fourth load of the last group (fp32 x16 of 1.2 M 13.2 / 12.1), in 16-bit floats behind all of
// them (x16 of 8 M 40.2, 39.1 so, 39.8 behind the fourth).  In a captured graph x8 of 2.5 M 14.5 / 13.1.
template <int POL, int NSRC, int THREADS, int GROUP, bool EARLY>
__global__ void __launch_bounds__(THREADS) reduce_nway_wide_kernel(const __grid_constant__ NwayArgs a) {
  using P = typename PolById<POL>::type;
  const unsigned long long i = (unsigned long long)blockIdx.x * THREADS + threadIdx.x;
  const bool ok = i < a.nvec;
  if (EARLY && blockIdx.x < a.seam.ahead && ok && !(threadIdx.x & 3)) {
#pragma unroll
    for (int k = 0; k < (NSRC > 0 ? NSRC : FT_MAX_FANIN); ++k) {
      if (NSRC == 0 && k >= a.n) break;
      l2_ahead((const unsigned char*)a.src[k] + i * 32);
    }
  }
  pdl_begin();
  constexpr int G = (NSRC > 0 && NSRC < GROUP) ? NSRC : GROUP;
  constexpr bool between = EARLY && NSRC > 0 && sizeof(typename ScalarOp<POL>::elem) < 8;   // (8-byte edges there take up to 166 registers)
  // the load of the last group behind which the successor is asked for
  constexpr int ASK = between ? 0 : NSRC > 0 ? (G - 1) / 2 : POL == POL_BF16 || POL == POL_F16 ? G - 1 : 3;
  typename P::Acc al, ah;
#pragma unroll
  for (int g0 = 0; g0 < (NSRC > 0 ? NSRC : FT_MAX_FANIN); g0 += G) {
    if (NSRC == 0 && g0 >= a.n) break;
    const bool last = g0 + G >= (NSRC > 0 ? NSRC : a.n);
    uint4 lo[G], hi[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      if (ok && g0 + g < (NSRC > 0 ? NSRC : a.n)) ld32<0>((const unsigned char*)a.src[g0 + g] + i * 32, lo[g], hi[g]);
      if (EARLY && g == ASK && last) pdl_next(blockIdx.x >= a.seam.ask);
    }
    if (between && last && a.edge && blockIdx.x == 0) reduce_edges<POL, ScalarOp>(a);
#pragma unroll
    for (int g = 0; g < G; ++g)
      if (g0 + g < (NSRC > 0 ? NSRC : a.n)) {
        if (g0 + g == 0) { P::init(al, lo[g]); P::init(ah, hi[g]); }
        else { P::add(al, lo[g]); P::add(ah, hi[g]); }
      }
  }
  if (ok) st32<1>((unsigned char*)a.dst + i * 32, P::fin(al), P::fin(ah));
  if (!between && (EARLY || !ok) && a.edge && blockIdx.x == (EARLY ? 0 : gridDim.x - 1)) reduce_edges<POL, ScalarOp>(a);
}

// The configurations that are asked for by number: one thread handles UNROLL 32-byte units per step, THREADS apart (every warp access is one
// contiguous 1 KiB run).  The grid either covers the vector once (one step per thread) or is
// capped and strides over it.  NSRC > 0: the fan-in is known at compile time; NSRC == 0: it is
// a.n (any value up to FT_MAX_FANIN).  Sources are taken GROUP at a time: all loads of a group are
// issued before its first add.
template <int POL, int NSRC, int UNROLL, int LD, int ST, int THREADS, int GROUP>
__global__ void __launch_bounds__(THREADS) reduce_nway_strided_kernel(const __grid_constant__ NwayArgs a) {
  using P = typename PolById<POL>::type;
  pdl_begin();
  const int edge_ctas = a.edge != 0;
  if (edge_ctas && blockIdx.x == gridDim.x - 1) {
    reduce_edges<POL, ScalarOp>(a);
    return;
  }
  const unsigned long long n32 = a.nvec;
  const int nsrc = NSRC > 0 ? NSRC : a.n;
  const unsigned long long stride = (unsigned long long)(gridDim.x - edge_ctas) * THREADS * UNROLL;
  for (unsigned long long base = (unsigned long long)blockIdx.x * THREADS * UNROLL; base < n32; base += stride) {
    unsigned long long idx[UNROLL];
    bool ok[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      idx[u] = base + (unsigned long long)u * THREADS + threadIdx.x;
      ok[u] = idx[u] < n32;
    }
    constexpr int G = (NSRC > 0 && NSRC < GROUP) ? NSRC : GROUP;
    typename P::Acc al[UNROLL], ah[UNROLL];
#pragma unroll
    for (int g0 = 0; g0 < (NSRC > 0 ? NSRC : FT_MAX_FANIN); g0 += G) {
      if (NSRC == 0 && g0 >= nsrc) break;
      uint4 lo[G][UNROLL], hi[G][UNROLL];
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
          if (ok[u] && g0 + g < nsrc) ld32<LD>((const unsigned char*)a.src[g0 + g] + idx[u] * 32, lo[g][u], hi[g][u]);
          else lo[g][u] = hi[g][u] = make_uint4(0, 0, 0, 0);
        }
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
          if (g0 + g == 0) { P::init(al[u], lo[g][u]); P::init(ah[u], hi[g][u]); }
          else if (g0 + g < nsrc) { P::add(al[u], lo[g][u]); P::add(ah[u], hi[g][u]); }
        }
    }
#pragma unroll
    for (int u = 0; u < UNROLL; ++u)
      if (ok[u]) st32<ST>((unsigned char*)a.dst + idx[u] * 32, P::fin(al[u]), P::fin(ah[u]));
  }
}

// Configurations by code = U*1000 + LD*100 + ST*10 + T, with U units per thread per step, LD/ST as above,
// T: 0 = 256 threads and one step per thread (the grid covers the vector), 1 = 512 threads likewise,
//    3 = 512 threads x 4 CTAs per SM striding over the vector; groups of four sources.
template <int POL, int NSRC, int UNROLL, int LD, int ST, int THREADS, int GROUP>
static cudaError_t launch_t(const NwayArgs& a, int ctas_per_sm, int sms, cudaStream_t st) {
  const unsigned long long per_cta = (unsigned long long)THREADS * UNROLL;
  unsigned long long grid = (a.nvec + per_cta - 1) / per_cta;
  if (ctas_per_sm && grid > (unsigned long long)sms * ctas_per_sm) grid = (unsigned long long)sms * ctas_per_sm;
  grid += a.edge != 0;
  if (grid > 0x7fffffffull || grid == 0) return cudaErrorInvalidValue;
  return launch_pdl(reduce_nway_strided_kernel<POL, NSRC, UNROLL, LD, ST, THREADS, GROUP>, (unsigned)grid, THREADS, 0, st, a);
}
template <int POL, int NSRC, int UNROLL, int LD, int ST>
static cudaError_t launch_v(const NwayArgs& a, int t, int sms, cudaStream_t st) {
  return t == 0 ? launch_t<POL, NSRC, UNROLL, LD, ST, 256, 4>(a, 0, sms, st)
                : launch_t<POL, NSRC, UNROLL, LD, ST, 512, 4>(a, t == 3 ? 4 : 0, sms, st);
}

template <int POL, int NSRC, bool TUNING>
static cudaError_t launch_cfg(const NwayArgs& a, int code, int sms, cudaStream_t st) {
  const int t = code % 10;
  if (t != 0 && t != 1 && t != 3) return cudaErrorInvalidValue;
  if (code == 0) {
    NwayArgs b = a;
    b.seam = seam_of((a.n + 1) * a.nvec * 32, a.n * kWideThreads * 32, body_ctas(a, kWideThreads));
    const unsigned long long grid = nway_grid(b, kWideThreads);
    if (grid > 0x7fffffffull || grid == 0) return cudaErrorInvalidValue;
    return launch_pdl(b.seam.ahead ? reduce_nway_wide_kernel<POL, NSRC, kWideThreads, 8, true>
                              : reduce_nway_wide_kernel<POL, NSRC, kWideThreads, NSRC == 0 ? 8 : 4, false>, (unsigned)grid, kWideThreads, 0, st, b);
  }
  if constexpr (TUNING) {
    switch (code / 10) {
      case 101: return launch_v<POL, NSRC, 1, 0, 1>(a, t, sms, st);
      case 100: return launch_v<POL, NSRC, 1, 0, 0>(a, t, sms, st);
      case 111: return launch_v<POL, NSRC, 1, 1, 1>(a, t, sms, st);
      case 200: return launch_v<POL, NSRC, 2, 0, 0>(a, t, sms, st);
      case 201: return launch_v<POL, NSRC, 2, 0, 1>(a, t, sms, st);
      case 211: return launch_v<POL, NSRC, 2, 1, 1>(a, t, sms, st);
      default: break;
    }
  }
  return cudaErrorInvalidValue;
}

template <int POL, bool TUNING>
static cudaError_t launch_n(const NwayArgs& a, int code, int sms, cudaStream_t st) {
  switch (a.n) {
    case 1: return launch_cfg<POL, 1, false>(a, code, sms, st);
    case 2: return launch_cfg<POL, 2, TUNING>(a, code, sms, st);
    case 3: return launch_cfg<POL, 3, TUNING>(a, code, sms, st);
    case 4: return launch_cfg<POL, 4, TUNING>(a, code, sms, st);
    case 5: return launch_cfg<POL, 5, false>(a, code, sms, st);
    case 6: return launch_cfg<POL, 6, false>(a, code, sms, st);
    case 7: return launch_cfg<POL, 7, false>(a, code, sms, st);
    case 8: return launch_cfg<POL, 8, TUNING>(a, code, sms, st);
    default: return launch_cfg<POL, 0, false>(a, code, sms, st);
  }
}

cudaError_t launch_wide(int pol, const NwayArgs& a, int code, int sms, cudaStream_t st) {
  switch (pol) {
    case POL_ADD8: return launch_n<POL_ADD8, false>(a, code, sms, st);
    case POL_ADD16: return launch_n<POL_ADD16, false>(a, code, sms, st);
    case POL_ADD32: return launch_n<POL_ADD32, false>(a, code, sms, st);
    case POL_ADD64: return launch_n<POL_ADD64, false>(a, code, sms, st);
    case POL_OR: return launch_n<POL_OR, false>(a, code, sms, st);
    case POL_AND: return launch_n<POL_AND, false>(a, code, sms, st);
    case POL_F32: return launch_n<POL_F32, true>(a, code, sms, st);
    case POL_F64: return launch_n<POL_F64, false>(a, code, sms, st);
    case POL_BF16: return launch_n<POL_BF16, true>(a, code, sms, st);
    case POL_F16: return launch_n<POL_F16, false>(a, code, sms, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace ftk
