// out = scale * sum_k src[k] on one GPU, fp32 accumulation, fp32 or bf16 in and out (gradient averaging with the cast
// fused into the store).
//
// HBM bounds it, as it does reduce_nway_wide.cu, whose layout it shares: 32 bytes of every source per thread, several
// sources in flight, the grid covers the vector once, dependent launch.  The unit
// is 8 fp32 or 16 bf16 elements, whatever the output type, so that the source side (n streams to one) stays on 256-bit
// loads.  fp32 -> bf16, 8 sources of 6.5 M: 38.9 us (5.7 TB/s, a strided loop with 16-byte loads of one source at a
// time) -> 31.6 us (7.0 TB/s).
#include <type_traits>

#include "../api/flextree.h"
#include "pdl.cuh"
#include "reduce_nway.cuh"
#include "vec.cuh"

namespace ftk {

constexpr int kThreads = kWideThreads;

template <bool WIDE>
__device__ __forceinline__ void load32(const unsigned char* p, uint4& a, uint4& b) {
  if (WIDE) {
    asm volatile("ld.global.L1::no_allocate.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w) : "l"(p) : "memory");
  } else {
    a = ld_stream(p);
    b = ld_stream(p + 16);
  }
}
template <bool WIDE>
__device__ __forceinline__ void store32(unsigned char* p, const uint4& a, const uint4& b) {
  if (WIDE) {
    asm volatile("st.global.L1::no_allocate.L2::evict_first.v8.u32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w) : "memory");
  } else {
    st_vec_cs(p, a);
    st_vec_cs(p + 16, b);
  }
}

// Element i (of a body that starts at element 0) of the result, G sources in flight at a time; G == 1: as many as eight, the
// rest one by one (in the kernel for nine sources and more any other form takes registers from the body).  The few edges of a
// vector are on a call's critical path: with all but the whole eights one by one fp32 x7 of 1 M took 7.2 us, now 6.3.
template <bool IN_BF16, bool OUT_BF16, int NSRC, int G>
__device__ __forceinline__ void scaled_element(const NwayArgs& a, long long i, float scale) {
  using T = std::conditional_t<IN_BF16, __nv_bfloat16, float>;
  const int n = NSRC > 0 ? NSRC : a.n;
  float acc = 0.f;
#pragma unroll(G == 1 ? 8 : 1)
  for (int k0 = 0; k0 < n; k0 += G) {
    T v[G];
    if (k0 + G <= n) {   // (a predicate on each load costs bf16 x8 of 6.5 M, one element off, 4 us of 29)
#pragma unroll
      for (int g = 0; g < G; ++g) v[g] = ((const T*)a.src[k0 + g])[i];
#pragma unroll
      for (int g = 0; g < G; ++g) acc += (float)v[g];
    } else {
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (k0 + g < n) v[g] = ((const T*)a.src[k0 + g])[i];
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (k0 + g < n) acc += (float)v[g];
    }
  }
  acc *= scale;
  if (OUT_BF16) ((__nv_bfloat16*)a.dst)[i] = __float2bfloat16_rn(acc);
  else ((float*)a.dst)[i] = acc;
}

// WIDE: 256-bit accesses (every source on a 32-byte boundary, the output on one of 16 bytes for fp32 -> bf16, else
// 32); not WIDE: 128-bit ones.  ASK: kPlain, or (calls that fetch ahead, pdl.cuh) the load of the last group behind which
// the successor is asked for, kAskLast behind all of them; the edges are the first CTA's then.  Registers: left alone the
// compiler takes 32 for two fp32 sources, and spills, and 72 for seven, and loads the edges one after the other.
constexpr int kPlain = -2, kAskLast = -1;
template <bool IN_BF16, bool OUT_BF16, bool WIDE, int NSRC, int GROUP, int ASK>
__global__ void __launch_bounds__(kThreads, ASK == kPlain ? 0 : NSRC == 2 ? 12 : NSRC == 7 ? 6 : 0) reduce_nway_scaled_kernel(const __grid_constant__ NwayArgs a) {
  constexpr int E = IN_BF16 ? 16 : 8;   // elements per thread: 32 bytes of every source
  constexpr bool early = ASK != kPlain;
  const unsigned long long i = (unsigned long long)blockIdx.x * kThreads + threadIdx.x;
  const bool ok = i < a.nvec;
  if (early && blockIdx.x < a.seam.ahead && ok && !(threadIdx.x & 3))
    for (int k = 0; k < (NSRC > 0 ? NSRC : a.n); ++k) l2_ahead((const unsigned char*)a.src[k] + i * 32);
  pdl_begin();
  const auto edges = [&] {
    for (int e = threadIdx.x; e < (int)a.edge; e += kThreads)
      scaled_element<IN_BF16, OUT_BF16, NSRC, (NSRC > 0 ? NSRC : early ? 1 : 8)>(a, e < a.head ? (long long)e - a.head : (long long)(a.nbody + (e - a.head)), a.scale);
  };
  if (!ok) {
    if (!early && a.edge && blockIdx.x == gridDim.x - 1) edges();
    return;
  }
  float acc[E];
#pragma unroll
  for (int j = 0; j < E; ++j) acc[j] = 0.f;
  const int n = NSRC > 0 ? NSRC : a.n;
  for (int k0 = 0; k0 < n; k0 += GROUP) {
    const bool last = k0 + GROUP >= n;
    uint4 lo[GROUP], hi[GROUP];
#pragma unroll
    for (int g = 0; g < GROUP; ++g) {
      if (k0 + g < n) load32<WIDE>((const unsigned char*)a.src[k0 + g] + i * 32, lo[g], hi[g]);
      if (ASK == g && last) pdl_next(blockIdx.x >= a.seam.ask);
    }
    if (early && last && a.edge && blockIdx.x == 0) edges();
    if (ASK == kAskLast && last) pdl_next(blockIdx.x >= a.seam.ask);
#pragma unroll
    for (int g = 0; g < GROUP; ++g)
      if (k0 + g < n) {
        const uint32_t w[8] = {lo[g].x, lo[g].y, lo[g].z, lo[g].w, hi[g].x, hi[g].y, hi[g].z, hi[g].w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (IN_BF16) { acc[(2 * j) % E] += bf_lo(w[j]); acc[(2 * j + 1) % E] += bf_hi(w[j]); }
          else acc[j] += __uint_as_float(w[j]);
        }
      }
  }
  constexpr int W = OUT_BF16 ? E / 2 : E;   // output words
  uint32_t o[W];
#pragma unroll
  for (int j = 0; j < W; ++j) o[j] = OUT_BF16 ? pack_bf16x2(acc[(2 * j) % E] * a.scale, acc[(2 * j + 1) % E] * a.scale) : __float_as_uint(acc[j] * a.scale);
  unsigned char* d = (unsigned char*)a.dst + i * (W * 4);
  if constexpr (W == 4) {
    st_vec_cs(d, make_uint4(o[0], o[1], o[2], o[3]));
  } else {
#pragma unroll
    for (int j = 0; j + 8 <= W; j += 8)
      store32<WIDE>(d + j * 4, make_uint4(o[j], o[j + 1], o[j + 2], o[j + 3]), make_uint4(o[j + 4], o[j + 5], o[j + 6], o[j + 7]));
  }
}

// Pointers no common vector fits, views summed into a result at another offset for instance: one element at a time.
// Eight sources of 6.5 M, one element off: fp32 36.3 us (33.2 with a common vector), fp32 -> bf16 34.6 (31.6); bf16, with two
// bytes an access, 28.8 us (15.8), 4.1 TB/s.  Five sources 26.8, 25.4 and 30.8 us (62.6, 61.2 and 59.6 while only whole eights of
// them were in flight together).
template <bool IN_BF16, bool OUT_BF16>
__global__ void __launch_bounds__(256) reduce_nway_scaled_scalar_kernel(const __grid_constant__ NwayArgs a) {
  pdl_begin();
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < a.nbody; i += (unsigned long long)gridDim.x * blockDim.x)
    scaled_element<IN_BF16, OUT_BF16, 0, 8>(a, (long long)i, a.scale);
}

// Calls that do not fetch ahead: two and three sources have kernels of their own (bf16 x3 of 4 M 4.0 -> 3.1 us); from four up
// the loop is as good or better (with the fan-in known the compiler keeps fewer loads in flight: bf16 x8 of 4 M 14.3 us, not
// 12.0).  Eight sources in flight pay from nine up only: they cost registers, and those CTAs (bf16 x4 of 13 M 20.4 us with
// four, 24.7 with eight and 256 threads; x16 of 1 M 5.0 us with eight, 5.5 with four).  Threads behind the end leave: with a
// predicate on each load fp32 x2 -> bf16 of 8 M took 14.8 us, not 12.9.
// Calls that do, up to eight sources: the fan-in known, all sources in flight, the successor asked for behind the first load.
// From nine up groups of eight, asked for behind the last load.  Of 13 forms (fan-in known, groups of four, of eight; asking
// behind the first, the second, all; threads behind the end leave, or not) over 64, 90 and 200 MB, fresh or all in L2, that is
// within 1 % of the best for every type and fan-in.  us for 90 MB of fresh tensors, plain form / this:
//   sources         2            3            4            5            6            7            8            16
//   fp32            14.5 / 12.7  14.2 / 12.8  14.3 / 12.9  14.7 / 12.9  14.7 / 12.9  14.8 / 13.0  14.7 / 13.0  15.0 / 13.9
//   fp32 -> bf16    14.1 / 12.9  14.2 / 12.9  14.3 / 12.9  14.9 / 13.0  14.6 / 13.0  14.8 / 13.0  14.7 / 13.0  14.9 / 14.0
//   bf16 -> fp32    14.5 / 13.2  14.5 / 13.3  14.4 / 13.2  14.8 / 13.1  14.8 / 13.2  14.8 / 13.1  14.4 / 12.9  14.9 / 14.2
//   bf16            14.5 / 12.7  14.3 / 12.8  14.5 / 12.9  15.1 / 13.0  14.6 / 13.0  14.8 / 13.0  14.9 / 13.0  15.0 / 14.1
// (12.9 is 7.0 TB/s.)
template <bool IN_BF16, bool OUT_BF16, bool WIDE, int NSRC, int GROUP, int ASK>
static cudaError_t launch_k(const NwayArgs& a, unsigned grid, cudaStream_t st) {
  return launch_pdl(reduce_nway_scaled_kernel<IN_BF16, OUT_BF16, WIDE, NSRC, GROUP, ASK>, grid, kThreads, 0, st, a);
}
template <bool IN_BF16, bool OUT_BF16, bool WIDE>
static cudaError_t launch_n(const NwayArgs& a, unsigned grid, cudaStream_t st) {
  if (!a.seam.ahead) {
    switch (a.n) {
      case 2: return launch_k<IN_BF16, OUT_BF16, WIDE, 2, 2, kPlain>(a, grid, st);
      case 3: return launch_k<IN_BF16, OUT_BF16, WIDE, 3, 3, kPlain>(a, grid, st);
      default: break;
    }
    return a.n <= 8 ? launch_k<IN_BF16, OUT_BF16, WIDE, 0, 4, kPlain>(a, grid, st) : launch_k<IN_BF16, OUT_BF16, WIDE, 0, 8, kPlain>(a, grid, st);
  }
  switch (a.n) {
    case 2: return launch_k<IN_BF16, OUT_BF16, WIDE, 2, 2, 0>(a, grid, st);
    case 3: return launch_k<IN_BF16, OUT_BF16, WIDE, 3, 3, 0>(a, grid, st);
    case 4: return launch_k<IN_BF16, OUT_BF16, WIDE, 4, 4, 0>(a, grid, st);
    case 5: return launch_k<IN_BF16, OUT_BF16, WIDE, 5, 5, 0>(a, grid, st);
    case 6: return launch_k<IN_BF16, OUT_BF16, WIDE, 6, 6, 0>(a, grid, st);
    case 7: return launch_k<IN_BF16, OUT_BF16, WIDE, 7, 7, 0>(a, grid, st);
    case 8: return launch_k<IN_BF16, OUT_BF16, WIDE, 8, 8, 0>(a, grid, st);
    default: return launch_k<IN_BF16, OUT_BF16, WIDE, 0, 8, kAskLast>(a, grid, st);
  }
}

template <bool IN_BF16, bool OUT_BF16>
static cudaError_t launch_t(const NwayArgs& in, unsigned long long len, int sms, cudaStream_t st) {
  NwayArgs a;
  bool wide;
  if (!layout_scaled(in, len, IN_BF16, OUT_BF16, &a, &wide)) {
    const unsigned long long want = (len + 255) / 256, cap = (unsigned long long)sms * 8;
    a = in;
    a.nbody = len;
    return launch_pdl(reduce_nway_scaled_scalar_kernel<IN_BF16, OUT_BF16>, (unsigned)(want < cap ? want : cap), 256, 0, st, a);
  }
  constexpr unsigned out_bytes = (IN_BF16 ? 16 : 8) * (OUT_BF16 ? 2 : 4);
  a.seam = seam_of(a.n > 1 ? (a.n * 32 + out_bytes) * a.nvec : 0, a.n * kThreads * 32, body_ctas(a, kThreads));
  const unsigned long long grid = nway_grid(a, kThreads);
  if (grid > 0x7fffffffull) return cudaErrorInvalidValue;
  return wide ? launch_n<IN_BF16, OUT_BF16, true>(a, (unsigned)grid, st) : launch_n<IN_BF16, OUT_BF16, false>(a, (unsigned)grid, st);
}

cudaError_t launch_scaled(bool in_bf16, bool out_bf16, const NwayArgs& a, unsigned long long len, int sms, cudaStream_t st) {
  if (in_bf16) return out_bf16 ? launch_t<true, true>(a, len, sms, st) : launch_t<true, false>(a, len, sms, st);
  return out_bf16 ? launch_t<false, true>(a, len, sms, st) : launch_t<false, false>(a, len, sms, st);
}

}  // namespace ftk
