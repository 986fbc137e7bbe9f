// out = scale * sum_k src[k] on one GPU, fp32 accumulation, fp32 or bf16 in and out (gradient averaging with the cast
// fused into the store).
//
// HBM bounds it, as it does reduce_nway_wide.cu, whose layout it shares: 32 bytes of every source per thread, four
// or more sources in flight, the grid covers the vector once, dependent launch.  The unit
// is 8 fp32 or 16 bf16 elements, whatever the output type, so that the source side (n streams to one) stays on 256-bit
// loads.  fp32 -> bf16, 8 sources of 6.5 M: 38.9 us (5.7 TB/s, a strided loop with 16-byte loads of one source at a
// time) -> 31.6 us (7.0 TB/s).
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

// Element i (of a body that starts at element 0) of the result.
template <bool IN_BF16, bool OUT_BF16>
__device__ __forceinline__ void scaled_element(const NwayArgs& a, long long i, float scale) {
  float acc = 0.f;
#pragma unroll 8
  for (int k = 0; k < a.n; ++k)
    acc += IN_BF16 ? __bfloat162float(((const __nv_bfloat16*)a.src[k])[i]) : ((const float*)a.src[k])[i];
  acc *= scale;
  if (OUT_BF16) ((__nv_bfloat16*)a.dst)[i] = __float2bfloat16_rn(acc);
  else ((float*)a.dst)[i] = acc;
}

// WIDE: 256-bit accesses (every source on a 32-byte boundary, the output on one of 16 bytes for fp32 -> bf16, else
// 32); not WIDE: 128-bit ones.  ASK: kPlain, or (calls that fetch ahead, pdl.cuh) the load of the last group behind which
// the successor is asked for, kAskLast behind all of them; the edges are the first CTA's then.  LEAVE: a thread behind the
// end leaves; else a predicate keeps it from each load.
constexpr int kPlain = -2, kAskLast = -1;
template <bool IN_BF16, bool OUT_BF16, bool WIDE, int NSRC, int GROUP, int ASK, bool LEAVE>
__global__ void __launch_bounds__(kThreads) reduce_nway_scaled_kernel(const __grid_constant__ NwayArgs a) {
  constexpr int E = IN_BF16 ? 16 : 8;   // elements per thread: 32 bytes of every source
  constexpr bool early = ASK != kPlain;
  const unsigned long long i = (unsigned long long)blockIdx.x * kThreads + threadIdx.x;
  const bool ok = i < a.nvec;
  if (early && blockIdx.x < a.seam.ahead && ok && !(threadIdx.x & 3))
    for (int k = 0; k < (NSRC > 0 ? NSRC : a.n); ++k) l2_ahead((const unsigned char*)a.src[k] + i * 32);
  pdl_begin();
  const auto edges = [&] {
    for (int e = threadIdx.x; e < (int)a.edge; e += kThreads)
      scaled_element<IN_BF16, OUT_BF16>(a, e < a.head ? (long long)e - a.head : (long long)(a.nbody + (e - a.head)), a.scale);
  };
  if (LEAVE && !ok) {
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
      if ((LEAVE || ok) && k0 + g < n) load32<WIDE>((const unsigned char*)a.src[k0 + g] + i * 32, lo[g], hi[g]);
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
  if (!LEAVE && !ok) return;
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
// Eight sources of 6.5 M, one element off: fp32 36.6 us (34.6 with a common vector), fp32 -> bf16 34.9 (33.1); bf16, with two
// bytes an access, 27.4 us (15.4), 4.3 TB/s.
template <bool IN_BF16, bool OUT_BF16>
__global__ void __launch_bounds__(256) reduce_nway_scaled_scalar_kernel(const __grid_constant__ NwayArgs a) {
  pdl_begin();
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < a.nbody; i += (unsigned long long)gridDim.x * blockDim.x)
    scaled_element<IN_BF16, OUT_BF16>(a, (long long)i, a.scale);
}

// Calls that do not fetch ahead: two and three sources have kernels of their own (bf16 x3 of 4 M 4.0 -> 3.1 us); from four up
// the loop is as good or better (with the fan-in known the compiler keeps fewer loads in flight: bf16 x8 of 4 M 14.3 us, not
// 12.0).  Eight sources in flight pay from nine up only: they cost registers, and those CTAs (bf16 x4 of 13 M 20.4 us with
// four, 24.7 with eight and 256 threads; x16 of 1 M 5.0 us with eight, 5.5 with four).  Threads behind the end leave: with a
// predicate on each load fp32 x2 -> bf16 of 8 M took 14.8 us, not 12.9.
// Calls that do, us on fresh tensors, not / asking behind all loads with the plain form / so: fp32 x2 of 6 M 11.9 / 11.1 / 10.9,
// -> bf16 10.0 / 9.5 / 8.8; x3 -> bf16 of 5 M 11.4 / 11.0 / 10.9, bf16 x3 of 9 M 11.8 / 11.2 / 10.3; fp32 x4 -> bf16 of 5 M
// 14.4 / 14.2 / 13.1 (four in flight; 14.0 with eight); fp32 x7 -> bf16 of 3 M 14.5 / 14.2 / 13.4, x8 -> bf16 of 6.5 M 33.0 / 32.4 /
// 31.6 (7.0 TB/s), x8 of 2.5 M 14.8 / 13.7 / 13.1; bf16 x4 of 8 M 13.1 / 12.7 / 11.5, x7 of 8 M 20.0 / 19.6 / 18.3, x8 of 4 M 12.1 /
// 11.1 / 10.7 (bf16 with the fan-in known; 11.8, 19.4 and 11.7 without); bf16 x16 of 5 M 26.1 / 25.4 / 25.1.
template <bool IN_BF16, bool OUT_BF16, bool WIDE, int NSRC, int GROUP, int ASK, bool LEAVE>
static cudaError_t launch_k(const NwayArgs& a, unsigned grid, cudaStream_t st) {
  return launch_pdl(reduce_nway_scaled_kernel<IN_BF16, OUT_BF16, WIDE, NSRC, GROUP, ASK, LEAVE>, grid, kThreads, 0, st, a);
}
template <bool IN_BF16, bool OUT_BF16, bool WIDE>
static cudaError_t launch_n(const NwayArgs& a, unsigned grid, cudaStream_t st) {
  if (!a.seam.ahead) {
    switch (a.n) {
      case 2: return launch_k<IN_BF16, OUT_BF16, WIDE, 2, 2, kPlain, true>(a, grid, st);
      case 3: return launch_k<IN_BF16, OUT_BF16, WIDE, 3, 3, kPlain, true>(a, grid, st);
      default: break;
    }
    return a.n <= 8 ? launch_k<IN_BF16, OUT_BF16, WIDE, 0, 4, kPlain, true>(a, grid, st)
                    : launch_k<IN_BF16, OUT_BF16, WIDE, 0, 8, kPlain, true>(a, grid, st);
  }
  constexpr bool some_bf16 = IN_BF16 || OUT_BF16;   // (fp32 to fp32 the leaving form spills: 12.8)
  if (a.n == 2) return launch_k<IN_BF16, OUT_BF16, WIDE, 2, 2, some_bf16 ? 0 : 1, some_bf16>(a, grid, st);
  if (a.n == 3) return launch_k<IN_BF16, OUT_BF16, WIDE, 3, 3, 0, false>(a, grid, st);
  if constexpr (IN_BF16) {
    switch (a.n) {
      case 4: return launch_k<true, OUT_BF16, WIDE, 4, 4, 0, false>(a, grid, st);
      case 5: return launch_k<true, OUT_BF16, WIDE, 5, 5, 0, false>(a, grid, st);
      case 6: return launch_k<true, OUT_BF16, WIDE, 6, 6, 0, false>(a, grid, st);
      case 7: return launch_k<true, OUT_BF16, WIDE, 7, 7, 0, false>(a, grid, st);
      case 8: return launch_k<true, OUT_BF16, WIDE, 8, 8, 0, false>(a, grid, st);
      default: break;
    }
  } else {
    if (a.n == 4) return launch_k<false, OUT_BF16, WIDE, 0, 4, 3, false>(a, grid, st);
    if (a.n > 4 && a.n <= 8) return launch_k<false, OUT_BF16, WIDE, 0, 8, 0, false>(a, grid, st);
  }
  return launch_k<IN_BF16, OUT_BF16, WIDE, 0, 8, kAskLast, true>(a, grid, st);
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
  const unsigned long long grid = nway_grid(a, kThreads);
  if (grid > 0x7fffffffull) return cudaErrorInvalidValue;
  constexpr unsigned out_bytes = (IN_BF16 ? 16 : 8) * (OUT_BF16 ? 2 : 4);
  a.seam = seam_of(a.n > 1 ? (a.n * 32 + out_bytes) * a.nvec : 0, a.n * kThreads * 32, grid);
  return wide ? launch_n<IN_BF16, OUT_BF16, true>(a, (unsigned)grid, st) : launch_n<IN_BF16, OUT_BF16, false>(a, (unsigned)grid, st);
}

cudaError_t launch_scaled(bool in_bf16, bool out_bf16, const NwayArgs& a, unsigned long long len, int sms, cudaStream_t st) {
  if (in_bf16) return out_bf16 ? launch_t<true, true>(a, len, sms, st) : launch_t<true, false>(a, len, sms, st);
  return out_bf16 ? launch_t<false, true>(a, len, sms, st) : launch_t<false, false>(a, len, sms, st);
}

}  // namespace ftk
