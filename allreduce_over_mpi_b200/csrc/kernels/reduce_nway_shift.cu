// Single-GPU n-way reduction of vectors that do not start at the same offset from a 32-byte boundary.
//
// Slices of flat buffers start wherever the previous parameter ended, so the sources and the result may each
// lie at another phase.  The body is cut on the RESULT's 16-byte boundaries; a source whose bytes lie `shift`
// bytes behind a boundary there is read with aligned 16-byte loads, and each lane puts its vector together from
// its own load and its right neighbour's (a warp shuffle; lane 31 loads the one vector more).  Memory bounds the
// kernel: every byte is still read once, where the one-element loads this replaces moved 4 bytes an instruction.
// The host keeps all loads inside the vectors (layout_shift in nway_layout.h).  Fetching ahead (pdl.cuh) gives it nothing:
// fp32 x5 of 4 M 18.4 us without, 18.5 with, bf16 x8 of 4 M 14.7 and 15.0.
//
// Where all sources lie at one phase and only the result at another (views summed into a new tensor), the second
// kernel keeps 256-bit loads on the sources' boundaries and moves the RESULT across: one shuffle step per 32 bytes of
// result instead of one per source.
#include <type_traits>

#include "pdl.cuh"
#include "reduce_nway.cuh"
#include "vec.cuh"

namespace ftk {

// 16 bytes from byte `shift` of the 32 in lo, hi.  `shift` is the same for the whole grid.
__device__ __forceinline__ uint4 join(uint4 lo, uint4 hi, uint32_t shift) {
  const uint32_t bits = (shift & 3) * 8;
  uint32_t w0, w1, w2, w3, w4;
  switch (shift >> 2) {
    case 0: w0 = lo.x; w1 = lo.y; w2 = lo.z; w3 = lo.w; w4 = hi.x; break;
    case 1: w0 = lo.y; w1 = lo.z; w2 = lo.w; w3 = hi.x; w4 = hi.y; break;
    case 2: w0 = lo.z; w1 = lo.w; w2 = hi.x; w3 = hi.y; w4 = hi.z; break;
    default: w0 = lo.w; w1 = hi.x; w2 = hi.y; w3 = hi.z; w4 = hi.w; break;
  }
  return make_uint4(__funnelshift_r(w0, w1, bits), __funnelshift_r(w1, w2, bits), __funnelshift_r(w2, w3, bits), __funnelshift_r(w3, w4, bits));
}

template <int POL, int UNROLL, int GROUP, int THREADS>
__global__ void __launch_bounds__(THREADS) reduce_nway_shift_kernel(const __grid_constant__ NwayArgs a) {
  using P = typename PolById<POL>::type;
  const unsigned long long base = (unsigned long long)blockIdx.x * THREADS * UNROLL + threadIdx.x;
  pdl_begin();
  const bool last_lane = (threadIdx.x & 31) == 31;
  typename P::Acc acc[UNROLL];
  for (int k0 = 0; k0 < a.n; k0 += GROUP) {
    uint4 lo[GROUP][UNROLL], ex[GROUP][UNROLL];
#pragma unroll
    for (int g = 0; g < GROUP; ++g)
      if (k0 + g < a.n) {
        const uint32_t shift = a.shift[k0 + g];
        const uint4* p = (const uint4*)((const unsigned char*)a.src[k0 + g] - shift);
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
          const unsigned long long i = base + u * THREADS;
          // vector nvec exists for a shifted source: the last result takes part of it
          lo[g][u] = i < a.nvec || (shift && i == a.nvec) ? ld_stream(p + i) : make_uint4(0, 0, 0, 0);
          ex[g][u] = shift && last_lane && i < a.nvec ? ld_stream(p + i + 1) : make_uint4(0, 0, 0, 0);
        }
      }
#pragma unroll
    for (int g = 0; g < GROUP; ++g)
      if (k0 + g < a.n) {
        const uint32_t shift = a.shift[k0 + g];
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
          uint4 v = lo[g][u];
          if (shift) {
            uint4 hi;
            hi.x = __shfl_down_sync(~0u, v.x, 1); hi.y = __shfl_down_sync(~0u, v.y, 1);
            hi.z = __shfl_down_sync(~0u, v.z, 1); hi.w = __shfl_down_sync(~0u, v.w, 1);
            v = join(v, last_lane ? ex[g][u] : hi, shift);
          }
          if (k0 + g == 0) P::init(acc[u], v);
          else P::add(acc[u], v);
        }
      }
  }
#pragma unroll
  for (int u = 0; u < UNROLL; ++u)
    if (base + u * THREADS < a.nvec) st_vec_cs((uint4*)a.dst + base + u * THREADS, P::fin(acc[u]));
  if (a.edge && blockIdx.x == gridDim.x - 1) reduce_edges<POL, ScalarOp>(a);
}

// 32 bytes from byte `shift` of the 64 in lo, hi.  `shift` is the same for the whole grid.
__device__ __forceinline__ void join32(const uint32_t (&lo)[8], const uint32_t (&hi)[8], uint32_t shift, uint32_t (&out)[8]) {
  const uint32_t bits = (shift & 3) * 8;
  auto from = [&](auto words) {
    constexpr int W = decltype(words)::value;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t a = W + k < 8 ? lo[(W + k) & 7] : hi[(W + k) & 7], b = W + k + 1 < 8 ? lo[(W + k + 1) & 7] : hi[(W + k + 1) & 7];
      out[k] = __funnelshift_r(a, b, bits);
    }
  };
  switch (shift >> 2) {
    case 0: from(std::integral_constant<int, 0>{}); break;
    case 1: from(std::integral_constant<int, 1>{}); break;
    case 2: from(std::integral_constant<int, 2>{}); break;
    case 3: from(std::integral_constant<int, 3>{}); break;
    case 4: from(std::integral_constant<int, 4>{}); break;
    case 5: from(std::integral_constant<int, 5>{}); break;
    case 6: from(std::integral_constant<int, 6>{}); break;
    default: from(std::integral_constant<int, 7>{}); break;
  }
}

// A warp sums 32 units of 32 bytes on the sources' boundaries and stores the 31 units of the result between them; the
// next warp sums the last one again (a hit in L2).  a.nvec: units of the result; shift[0]: bytes by which it lies behind
// the sources' boundaries.  bf16 x8 of 4 M, sources one element off: 14.3 us by the kernel above, 11.2 here, 10.1 in a row
// with fetching ahead (pdl.cuh); the edges are the first CTA's then, which is not the last to end.  All CTAs ask for the
// successor: they do enough for that not to count (fp32 x3 of 5 M 10.35 us, 10.45 if only the last ones do).
template <int POL, int GROUP>
__global__ void __launch_bounds__(kRealignThreads) reduce_nway_realign_kernel(const __grid_constant__ NwayArgs a) {
  using P = typename PolById<POL>::type;
  const uint32_t lane = threadIdx.x & 31, shift = a.shift[0];
  const unsigned long long i = (unsigned long long)blockIdx.x * kRealignPerCta + threadIdx.x / 32 * 31 + lane;
  const bool ok = i <= a.nvec;   // one unit more than the result has
  if (blockIdx.x < a.seam.ahead && ok && !(lane & 3))
    for (int k = 0; k < a.n; ++k) l2_ahead((const unsigned char*)a.src[k] - shift + i * 32);
  pdl_begin();
  typename P::Acc al, ah;
  for (int k0 = 0; k0 < a.n; k0 += GROUP) {
    uint4 lo[GROUP], hi[GROUP];
#pragma unroll
    for (int g = 0; g < GROUP; ++g)
      if (ok && k0 + g < a.n) {
        const unsigned char* p = (const unsigned char*)a.src[k0 + g] - shift + i * 32;
        asm volatile("ld.global.L1::no_allocate.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(lo[g].x), "=r"(lo[g].y), "=r"(lo[g].z), "=r"(lo[g].w), "=r"(hi[g].x), "=r"(hi[g].y), "=r"(hi[g].z), "=r"(hi[g].w)
                     : "l"(p) : "memory");
      }
    if (k0 + GROUP >= a.n) pdl_next(a.seam.ahead);
#pragma unroll
    for (int g = 0; g < GROUP; ++g)
      if (k0 + g < a.n) {
        if (k0 + g == 0) { P::init(al, lo[g]); P::init(ah, hi[g]); }
        else { P::add(al, lo[g]); P::add(ah, hi[g]); }
      }
  }
  const uint4 l = P::fin(al), h = P::fin(ah);
  const uint32_t mine[8] = {l.x, l.y, l.z, l.w, h.x, h.y, h.z, h.w};
  uint32_t next[8], w[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) next[k] = __shfl_down_sync(~0u, mine[k], 1);
  join32(mine, next, shift, w);
  if (lane < 31 && i < a.nvec)
    asm volatile("st.global.L1::no_allocate.L2::evict_first.v8.u32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"l"((unsigned char*)a.dst + i * 32), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
  if (a.edge && blockIdx.x == (a.seam.ahead ? 0 : gridDim.x - 1)) reduce_edges<POL, ScalarOp>(a);
}

template <int POL, int UNROLL, int GROUP, int THREADS>
static cudaError_t launch_t(const NwayArgs& a, cudaStream_t st) {
  const unsigned long long grid = nway_grid(a, THREADS * UNROLL);
  if (grid > 0x7fffffffull || grid == 0) return cudaErrorInvalidValue;
  return launch_pdl(reduce_nway_shift_kernel<POL, UNROLL, GROUP, THREADS>, (unsigned)grid, THREADS, 0, st, a);
}
// Long vectors want many small CTAs with few registers, two vectors of two sources at a time: with 256 threads and two
// vectors of four sources 100 MB of fp32 x4 took 117 us, so they take 77 (6.5 TB/s).  Below 3 MB the chip is not full and
// one vector of four sources at a time has the shorter chain: fp32 x8 of 2 MB 5.1 us against 6.0.  (18 shapes measured,
// 64 KB to 100 MB, 2 to 16 sources.)
template <int POL>
static cudaError_t launch_t(const NwayArgs& a, bool realign, cudaStream_t st) {
  if (realign) {
    NwayArgs b = a;
    b.seam = seam_of((a.n + 1) * a.nvec * 32, a.n * kRealignPerCta * 32, body_ctas(a, kRealignPerCta));
    const unsigned long long grid = nway_grid(b, kRealignPerCta);
    if (grid > 0x7fffffffull) return cudaErrorInvalidValue;
    return a.n <= 8 ? launch_pdl(reduce_nway_realign_kernel<POL, 4>, (unsigned)grid, kRealignThreads, 0, st, b)
                    : launch_pdl(reduce_nway_realign_kernel<POL, 8>, (unsigned)grid, kRealignThreads, 0, st, b);
  }
  return shift_long(a) ? launch_t<POL, 2, 2, 64>(a, st) : launch_t<POL, 1, 4, 128>(a, st);
}

cudaError_t launch_shift(int pol, const NwayArgs& a, bool realign, cudaStream_t st) {
  switch (pol) {
    case POL_ADD8: return launch_t<POL_ADD8>(a, realign, st);
    case POL_ADD16: return launch_t<POL_ADD16>(a, realign, st);
    case POL_ADD32: return launch_t<POL_ADD32>(a, realign, st);
    case POL_ADD64: return launch_t<POL_ADD64>(a, realign, st);
    case POL_OR: return launch_t<POL_OR>(a, realign, st);
    case POL_AND: return launch_t<POL_AND>(a, realign, st);
    case POL_F32: return launch_t<POL_F32>(a, realign, st);
    case POL_F64: return launch_t<POL_F64>(a, realign, st);
    case POL_BF16: return launch_t<POL_BF16>(a, realign, st);
    case POL_F16: return launch_t<POL_F16>(a, realign, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace ftk
