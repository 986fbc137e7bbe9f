// Single-GPU n-way reduction of vectors that do not start at the same offset from a 32-byte boundary.
//
// Slices of flat buffers start wherever the previous parameter ended, so the sources and the result may each
// lie at another phase.  The body is cut on the RESULT's 16-byte boundaries; a source whose bytes lie `shift`
// bytes behind a boundary there is read with aligned 16-byte loads, and each lane puts its vector together from
// its own load and its right neighbour's (a warp shuffle; lane 31 loads the one vector more).  Memory bounds the
// kernel: every byte is still read once, where the one-element loads this replaces moved 4 bytes an instruction.
// The host keeps all loads inside the vectors (layout_shift in reduce_nway.cu).
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
  pdl_begin();
  const unsigned long long base = (unsigned long long)blockIdx.x * THREADS * UNROLL + threadIdx.x;
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

template <int POL, int UNROLL, int GROUP, int THREADS>
static cudaError_t launch_t(const NwayArgs& a, cudaStream_t st) {
  const unsigned long long grid = (a.nvec + THREADS * UNROLL - 1) / (THREADS * UNROLL) + (a.edge != 0);
  if (grid > 0x7fffffffull || grid == 0) return cudaErrorInvalidValue;
  return launch_pdl(reduce_nway_shift_kernel<POL, UNROLL, GROUP, THREADS>, (unsigned)grid, THREADS, 0, st, a);
}
// Long vectors want many small CTAs with few registers, two vectors of two sources at a time: with 256 threads and two
// vectors of four sources 100 MB of fp32 x4 took 117 us, so they take 77 (6.5 TB/s).  Below 3 MB the chip is not full and
// one vector of four sources at a time has the shorter chain: fp32 x8 of 2 MB 5.1 us against 6.0.  (18 shapes measured,
// 64 KB to 100 MB, 2 to 16 sources.)
template <int POL>
static cudaError_t launch_t(const NwayArgs& a, cudaStream_t st) {
  return a.nvec >= (3u << 20) / 16 ? launch_t<POL, 2, 2, 64>(a, st) : launch_t<POL, 1, 4, 128>(a, st);
}

cudaError_t launch_shift(int pol, const NwayArgs& a, cudaStream_t st) {
  switch (pol) {
    case POL_ADD8: return launch_t<POL_ADD8>(a, st);
    case POL_ADD16: return launch_t<POL_ADD16>(a, st);
    case POL_ADD32: return launch_t<POL_ADD32>(a, st);
    case POL_ADD64: return launch_t<POL_ADD64>(a, st);
    case POL_OR: return launch_t<POL_OR>(a, st);
    case POL_AND: return launch_t<POL_AND>(a, st);
    case POL_F32: return launch_t<POL_F32>(a, st);
    case POL_F64: return launch_t<POL_F64>(a, st);
    case POL_BF16: return launch_t<POL_BF16>(a, st);
    case POL_F16: return launch_t<POL_F16>(a, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace ftk
