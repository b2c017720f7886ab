// fft_small.cuh -- a row pass over contiguous transforms without TMA: one tile
// of 4096 points per CTA, copied in with 16-byte asynchronous copies and out
// with 16-byte stores.
//
// What bounds it: latency.  A small exec is one or two tiles per SM, and what
// it takes is the chain launch, load, phases, store.  Through TMA (fft_reg.cuh)
// that chain holds a barrier's initialisation, the fetch of two tensor maps,
// and the hand-over of the tile to and from the copying warp; here the tables
// and the tile are requested by the first instructions of all warps and one
// block barrier separates them from the phases.  Measured, back-to-back execs,
// with TMA / without: 1024 x 8 6.15 / 4.10 us, 4096 x 256 8.2 / 6.15 us (FP16
// in, FP32 out too), 512 x 9001 14.3 / 12.3 us.
//
// Why 16-byte copies through shared memory: the phases' own accesses are 16
// bytes of a swizzled layout, so a straight copy keeps them and needs only the
// inverse of TMA's placement (in_map, out_map).  The FP32 4096-point routine
// reads and writes half-warp lines by itself: it takes its first operands from
// global memory and stores its last results there.
#pragma once
#include "fft_mma.cuh"
#include "fft_reg.cuh"
#include "fft_rows.cuh"

namespace mcfft {

struct SmallArgs {
  const void* in;
  void* out;
  const float4* tw;
  const uint4* bmat;
  uint64_t points;  // of the whole pass
};

namespace reg {

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

template <class P>
struct IsReg4096 : std::false_type {};
template <bool IN16, bool INV>
struct IsReg4096<Reg4096<IN16, INV>> : std::true_type {};

template <class P>
__global__ void __launch_bounds__(P::T, P::MINB) fft_small(const __grid_constant__ SmallArgs a) {
  static_assert(P::KIND == kRR && !P::POST && P::NG == 1, "contiguous rows");
  constexpr int T = P::T, IN = P::TP * P::EI, OUT = P::TP * P::EO;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_u = sm100::smem_u32(smem_raw);
  const uint32_t base_u = (raw_u + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base_u - raw_u);
  const int t = threadIdx.x;
  const uint64_t first = (uint64_t)blockIdx.x * P::TP;
  const uint32_t n = a.points - first < P::TP ? (uint32_t)(a.points - first) : P::TP;  // whole transforms
  for (int i = t; i < P::TWB / 16; i += T) cp_async16(base_u + P::BUF + 16 * i, a.tw + i, true);
  sm100::grid_dep_wait();
  const uint8_t* in = static_cast<const uint8_t*>(a.in) + first * P::EI;
  uint8_t* out = static_cast<uint8_t*>(a.out) + first * P::EO;
  if constexpr (IsReg4096<P>::value) {
    sm100::grid_dep_launch();
    P::template phases<true>(base_u, base_u + P::BUF, t, in, out);
  } else {
#pragma unroll
    for (int i = 0; i < IN / 16 / T; ++i) {
      const uint32_t o = (i * T + t) * 16, g = P::in_map(o);
      const bool valid = g < n * P::EI;
      cp_async16(base_u + o, in + (valid ? g : 0), valid);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    const typename P::State st(a, t);
    sm100::grid_dep_launch();
    __syncthreads();
    P::run(a, st, base_u, base_u + P::BUF, t, 0, Sync<T>{1});
    __syncthreads();
#pragma unroll 8
    for (int i = 0; i < OUT / 16 / T; ++i) {
      const uint32_t o = (i * T + t) * 16, g = P::out_map(o);
      if (g < n * P::EO) *reinterpret_cast<uint4*>(out + g) = *reinterpret_cast<const uint4*>(smem + o);
    }
  }
}

template <class P>
constexpr int small_smem() {
  return P::BUF + P::TWB + 1024;
}

}  // namespace reg
}  // namespace mcfft
