// reg_pass.h -- host side of the register pass kernels (fft_reg.cuh):
// variant entries, staging descriptions and twiddle tables.
#pragma once
#include "fft_mma.cuh"
#include "fft_reg.cuh"
#include "fft_rows.cuh"
#include "fft_small.cuh"
#include "tile_pass.h"

namespace mcfft {

// Variants by form, each in a translation unit of its own.
const std::vector<TileKernel>& reg_registry_plain();    // reg_plain.cu
const std::vector<TileKernel>& reg_registry_split();    // reg_split.cu
const std::vector<TileKernel>& reg_registry_split16();  // reg_split16.cu

// Register kernel of a pass with points along `ik` in and `ok` out, or null.
const TileKernel* find_reg_kernel(int L, layout::Kind ik, layout::Kind ok, bool posttw, bool split,
                                  int tile_points, bool in16);

// Where TMA places a tile of the variant in shared memory (RegPass::load1_*
// and store2_*), for a pass with the given strides (elements).
void reg_stagings(const TileKernel& k, layout::Kind ik, layout::Kind ok, int in_elem, int out_elem,
                  int64_t in_sp, int64_t in_sc, int64_t in_so, int64_t out_sp, int64_t out_sc,
                  int64_t out_so, int64_t ncols, int64_t nouter, layout::Staging* in,
                  layout::Staging* out);
// The same for transforms at unrelated offsets (reg_staging.h).
bool reg_gather_staging(const TileKernel& k, bool out, int elem, const std::vector<int64_t>& offs,
                        layout::Staging* st, std::vector<int32_t>* tab);

// Phase-1 twiddles W_L^(k v) * scale in the layout of RegPass (at k NV + v: 8
// bytes, or doubled for two columns, 16 bytes); sign -1 forward, +1 inverse.
cudaError_t gen_reg_twiddles(void* dst, int L, int NV, bool doubled, int sign, double scale,
                             cudaStream_t st);

// The kernels without TMA of a 4096-point row tile.
template <class P, class Q>
void add_small(TileKernel* k) {
  if constexpr (P::TP == 4096 && P::KIND == reg::kRR) {
    k->fn_small[0] = reinterpret_cast<const void*>(&reg::fft_small<P>);
    k->fn_small[1] = reinterpret_cast<const void*>(&reg::fft_small<Q>);
    k->small_smem = reg::small_smem<P>();
    k->small_threads = P::T;
  }
}

template <int L, int R1, int R2, int TP, bool IN16, bool OUT16, int KIND, bool POST>
TileKernel make_reg() {
  using P = reg::RegPass<L, R1, R2, TP, IN16, OUT16, KIND, POST, false>;
  using Q = reg::RegPass<L, R1, R2, TP, IN16, OUT16, KIND, POST, true>;
  TileKernel k{reinterpret_cast<const void*>(&reg::fft_reg<P>), L, R1, P::C, POST, !OUT16, P::THREADS,
               P::SMEM_BYTES, 0, TP, IN16};
  k.fn_inv = reinterpret_cast<const void*>(&reg::fft_reg<Q>);
  k.reg_kind = KIND;
  k.reg_h = P::h;
  k.tw_bytes = P::TWB;
  k.tab_bytes = P::TABB;
  k.tw_doubled = P::PK;
  add_small<P, Q>(&k);
  return k;
}

template <int L, int KIND, bool POST, int TP = 16384>
TileKernel make_mma() {
  using P = reg::MmaPass<L, KIND, POST, false, TP>;
  using Q = reg::MmaPass<L, KIND, POST, true, TP>;
  TileKernel k{reinterpret_cast<const void*>(&reg::fft_reg<P>), L, P::R, P::C, POST, false, P::THREADS,
               P::SMEM_BYTES, 0, P::TP, true};
  k.fn_inv = reinterpret_cast<const void*>(&reg::fft_reg<Q>);
  k.reg_kind = KIND;
  k.tw_bytes = P::TWB;
  k.tab_bytes = P::TABB;
  k.mma = true;
  k.fill_tw[0] = &P::fill_twiddles;
  k.fill_tw[1] = &Q::fill_twiddles;
  k.fill_frag[0] = &P::fill_fragments;
  k.fill_frag[1] = &Q::fill_fragments;
  add_small<P, Q>(&k);
  return k;
}

// Rows of 2048 and 4096 points (fft_rows.cuh), plain form.
template <class P, class Q>
TileKernel make_mma_rows() {
  TileKernel k{reinterpret_cast<const void*>(&reg::fft_reg<P>), P::L, P::R, P::C, false, false, P::THREADS,
               P::SMEM_BYTES, 0, P::TP, true};
  k.fn_inv = reinterpret_cast<const void*>(&reg::fft_reg<Q>);
  k.reg_kind = reg::kRR;
  k.tw_bytes = P::TWB;
  k.tab_bytes = P::TABB;
  k.mma = true;
  k.fill_tw[0] = &P::fill_twiddles;
  k.fill_tw[1] = &Q::fill_twiddles;
  k.fill_frag[0] = &P::fill_fragments;
  k.fill_frag[1] = &Q::fill_fragments;
  add_small<P, Q>(&k);
  return k;
}
// 4096-point rows, FP32 exchange.
template <bool IN16>
TileKernel make_reg4096() {
  using P = reg::Reg4096<IN16, false>;
  using Q = reg::Reg4096<IN16, true>;
  TileKernel k{reinterpret_cast<const void*>(&reg::fft_reg<P>), 4096, 16, 1, false, true, P::THREADS,
               P::SMEM_BYTES, 0, P::TP, IN16};
  k.fn_inv = reinterpret_cast<const void*>(&reg::fft_reg<Q>);
  k.reg_kind = reg::kRR;
  k.tw_bytes = P::TWB;
  k.fill_tw[0] = &P::fill_twiddles;
  k.fill_tw[1] = &Q::fill_twiddles;
  add_small<P, Q>(&k);
  return k;
}

}  // namespace mcfft
