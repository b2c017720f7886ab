// reg_pass.cu -- host side of the register pass kernels (see reg_pass.h).
#include "reg_pass.h"
#include "reg_staging.h"

namespace mcfft {

namespace {

constexpr int reg_kind_of(layout::Kind ik, layout::Kind ok) {
  return ik == layout::ROW ? (ok == layout::ROW ? reg::kRR : reg::kRC) : (ok == layout::COL ? reg::kCC : -1);
}

__global__ void k_gen_reg_twiddles(float* dst, int L, int NV, bool doubled, int sign, double scale) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= L) return;
  const int v = i % NV, k = i / NV;
  double ds, dc;
  sincospi(2.0 * (double)(k * v) / (double)L, &ds, &dc);
  const float c = (float)(scale * dc), s = (float)(scale * sign * ds);
  if (doubled) reinterpret_cast<float4*>(dst)[i] = make_float4(c, c, s, s);
  else reinterpret_cast<float2*>(dst)[i] = make_float2(c, s);
}

}  // namespace

const TileKernel* find_reg_kernel(int L, layout::Kind ik, layout::Kind ok, bool posttw, bool split,
                                  int tile_points, bool in16) {
  const int kind = reg_kind_of(ik, ok);
  if (kind < 0) return nullptr;
  const auto& reg = !split ? reg_registry_plain() : in16 ? reg_registry_split16() : reg_registry_split();
  for (const auto& k : reg)
    if (k.L == L && k.reg_kind == kind && k.posttw == posttw && k.tile_points == tile_points) return &k;
  return nullptr;
}

void reg_stagings(const TileKernel& k, layout::Kind ik, layout::Kind ok, int in_elem, int out_elem,
                  int64_t in_sp, int64_t in_sc, int64_t in_so, int64_t out_sp, int64_t out_sc,
                  int64_t out_so, int64_t ncols, int64_t nouter, layout::Staging* in,
                  layout::Staging* out) {
  const RegShape s{k.L, k.R, k.C, k.reg_h, k.mma};
  *in = reg_staging_in(s, ik, in_elem, in_sp, in_sc, in_so, ncols, nouter);
  *out = reg_staging_out(s, ik, ok, out_elem, out_sp, out_sc, out_so, ncols, nouter);
}

bool reg_gather_staging(const TileKernel& k, bool out, int elem, const std::vector<int64_t>& offs,
                        layout::Staging* st, std::vector<int32_t>* tab) {
  return reg_gather_staging(RegShape{k.L, k.R, k.C, k.reg_h, k.mma}, out, elem, offs, st, tab);
}

cudaError_t gen_reg_twiddles(void* dst, int L, int NV, bool doubled, int sign, double scale,
                             cudaStream_t st) {
  const int threads = 256;
  k_gen_reg_twiddles<<<(L + threads - 1) / threads, threads, 0, st>>>(static_cast<float*>(dst), L, NV, doubled,
                                                                      sign, scale);
  return cudaGetLastError();
}

}  // namespace mcfft
