// reg_pass.cu -- host side of the register pass kernels (see reg_pass.h).
#include "reg_pass.h"

namespace mcfft {

namespace {

constexpr int reg_kind_of(layout::Kind ik, layout::Kind ok) {
  return ik == layout::ROW ? (ok == layout::ROW ? reg::kRR : reg::kRC) : (ok == layout::COL ? reg::kCC : -1);
}

void add_dim(layout::Staging* s, uint64_t extent, uint32_t box, int64_t stride_elems, int cmul, int omul) {
  const int d = s->ndims++;
  s->gdim[d] = extent;
  s->box[d] = box;
  s->gstride_bytes[d] = (uint64_t)stride_elems * s->elem;
  s->cmul[d] = cmul;
  s->omul[d] = omul;
}

// Points along rows: 128-byte rows of E points, row (pos / E) C + c, 128-byte
// swizzle.
layout::Staging row_staging(int L, int C, int elem, int64_t sc, int64_t so, int64_t ncols, int64_t nouter) {
  layout::Staging s;
  s.kind = layout::ROW;
  s.L = L;
  s.C = C;
  s.elem = elem;
  s.E = 128 / elem;
  s.row_bytes = 128;
  s.swz = 7;
  add_dim(&s, s.E, s.E, 1, 0, 0);
  add_dim(&s, ncols, C, sc, C, 0);
  add_dim(&s, L / s.E, L / s.E, s.E, 0, 0);
  if (nouter > 1) add_dim(&s, nouter, 1, so, 0, 1);
  return s;
}

// Columns contiguous, one point row of C columns after another, no swizzle.
// Digits d[0..nd): the point's position is sum digit_i * step_i and the rows
// follow with digit 0 fastest.
layout::Staging col_staging(int L, int C, int elem, const int* count, const int64_t* step, int nd,
                            int64_t sp, int64_t so, int64_t ncols, int64_t nouter) {
  layout::Staging s;
  s.kind = layout::COL;
  s.L = L;
  s.C = C;
  s.elem = elem;
  s.E = C;
  s.row_bytes = C * elem;
  s.swz = 0;
  add_dim(&s, ncols, C, 1, C, 0);
  for (int i = 0; i < nd; ++i)
    if (count[i] > 1) add_dim(&s, count[i], count[i], step[i] * sp, 0, 0);
  if (nouter > 1) add_dim(&s, nouter, 1, so, 0, 1);
  // the kernels' copies are of three to five dimensions
  while (s.ndims < 3) add_dim(&s, 1, 1, L * sp, 0, 0);
  return s;
}

__global__ void k_gen_reg_twiddles(float* dst, int L, int NV, int mode, int sign, double scale) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int R1 = L / NV, n = mode == 2 ? L / 2 : L;
  if (i >= n) return;
  const int v = i % NV, k = i / NV;
  float c[2], s[2];
  for (int u = 0; u < 2; ++u) {
    const int kk = mode == 2 ? 2 * k + u : k;
    double ds, dc;
    sincospi(2.0 * (double)((kk % R1) * v) / (double)L, &ds, &dc);
    c[u] = (float)(scale * dc);
    s[u] = (float)(scale * sign * ds);
  }
  if (mode == 0) reinterpret_cast<float2*>(dst)[i] = make_float2(c[0], s[0]);
  else reinterpret_cast<float4*>(dst)[i] = make_float4(c[0], c[1], s[0], s[1]);
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
  const int lo = k.L < 256 ? k.L : 256;  // a box spans at most 256 points per dimension
  const int nat[2] = {lo, k.L / lo};
  const int64_t nat_step[2] = {1, lo};
  *in = ik == layout::ROW ? row_staging(k.L, k.C, in_elem, in_sc, in_so, ncols, nouter)
                          : col_staging(k.L, k.C, in_elem, nat, nat_step, 2, in_sp, in_so, ncols, nouter);
  if (ok == layout::ROW) {
    *out = row_staging(k.L, k.C, out_elem, out_sc, out_so, ncols, nouter);
  } else if (ik == layout::ROW) {
    *out = col_staging(k.L, k.C, out_elem, nat, nat_step, 2, out_sp, out_so, ncols, nouter);
  } else {
    // digit-reversed tile: rows [k1 high][k2][k1 low], X[k1 + R1 k2]
    const int R1 = k.R, R2 = k.L / k.R, h = k.reg_h;
    const int dig[3] = {1 << h, R2, R1 >> h};
    const int64_t step[3] = {1, R1, int64_t(1) << h};
    *out = col_staging(k.L, k.C, out_elem, dig, step, 3, out_sp, out_so, ncols, nouter);
  }
}

cudaError_t gen_reg_twiddles(void* dst, int L, int NV, int mode, int sign, double scale,
                             cudaStream_t st) {
  const int n = mode == 2 ? L / 2 : L, threads = 256;
  k_gen_reg_twiddles<<<(n + threads - 1) / threads, threads, 0, st>>>(static_cast<float*>(dst), L, NV, mode,
                                                                      sign, scale);
  return cudaGetLastError();
}

}  // namespace mcfft
