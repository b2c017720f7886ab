// reg_staging.h -- where TMA places a tile of a register pass in shared memory
// and where it takes the result from: tensor-map dimensions of the layouts
// that RegPass (fft_reg.cuh) and MmaPass (fft_mma.cuh) address.
#pragma once
#include <vector>

#include "layout.h"

namespace mcfft {

// Shape of a variant: R the first radix (RegPass) or the last (MmaPass), h
// RegPass::h.
struct RegShape {
  int L, R, C, h;
  bool mma;
};

inline void reg_add_dim(layout::Staging* s, uint64_t extent, uint32_t box, int64_t stride_elems, int cmul,
                        int omul) {
  const int d = s->ndims++;
  s->gdim[d] = extent;
  s->box[d] = box;
  s->gstride_bytes[d] = (uint64_t)stride_elems * s->elem;
  s->cmul[d] = cmul;
  s->omul[d] = omul;
}

// Points along rows: 128-byte rows of E points with the 128-byte swizzle.
// by_col: a column's rows follow one another (row c (L / E) + pos / E), else
// the columns' (row (pos / E) C + c).
inline layout::Staging reg_row_staging(int L, int C, int elem, bool by_col, int64_t sc, int64_t so,
                                       int64_t ncols, int64_t nouter) {
  layout::Staging s;
  s.kind = layout::ROW;
  s.L = L;
  s.C = C;
  s.elem = elem;
  s.E = 128 / elem;
  s.row_bytes = 128;
  s.swz = 7;
  reg_add_dim(&s, s.E, s.E, 1, 0, 0);
  if (by_col) reg_add_dim(&s, L / s.E, L / s.E, s.E, 0, 0);
  reg_add_dim(&s, ncols, C, sc, C, 0);
  if (!by_col) reg_add_dim(&s, L / s.E, L / s.E, s.E, 0, 0);
  if (nouter > 1) reg_add_dim(&s, nouter, 1, so, 0, 1);
  return s;
}

// Columns contiguous: one point row after another.  The position is the sum
// of digit_i * step_i and the rows follow with digit 0 fastest.  swizzled:
// rows of at most 32 columns under the swizzle of their width, wider tiles in
// blocks of 32 columns.
inline layout::Staging reg_col_staging(int L, int C, int elem, bool swizzled, const int* count,
                                       const int64_t* step, int nd, int64_t sp, int64_t so, int64_t ncols,
                                       int64_t nouter) {
  layout::Staging s;
  s.kind = layout::COL;
  s.L = L;
  s.C = C;
  s.elem = elem;
  const int blocks = swizzled && C > 32 ? C / 32 : 1;
  s.E = C / blocks;
  s.row_bytes = s.E * elem;
  s.swz = !swizzled ? 0 : s.row_bytes >= 128 ? 7 : s.row_bytes == 64 ? 3 : 0;
  reg_add_dim(&s, blocks > 1 && ncols > s.E ? s.E : ncols, s.E, 1, blocks > 1 ? 0 : C, 0);
  for (int i = 0; i < nd; ++i)
    if (count[i] > 1) reg_add_dim(&s, count[i], count[i], step[i] * sp, 0, 0);
  if (blocks > 1) reg_add_dim(&s, ncols > s.E ? (ncols + s.E - 1) / s.E : 1, blocks, s.E, blocks, 0);
  if (nouter > 1) reg_add_dim(&s, nouter, 1, so, 0, 1);
  // the kernels' copies are of three to five dimensions
  while (s.ndims < 3) reg_add_dim(&s, 1, 1, L * sp, 0, 0);
  return s;
}

// Rows of 2048 and 4096 points.  Plain: swizzled 128-byte rows of 32 points,
// within a transform row 16 (p / 32 mod B) + p / (32 B) with B = L / 512 (the
// 2048-point output: natural); FP32 exchange: natural order, no swizzle.
inline layout::Staging reg_rows_staging(const RegShape& k, bool out, int elem, int64_t sc, int64_t so,
                                        int64_t ncols, int64_t nouter) {
  layout::Staging s;
  s.kind = layout::ROW;
  s.L = k.L;
  s.C = k.C;
  s.elem = elem;
  s.E = k.mma ? 32 : 256;
  s.row_bytes = s.E * elem;
  s.swz = k.mma ? 7 : 0;
  const int B = k.L / 512;
  reg_add_dim(&s, s.E, s.E, 1, 0, 0);
  if (!k.mma) {
    reg_add_dim(&s, k.L / 256, k.L / 256, 256, 0, 0);
  } else if (out && k.L == 2048) {
    reg_add_dim(&s, 64, 64, 32, 0, 0);
  } else {
    reg_add_dim(&s, 16, 16, 32 * B, 0, 0);
    reg_add_dim(&s, B, B, 32, 0, 0);
  }
  reg_add_dim(&s, ncols, k.C, sc, k.C, 0);
  if (nouter > 1) reg_add_dim(&s, nouter, 1, so, 0, 1);
  return s;
}

// Transforms at unrelated offsets, each copied by itself: box = one
// transform of the row layouts that keep a column's rows together; `tab`
// receives each transform's first 32-point row.  False if the variant's
// layout or an offset does not allow it.
inline bool reg_gather_staging(const RegShape& k, bool out, int elem, const std::vector<int64_t>& offs,
                               layout::Staging* st, std::vector<int32_t>* tab) {
  if (!k.mma || k.L < 256 || elem != 4) return false;
  // positions split as [rows of a box's last dimension][dim 1]: see
  // reg_row_staging, reg_rows_staging
  const bool inner = k.L > 1024 && !(out && k.L == 2048);
  const int rows = inner ? k.L / 512 : k.L / 32, step = 32 * (k.L / 512);
  int64_t last = 0;
  tab->clear();
  for (int64_t o : offs) {
    if (o < 0 || o % 32 || (o + k.L) / 32 >= (int64_t(1) << 31)) return false;
    tab->push_back((int32_t)(o / 32));
    last = o > last ? o : last;
  }
  layout::Staging s;
  s.kind = layout::ROW;
  s.L = k.L;
  s.C = k.C;
  s.elem = elem;
  s.E = 32;
  s.row_bytes = 128;
  s.swz = 7;
  reg_add_dim(&s, 32, 32, 1, 0, 0);
  if (inner) reg_add_dim(&s, 16, 16, step, 0, 0);
  else reg_add_dim(&s, 1, 1, 32, 0, 0);
  reg_add_dim(&s, last / 32 + rows, rows, 32, 0, 0);
  *st = s;
  return true;
}

inline layout::Staging reg_staging_in(const RegShape& k, layout::Kind ik, int elem, int64_t sp, int64_t sc,
                                      int64_t so, int64_t ncols, int64_t nouter) {
  if (k.L > 1024) return reg_rows_staging(k, false, elem, sc, so, ncols, nouter);
  if (ik == layout::ROW) return reg_row_staging(k.L, k.C, elem, k.mma, sc, so, ncols, nouter);
  if (k.mma) {  // rows [v][n1], n = n1 (L / 16) + v
    const int dig[2] = {16, k.L / 16};
    const int64_t step[2] = {k.L / 16, 1};
    return reg_col_staging(k.L, k.C, elem, true, dig, step, 2, sp, so, ncols, nouter);
  }
  const int lo = k.L < 256 ? k.L : 256;  // a box spans at most 256 points per dimension
  const int dig[2] = {lo, k.L / lo};
  const int64_t step[2] = {1, lo};
  return reg_col_staging(k.L, k.C, elem, false, dig, step, 2, sp, so, ncols, nouter);
}

inline layout::Staging reg_staging_out(const RegShape& k, layout::Kind ik, layout::Kind ok, int elem,
                                       int64_t sp, int64_t sc, int64_t so, int64_t ncols, int64_t nouter) {
  if (k.L > 1024) return reg_rows_staging(k, true, elem, sc, so, ncols, nouter);
  if (ok == layout::ROW) return reg_row_staging(k.L, k.C, elem, k.mma, sc, so, ncols, nouter);
  if (k.mma) {  // rows [k1][k3][k2], X[k1 + 16 k2 + 256 k3]
    const int dig[3] = {16, k.R, 16};
    const int64_t step[3] = {16, 256, 1};
    return reg_col_staging(k.L, k.C, elem, true, dig, step, 3, sp, so, ncols, nouter);
  }
  if (ik == layout::ROW) {
    const int lo = k.L < 256 ? k.L : 256;
    const int dig[2] = {lo, k.L / lo};
    const int64_t step[2] = {1, lo};
    return reg_col_staging(k.L, k.C, elem, false, dig, step, 2, sp, so, ncols, nouter);
  }
  // digit-reversed tile: rows [k1 high][k2][k1 low], X[k1 + R1 k2]
  const int dig[3] = {1 << k.h, k.L / k.R, k.R >> k.h};
  const int64_t step[3] = {1, k.R, int64_t(1) << k.h};
  return reg_col_staging(k.L, k.C, elem, false, dig, step, 3, sp, so, ncols, nouter);
}

}  // namespace mcfft
