// reg_plain.cu -- plain-form (FP16) register pass kernels: 16K-point tiles,
// and 8K-point ones for passes with too few tiles to fill the SMs.
//
// The radices of a length are chosen so that the vectors a thread holds share
// their twiddles (RegPass): 32 x 16 and 32 x 32 in column passes, where a
// tile has few columns, 16 x 32 in row passes, whose lanes run along 32
// consecutive points.
#include "reg_pass.h"

namespace mcfft {

#define MCFFT_REG_PLAIN(TP, R256)                                                          \
  make_reg<64, 8, 8, TP, true, true, reg::kRR, false>(),                                   \
      make_reg<128, 8, 16, TP, true, true, reg::kRR, false>(),                             \
      make_reg<256, 16, 16, TP, true, true, reg::kRR, false>(),                            \
      make_reg<512, 16, 32, TP, true, true, reg::kRR, false>(),                            \
      make_reg<1024, 32, 32, TP, true, true, reg::kRR, false>(),                           \
      make_reg<64, 8, 8, TP, true, true, reg::kRC, false>(),                               \
      make_reg<128, 8, 16, TP, true, true, reg::kRC, false>(),                             \
      make_reg<256, 16, 16, TP, true, true, reg::kRC, false>(),                            \
      make_reg<512, 16, 32, TP, true, true, reg::kRC, false>(),                            \
      make_reg<1024, 32, 32, TP, true, true, reg::kRC, false>(),                           \
      make_reg<64, 8, 8, TP, true, true, reg::kCC, false>(),                               \
      make_reg<128, 16, 8, TP, true, true, reg::kCC, false>(),                             \
      make_reg<256, R256, 256 / R256, TP, true, true, reg::kCC, false>(),                  \
      make_reg<512, 32, 16, TP, true, true, reg::kCC, false>(),                            \
      make_reg<1024, 32, 32, TP, true, true, reg::kCC, false>(),                           \
      make_reg<64, 8, 8, TP, true, true, reg::kCC, true>(),                                \
      make_reg<128, 16, 8, TP, true, true, reg::kCC, true>(),                              \
      make_reg<256, R256, 256 / R256, TP, true, true, reg::kCC, true>(),                   \
      make_reg<512, 32, 16, TP, true, true, reg::kCC, true>(),                             \
      make_reg<1024, 32, 32, TP, true, true, reg::kCC, true>()

const std::vector<TileKernel>& reg_registry_plain() {
  static const std::vector<TileKernel> v = {MCFFT_REG_PLAIN(16384, 16)};
  return v;
}

}  // namespace mcfft
