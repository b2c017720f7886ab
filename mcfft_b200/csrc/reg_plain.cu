// reg_plain.cu -- plain-form (FP16) register pass kernels, 16K-point tiles
// (4096 points for small batches of rows):
// 64 and 128 points as two register phases (RegPass), 256 to 1024 and rows of
// 2048 and 4096 with the radix-16 stages on the tensor cores (MmaPass,
// Mma2048, Mma4096).
#include "reg_pass.h"

namespace mcfft {

const std::vector<TileKernel>& reg_registry_plain() {
  static const std::vector<TileKernel> v = {
      make_reg<64, 8, 8, 16384, true, true, reg::kRR, false>(),
      make_reg<128, 8, 16, 16384, true, true, reg::kRR, false>(),
      make_reg<64, 8, 8, 16384, true, true, reg::kRC, false>(),
      make_reg<128, 8, 16, 16384, true, true, reg::kRC, false>(),
      make_reg<64, 8, 8, 16384, true, true, reg::kCC, false>(),
      make_reg<128, 16, 8, 16384, true, true, reg::kCC, false>(),
      make_reg<64, 8, 8, 16384, true, true, reg::kCC, true>(),
      make_reg<128, 16, 8, 16384, true, true, reg::kCC, true>(),
      make_mma<256, reg::kRR, false>(),
      make_mma<512, reg::kRR, false>(),
      make_mma<1024, reg::kRR, false>(),
      make_mma<256, reg::kRC, false>(),
      make_mma<512, reg::kRC, false>(),
      make_mma<1024, reg::kRC, false>(),
      make_mma<256, reg::kCC, false>(),
      make_mma<512, reg::kCC, false>(),
      make_mma<1024, reg::kCC, false>(),
      make_mma<256, reg::kCC, true>(),
      make_mma<512, reg::kCC, true>(),
      make_mma<1024, reg::kCC, true>(),
      make_reg<64, 8, 8, 4096, true, true, reg::kRR, false>(),
      make_reg<128, 8, 16, 4096, true, true, reg::kRR, false>(),
      make_mma<256, reg::kRR, false, 4096>(),
      make_mma<512, reg::kRR, false, 4096>(),
      make_mma<1024, reg::kRR, false, 4096>(),
      make_mma_rows<reg::Mma4096<false>, reg::Mma4096<true>>(),
      make_mma_rows<reg::Mma4096<false, 16384>, reg::Mma4096<true, 16384>>(),
      make_mma_rows<reg::Mma2048<false>, reg::Mma2048<true>>()};
  return v;
}

}  // namespace mcfft
