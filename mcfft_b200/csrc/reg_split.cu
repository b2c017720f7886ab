// reg_split.cu -- split-form register pass kernels with FP32 input: 8K-point
// tiles (64 KB of FP32, as the plain form's 16K points of FP16).
#include "reg_pass.h"

namespace mcfft {

const std::vector<TileKernel>& reg_registry_split() {
  static const std::vector<TileKernel> v = {
      make_reg<64, 8, 8, 8192, false, false, reg::kRR, false>(),
      make_reg<128, 8, 16, 8192, false, false, reg::kRR, false>(),
      make_reg<256, 16, 16, 8192, false, false, reg::kRR, false>(),
      make_reg<512, 16, 32, 8192, false, false, reg::kRR, false>(),
      make_reg<1024, 32, 32, 8192, false, false, reg::kRR, false>(),
      make_reg<64, 8, 8, 8192, false, false, reg::kRC, false>(),
      make_reg<128, 8, 16, 8192, false, false, reg::kRC, false>(),
      make_reg<256, 16, 16, 8192, false, false, reg::kRC, false>(),
      make_reg<512, 16, 32, 8192, false, false, reg::kRC, false>(),
      make_reg<1024, 32, 32, 8192, false, false, reg::kRC, false>(),
      make_reg<64, 8, 8, 8192, false, false, reg::kCC, false>(),
      make_reg<128, 8, 16, 8192, false, false, reg::kCC, false>(),
      make_reg<256, 16, 16, 8192, false, false, reg::kCC, false>(),
      make_reg<512, 32, 16, 8192, false, false, reg::kCC, false>(),
      make_reg<1024, 32, 32, 8192, false, false, reg::kCC, false>(),
      make_reg<64, 8, 8, 8192, false, false, reg::kCC, true>(),
      make_reg<128, 8, 16, 8192, false, false, reg::kCC, true>(),
      make_reg<256, 16, 16, 8192, false, false, reg::kCC, true>(),
      make_reg<512, 32, 16, 8192, false, false, reg::kCC, true>(),
      make_reg<1024, 32, 32, 8192, false, false, reg::kCC, true>(),
      // small batches of rows
      make_reg<64, 8, 8, 4096, false, false, reg::kRR, false>(),
      make_reg<128, 8, 16, 4096, false, false, reg::kRR, false>(),
      make_reg<256, 16, 16, 4096, false, false, reg::kRR, false>(),
      make_reg<512, 16, 32, 4096, false, false, reg::kRR, false>(),
      make_reg4096<false>()};
  return v;
}

}  // namespace mcfft
