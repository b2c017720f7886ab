// reg_split16.cu -- split-form register pass kernels with FP16 input (the
// first pass of a transform), FP32 exchange and output.
#include "reg_pass.h"

namespace mcfft {

const std::vector<TileKernel>& reg_registry_split16() {
  static const std::vector<TileKernel> v = {
      make_reg<64, 8, 8, 8192, true, false, reg::kRR, false>(),
      make_reg<128, 8, 16, 8192, true, false, reg::kRR, false>(),
      make_reg<256, 16, 16, 8192, true, false, reg::kRR, false>(),
      make_reg<512, 16, 32, 8192, true, false, reg::kRR, false>(),
      make_reg<1024, 32, 32, 8192, true, false, reg::kRR, false>(),
      make_reg<64, 8, 8, 8192, true, false, reg::kCC, true>(),
      make_reg<128, 8, 16, 8192, true, false, reg::kCC, true>(),
      make_reg<256, 16, 16, 8192, true, false, reg::kCC, true>(),
      make_reg<512, 32, 16, 8192, true, false, reg::kCC, true>(),
      make_reg<1024, 32, 32, 8192, true, false, reg::kCC, true>(),
      // small batches of rows
      make_reg<64, 8, 8, 4096, true, false, reg::kRR, false>(),
      make_reg<128, 8, 16, 4096, true, false, reg::kRR, false>(),
      make_reg<256, 16, 16, 4096, true, false, reg::kRR, false>(),
      make_reg<512, 16, 32, 4096, true, false, reg::kRR, false>(),
      make_reg4096<true>()};
  return v;
}

}  // namespace mcfft
