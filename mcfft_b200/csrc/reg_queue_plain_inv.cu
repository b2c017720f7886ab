// reg_queue_plain_inv.cu -- the one-launch kernel of plain plans, inverse.
#define MCFFT_REG_QUEUE_KERNEL
#include "reg_queue.cuh"

namespace mcfft {

const void* reg_queue_plain_inv() {
  return reinterpret_cast<const void*>(&reg::fft_reg_queue<true>);
}

}  // namespace mcfft
