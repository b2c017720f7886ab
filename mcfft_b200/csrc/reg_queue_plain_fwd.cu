// reg_queue_plain_fwd.cu -- the one-launch kernel of plain plans, forward.
#define MCFFT_REG_QUEUE_KERNEL
#include "reg_queue.cuh"

namespace mcfft {

const void* reg_queue_plain_fwd() {
  return reinterpret_cast<const void*>(&reg::fft_reg_queue<false>);
}

}  // namespace mcfft
