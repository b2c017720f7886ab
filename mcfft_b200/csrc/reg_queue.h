// reg_queue.h -- host interface of the one-launch kernel on the register
// pass routines (reg_queue.cuh).
#pragma once
#include "reg_queue.cuh"
#include "tile_pass.h"

namespace mcfft {

// Variant index of a register pass in that kernel, or -1.
int reg_queue_variant(const TileKernel& k);
// Queue entry of a pass for one exec; dependencies, index tables and table
// offset unset.  False if encoding fails.
bool fill_rpass(const TilePass& tp, int dir, const void* in, void* out, RPass* q);
// CTAs that can be resident at once (0 on error); sets the shared-memory
// limit of both directions' kernels.
int reg_queue_max_grid(int sms);
cudaError_t launch_reg_queue(const RArgs& a, int grid, int dir, cudaStream_t st);

}  // namespace mcfft
