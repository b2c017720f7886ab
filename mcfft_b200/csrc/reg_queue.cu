// reg_queue.cu -- host side of the one-launch kernel on the register pass
// routines (reg_queue.cuh).
#include <cstring>
#include <utility>
#include <vector>

#include "reg_pass.h"
#include "reg_queue.h"

namespace mcfft {

const void* reg_queue_plain_fwd();
const void* reg_queue_plain_inv();

namespace {
const void* queue_fn(int dir) { return dir ? reg_queue_plain_inv() : reg_queue_plain_fwd(); }

// Length, columns, kind, four-step twiddle and tables of each variant's tile
// routine, to check a pass against before it is queued.
struct VariantInfo {
  int L, C, kind;
  bool post;
  int tw_bytes, tab_bytes;
};
template <int V>
VariantInfo info_of() {
  using X = typename reg::PlainVariant<V, false>::type;
  return {X::L, X::C, X::KIND, X::POST, X::TWB, X::TABB};
}
template <int... V>
std::vector<VariantInfo> infos(std::integer_sequence<int, V...>) {
  return {info_of<V>()...};
}
}  // namespace

int reg_queue_variant(const TileKernel& k) {
  static const std::vector<VariantInfo> all = infos(std::make_integer_sequence<int, reg::kPlainVariants>());
  if (k.split || k.reg_kind < 0 || k.L < 64 || k.L > 4096 || k.tile_points != 16384) return -1;
  int lg = 6;
  while ((1 << lg) < k.L) ++lg;
  const int v = k.L > 1024 ? 20 + (lg - 11) : reg::queue_variant_of(lg, k.reg_kind, k.posttw);
  const VariantInfo& x = all[v];
  const bool same = x.L == k.L && x.C == k.C && x.kind == k.reg_kind && x.post == k.posttw &&
                    x.tw_bytes == k.tw_bytes && x.tab_bytes == k.tab_bytes;
  return same ? v : -1;
}

bool fill_rpass(const TilePass& tp, int dir, const void* in, void* out, RPass* q) {
  const TileArgs& a = tp.args;
  std::memset(q, 0, sizeof(*q));
  if (!tile_encode(&q->tmap_in, tp.lay.in, in) || !tile_encode(&q->tmap_out, tp.lay.out, out)) return false;
  q->tw = tp.tw[dir];
  q->post_a = tp.post_a[dir];
  q->post_b = tp.post_b[dir];
  q->post_mask = a.post_mask;
  q->post_shift = a.post_shift;
  q->post_scale = a.post_scale;
  std::memcpy(q->in_cmul, a.in_cmul, sizeof(q->in_cmul));
  std::memcpy(q->in_omul, a.in_omul, sizeof(q->in_omul));
  std::memcpy(q->out_cmul, a.out_cmul, sizeof(q->out_cmul));
  std::memcpy(q->out_omul, a.out_omul, sizeof(q->out_omul));
  q->in_ndims = a.in_ndims;
  q->out_ndims = a.out_ndims;
  q->col_blocks = (uint32_t)a.col_blocks;
  q->in_tile_bytes = a.in_tile_bytes;
  q->variant = reg_queue_variant(*tp.k);
  q->tw_bytes = (uint32_t)tp.k->tw_bytes;
  q->tab_bytes = (uint32_t)tp.k->tab_bytes;
  q->wait_base = q->sig_base = -1;
  q->sig_mul = q->sig_div = 1;
  return q->variant >= 0;
}

int reg_queue_max_grid(int sms) {
  int occ = 0;
  for (int dir = 0; dir < 2; ++dir) {
    const void* fn = queue_fn(dir);
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, reg::QueueShape::SMEM_BYTES) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, 640, reg::QueueShape::SMEM_BYTES) !=
            cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    if (occ < 1) return 0;
  }
  return sms;
}

cudaError_t launch_reg_queue(const RArgs& a, int grid, int dir, cudaStream_t st) {
  void* args[] = {const_cast<RArgs*>(&a)};
  // Cooperative: every CTA is resident, so a tile waiting for another CTA's
  // output never waits for one that has not started.
  return cudaLaunchCooperativeKernel(queue_fn(dir), dim3(grid), dim3(640), args,
                                     (size_t)reg::QueueShape::SMEM_BYTES, st);
}

}  // namespace mcfft
