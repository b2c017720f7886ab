// reg_queue.cuh -- every pass of a plain uneven batch in one persistent launch
// on the register pass kernels' tile routines (RegPass, MmaPass, Mma2048,
// Mma4096).
//
// What bounds it: in a long run of one pass HBM, as in the pass kernels
// (2^16 x 1024 in 194 us, 190 as two launches).  Measured, uneven batches of
// 1D lengths 2^8 .. 2^16 and some 2D shapes, batch kernel (fft_queue.cuh)
// against this one: 4160 transforms 349 / 235 us, 1015 116 / 78, 304 48 / 19,
// 65 37 / 19 (tables loaded only at the start of a run: 243, 80, 21, 21).
//
// The queue is the batch kernel's (queue_order.h): items of (pass, tile),
// dealt to the CTAs in turn, every dependency pointing backwards, counters in
// global memory, one CTA per SM, all resident (cooperative launch).  Beside
// the sixteen consumer warps there are three working ones:
//   loader   item k: buffer k % 3 free, dependency met (acquire), TMA load;
//   storers  (items in turn) tile done (all its warps arrived), TMA store,
//            buffer free once the store has read it; then, for passes others
//            wait for, the store's completion, a proxy fence and a release
//            add per key.
// Waiting for a store's completion thus delays neither a load nor the next
// store.
//
// Why a switch over whole runs: the items of a CTA come in runs of one pass
// (queue_order.h), and a routine's per-thread offsets and table are set up
// once per run.  Tables stay in shared memory for the whole launch when those
// of all passes fit (34 KB), else a run's table is copied while the last item
// of the run before is worked on.
//
// The counters are zeroed by the last CTA to leave, for the next launch.
// Every wait is bounded; a timeout sets the abort flag, after which all waits
// return at once and nothing more is stored (see fft_reg.cuh).
#pragma once
#include "fft_mma.cuh"
#include "fft_reg.cuh"
#include "fft_rows.cuh"
#include "fft_small.cuh"

namespace mcfft {

constexpr int kRegQueueMaxPasses = 48;

// One pass (field names as in TileArgs where the tile routines read them).
struct alignas(64) RPass {
  CUtensorMap tmap_in;
  CUtensorMap tmap_out;
  const float4* tw;
  const float2* post_a;
  const float2* post_b;
  uint64_t post_mask;
  uint32_t post_shift;
  float post_scale;
  int32_t in_cmul[5], in_omul[5], out_cmul[5], out_omul[5];
  int32_t in_ndims, out_ndims;
  uint32_t col_blocks;
  uint32_t in_tile_bytes;
  int32_t variant;
  uint32_t tw_off;  // resident tables: offset in the table area
  uint32_t tw_bytes, tab_bytes;
  // Before loading tile (cb, outer): counters[wait_base + outer]
  // >= wait_count; wait_base -1: none.
  int32_t wait_base, wait_count;
  // After the store of tile t: +1 on counters[sig_base + k], k from t sig_mul
  // / sig_div to ((t + 1) sig_mul - 1) / sig_div, at most sig_kmax; -1: none.
  int32_t sig_base, sig_mul, sig_div, sig_kmax;
  // Transforms at unrelated offsets (device tables; null: none): otab[o] is
  // the outer coordinate of outer index o; gtab[c] (one-pass 1D groups, whose
  // tiles span transforms) the first 32-point row of column c, copied
  // transform by transform, g_bytes each, g_cols of them in all.
  const int32_t *in_otab, *out_otab, *in_gtab, *out_gtab;
  uint32_t g_cols, g_bytes, g_tile;  // g_tile: columns per tile
};

struct RItem {
  uint32_t pass, tile;
};

struct alignas(64) RArgs {
  const RItem* items;
  uint32_t nitems;
  int32_t npass;
  int* counters;  // [ncounters], then the leave ticket
  int32_t ncounters;
  int32_t resident;
  int* status;
  const uint4* bmat;  // matrix fragments (plain form)
  RPass pass[kRegQueueMaxPasses];
};
static_assert(sizeof(RArgs) <= 32764, "kernel parameter block");

namespace reg {

// Variant index up to 1024 points: 5 * kind + log2(L / 64), kinds row-row,
// row-column, column, column with four-step twiddle; 20 and 21: rows of 2048
// and 4096 points.
constexpr int kPlainVariants = 22;
__host__ __device__ constexpr int queue_variant_of(int lgL, int kind, bool post) {
  return 5 * (kind == kRR ? 0 : kind == kRC ? 1 : post ? 3 : 2) + (lgL - 6);
}

// The tile routine of a variant.  Radices as in the per-pass registries.
template <int V, bool INV>
struct PlainVariant {
  static constexpr int L = 64 << (V % 5), K = V / 5, KIND = K == 0 ? kRR : K == 1 ? kRC : kCC;
  static constexpr bool POST = K == 3;
  static constexpr int R1 = L == 64 ? 8 : L == 128 ? (KIND == kCC ? 16 : 8) : 16;
  template <int LL, class D>
  struct Pick {
    using type = MmaPass<LL, KIND, POST, INV>;
  };
  template <class D>
  struct Pick<64, D> {
    using type = RegPass<64, 8, 8, 16384, true, true, KIND, POST, INV>;
  };
  template <class D>
  struct Pick<128, D> {
    using type = RegPass<128, R1, 128 / R1, 16384, true, true, KIND, POST, INV>;
  };
  using type = typename Pick<L, void>::type;
};
template <bool INV>
struct PlainVariant<20, INV> {
  using type = Mma2048<INV>;
};
template <bool INV>
struct PlainVariant<21, INV> {
  using type = Mma4096<INV, 16384>;
};
struct QueueShape {
  // NDONE: a ring in which each of the two storers has barriers of its own
  static constexpr int BUF = 65536, NBUF = 3, NDONE = 6, OFF_TAB = NBUF * BUF;
  static constexpr int SMEM_BYTES = 232448, OFF_BAR = SMEM_BYTES - 1024 - 256, TAB_BYTES = OFF_BAR - OFF_TAB;
};

#ifdef MCFFT_REG_QUEUE_KERNEL

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_add(int* p, int v) {
  asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void fence_proxy_async_global() {
  asm volatile("fence.proxy.async.global;" ::: "memory");
}

// What a tile routine keeps per thread: the matrix fragments, held for the
// whole launch, or a state of its own.
template <class X, bool FRAGS = std::is_same<typename X::State, MmaFrags>::value>
struct RunState {
  __device__ __forceinline__ RunState(const RPass&, const MmaFrags&, int) {}
  __device__ __forceinline__ const MmaFrags& get(const MmaFrags& fr) const { return fr; }
};
template <class X>
struct RunState<X, false> {
  typename X::State s;
  __device__ __forceinline__ RunState(const RPass& P, const MmaFrags&, int t) : s(P, t) {}
  __device__ __forceinline__ const typename X::State& get(const MmaFrags&) const { return s; }
};

struct QueueBars {
  uint64_t *full, *done, *freeb;
  volatile uint32_t* ring;  // [NBUF][2]: pass and tile of the item in a buffer
  volatile int* abort_flag;
  uint32_t base_u;
};

__device__ __forceinline__ void queue_loader(const RArgs& a, const QueueBars& q, uint32_t nlocal) {
  constexpr uint32_t NBUF = QueueShape::NBUF;
  const uint32_t G = gridDim.x;
  uint32_t k = 0;
  RItem it = nlocal ? a.items[blockIdx.x] : RItem{0u, 0u};
  for (; k < nlocal; ++k) {
    const RItem nxt = k + 1 < nlocal ? a.items[blockIdx.x + (k + 1) * G] : it;
    const RPass& P = a.pass[it.pass];
    const uint32_t b = k % NBUF, cb = it.tile % P.col_blocks, outer = it.tile / P.col_blocks;
    tile::prefetch_tmap(&P.tmap_in);
    if (k >= NBUF) wait_or_abort(&q.freeb[b], (k / NBUF - 1) & 1u, q.abort_flag);
    if (P.wait_base >= 0 && !*q.abort_flag) {
      const int* c = a.counters + P.wait_base + outer;
      if (ld_acquire(c) < P.wait_count) {
        const uint32_t t0 = sm100::globaltimer_ns();
        while (ld_acquire(c) < P.wait_count && !*q.abort_flag) {
          if (sm100::globaltimer_ns() - t0 > kWaitLimit) *q.abort_flag = 1;
          __nanosleep(64);
        }
      }
      fence_proxy_async_global();
    }
    if (*q.abort_flag) break;
    q.ring[2 * b] = it.pass;
    q.ring[2 * b + 1] = it.tile;
    const uint32_t dst = q.base_u + b * QueueShape::BUF;
    uint64_t* bar = &q.full[k % NBUF];
    if (P.in_gtab) {
      // one copy per transform; a last tile's missing ones are neither loaded
      // nor stored (columns do not mix)
      const uint32_t c0 = cb * P.g_tile, n = P.g_cols - c0 < P.g_tile ? P.g_cols - c0 : P.g_tile;
      sm100::mbar_arrive_expect_tx(bar, n * P.g_bytes);
      for (uint32_t c = 0; c < n; ++c) {
        const int32_t crd[5] = {0, 0, P.in_gtab[c0 + c], 0, 0};
        tile::tma_load(&P.tmap_in, 3, crd, dst + c * P.g_bytes, bar);
      }
    } else {
      int32_t crd[5];
      tile::tile_coords(P.in_cmul, P.in_omul, cb,
                        P.in_otab ? (uint32_t)P.in_otab[outer] : outer, crd);
      sm100::mbar_arrive_expect_tx(bar, P.in_tile_bytes);
      tile::tma_load(&P.tmap_in, P.in_ndims, crd, dst, bar);
    }
    it = nxt;
  }
  // loads in flight must land before the shared memory is released
  for (uint32_t j = k > NBUF ? k - NBUF : 0; j < k; ++j)
    sm100::mbar_wait_bounded(&q.full[j % NBUF], (j / NBUF) & 1u, kWaitLimit);
}

__device__ __forceinline__ void queue_storer(const RArgs& a, const QueueBars& q, uint32_t nlocal, uint32_t which) {
  constexpr uint32_t NBUF = QueueShape::NBUF, NDONE = QueueShape::NDONE;
  for (uint32_t k = which; k < nlocal; k += 2) {
    const uint32_t b = k % NBUF;
    wait_or_abort(&q.done[k % NDONE], (k / NDONE) & 1u, q.abort_flag);
    if (*q.abort_flag) break;
    const RItem it{q.ring[2 * b], q.ring[2 * b + 1]};
    const RPass& P = a.pass[it.pass];
    const uint32_t cb = it.tile % P.col_blocks, outer = it.tile / P.col_blocks;
    const uint32_t src = q.base_u + b * QueueShape::BUF;
    if (P.out_gtab) {
      const uint32_t c0 = cb * P.g_tile, n = P.g_cols - c0 < P.g_tile ? P.g_cols - c0 : P.g_tile;
      for (uint32_t c = 0; c < n; ++c) {
        const int32_t crd[5] = {0, 0, P.out_gtab[c0 + c], 0, 0};
        tile::tma_store(&P.tmap_out, 3, crd, src + c * P.g_bytes);
      }
    } else {
      int32_t crd[5];
      tile::tile_coords(P.out_cmul, P.out_omul, cb,
                        P.out_otab ? (uint32_t)P.out_otab[outer] : outer, crd);
      tile::tma_store(&P.tmap_out, P.out_ndims, crd, src);
    }
    tile::tma_store_wait_read();
    tile::mbar_arrive(&q.freeb[b]);
    if (P.sig_base >= 0) {
      tile::tma_store_wait_all();
      fence_proxy_async_global();
      const uint32_t k0 = (uint32_t)((uint64_t)it.tile * P.sig_mul / P.sig_div);
      uint32_t k1 = (uint32_t)(((uint64_t)it.tile * P.sig_mul + P.sig_mul - 1) / P.sig_div);
      if (k1 > (uint32_t)P.sig_kmax) k1 = (uint32_t)P.sig_kmax;
      for (uint32_t key = k0; key <= k1; ++key) red_release_add(a.counters + P.sig_base + key, 1);
    }
  }
  tile::tma_store_wait_all();
}

// A consumer thread's place in the queue.  Which pass an item is of is read
// from the item list itself, two items ahead: also after a timeout every
// thread runs the same items and meets the same barriers.
struct QueuePlace {
  const RItem* items;
  uint32_t k = 0, nlocal, step;
  RItem it, nx;
  __device__ __forceinline__ QueuePlace(const RArgs& a, uint32_t n)
      : items(a.items + blockIdx.x), nlocal(n), step(gridDim.x) {
    it = nx = RItem{0u, 0u};
    if (n) it = items[0];
    nx = n > 1 ? items[step] : it;
  }
};

// The table of the run at hand: runs alternate between the two ends of the
// table area, so that a table can be copied while the one before is in use.
struct TabState {
  uint32_t off = 0, size = 0, end = 0;
  __device__ __forceinline__ uint32_t next_off(const RPass& P) const {
    return end ? 0u : ((uint32_t)QueueShape::TAB_BYTES - P.tab_bytes) & ~127u;
  }
  __device__ __forceinline__ bool fits(const RPass& P) const {
    return size + P.tab_bytes + 128u <= (uint32_t)QueueShape::TAB_BYTES;
  }
  __device__ __forceinline__ static void copy(const RPass& P, uint32_t to, int t) {
    for (uint32_t i = t; i < P.tw_bytes / 16; i += 512) cp_async16(to + 16 * i, P.tw + i, true);
  }
};

// Runs the items from pl.k on as long as they are of one pass (tile routine
// X); during the last of them the next run's table is on its way.
template <class X>
__device__ __forceinline__ void queue_run(const RArgs& a, const RPass& P, const MmaFrags& fr, const QueueBars& q,
                                          uint32_t tab, const TabState& ts, int t, QueuePlace& pl,
                                          const Sync<512>& sync) {
  constexpr uint32_t NBUF = QueueShape::NBUF;
  const uint32_t ncb = P.col_blocks;
  const RunState<X> st(P, fr, t);
  for (;;) {
    const uint32_t k = pl.k, b = k % NBUF;
    const RItem nn = k + 2 < pl.nlocal ? pl.items[(k + 2) * pl.step] : pl.nx;
    const bool last = k + 1 >= pl.nlocal || pl.nx.pass != pl.it.pass;
    if (last && !a.resident && k + 1 < pl.nlocal) {
      const RPass& N = a.pass[pl.nx.pass];
      if (ts.fits(N)) TabState::copy(N, q.base_u + QueueShape::OFF_TAB + ts.next_off(N), t);
    }
    wait_or_abort(&q.full[b], (k / NBUF) & 1u, q.abort_flag);
    X::run(P, st.get(fr), q.base_u + b * QueueShape::BUF, tab, t, pl.it.tile % ncb, sync);
    sm100::fence_proxy_async_smem();
    __syncwarp();
    if ((t & 31) == 0) tile::mbar_arrive(&q.done[k % QueueShape::NDONE]);
    pl.it = pl.nx;
    pl.nx = nn;
    ++pl.k;
    if (last) return;
  }
}

template <bool INV>
__global__ void __launch_bounds__(640, 1) fft_reg_queue(const __grid_constant__ RArgs a) {
  constexpr int NW = 16, NBUF = QueueShape::NBUF;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_u = sm100::smem_u32(smem_raw);
  const uint32_t base_u = (raw_u + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base_u - raw_u);
  QueueBars q;
  q.full = reinterpret_cast<uint64_t*>(smem + QueueShape::OFF_BAR);
  q.done = q.full + NBUF;
  q.freeb = q.done + QueueShape::NDONE;
  q.ring = reinterpret_cast<volatile uint32_t*>(q.freeb + NBUF);
  q.abort_flag = reinterpret_cast<volatile int*>(q.freeb + NBUF + NBUF);
  q.base_u = base_u;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 512) {
    for (int f = 0; f < NBUF; ++f) sm100::mbar_init(&q.full[f], 1);
    for (int d = 0; d < QueueShape::NDONE; ++d) sm100::mbar_init(&q.done[d], NW);
    for (int b = 0; b < NBUF; ++b) sm100::mbar_init(&q.freeb[b], 1);
    *q.abort_flag = 0;
    sm100::fence_mbar_init();
  }
#define MCFFT_RQ_ALL(M)                                                                          \
  M(0) M(1) M(2) M(3) M(4) M(5) M(6) M(7) M(8) M(9) M(10) M(11) M(12) M(13) M(14) M(15) M(16)  \
  M(17) M(18) M(19) M(20) M(21)
  // the part of a pass's tables that depends on the plan
  auto setup = [&](const RPass& P, uint32_t to) {
    switch (P.variant) {
#define MCFFT_RQ_TAB(V)                                                        \
  case V:                                                                      \
    PlainVariant<V, INV>::type::setup(P, smem + QueueShape::OFF_TAB + to, tid); \
    break;
      MCFFT_RQ_ALL(MCFFT_RQ_TAB)
      default: break;
    }
  };
  if (a.resident && tid < 512)
    for (int pi = 0; pi < a.npass; ++pi) {
      const RPass& P = a.pass[pi];
      TabState::copy(P, base_u + QueueShape::OFF_TAB + P.tw_off, tid);
      setup(P, P.tw_off);
    }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const uint32_t G = gridDim.x, nlocal = a.nitems > blockIdx.x ? (a.nitems - blockIdx.x + G - 1) / G : 0;
  if (warp >= 16) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 24;");
    if (warp == 16 && lane == 0) queue_loader(a, q, nlocal);
    if ((warp == 17 || warp == 18) && lane == 0) queue_storer(a, q, nlocal, warp - 17);
    __syncwarp();
    __syncthreads();
    return;  // the rest belongs to the warps that hold registers for it
  }
  {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    const Sync<512> sync{1};
    const MmaFrags fr(a, tid);
    TabState ts;
    QueuePlace pl(a, nlocal);
    while (pl.k < nlocal) {
      const RPass& P = a.pass[pl.it.pass];
      if (a.resident) {
        ts.off = P.tw_off;
      } else {
        // The barrier of the last switch: nobody reads the table before the
        // current one any more, whose end of the area this one takes.
        const bool fits = ts.fits(P) && pl.k > 0;  // copied already
        const uint32_t off = ts.next_off(P);
        if (!fits) {
          sync.group();
          TabState::copy(P, base_u + QueueShape::OFF_TAB + off, tid);
        }
        setup(P, off);
        asm volatile("cp.async.wait_all;" ::: "memory");
        sync.group();
        ts.off = off;
        ts.size = P.tab_bytes;
        ts.end ^= 1u;
      }
      const uint32_t tab = base_u + QueueShape::OFF_TAB + ts.off;
      switch (P.variant) {
#define MCFFT_RQ_RUN(V)                                                                       \
  case V:                                                                                     \
    queue_run<typename PlainVariant<V, INV>::type>(a, P, fr, q, tab, ts, tid, pl, sync);      \
    break;
        MCFFT_RQ_ALL(MCFFT_RQ_RUN)
        default: pl.k = nlocal; break;
      }
    }
  }
  __syncthreads();
  // The last CTA to leave zeroes the counters for the next launch (every
  // signal and every wait of this one is over).
  if (tid == 0) {
    if (*q.abort_flag && a.status) atomicExch(a.status, kStatusTimeout);
    __threadfence();
    *q.abort_flag = atomicAdd(a.counters + a.ncounters, 1) == (int)gridDim.x - 1;
  }
  asm volatile("bar.sync 3, 512;" ::: "memory");
  if (*q.abort_flag)
    for (int i = tid; i <= a.ncounters; i += 512) a.counters[i] = 0;
}

#endif  // MCFFT_REG_QUEUE_KERNEL

}  // namespace reg
}  // namespace mcfft
