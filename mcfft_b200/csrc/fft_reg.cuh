// fft_reg.cuh -- TMA-fed FFT pass kernel whose butterflies stay in registers.
//
// Persistent, one CTA per SM (small tiles: three); a tile holds C columns x L
// points, L = R1 R2, both radices at most 32.  A thread holds 32 points of the tile in FP32: one
// 32-point vector, two of 16 or four of 8 (fft_codelets.cuh), so a pass of up
// to 1024 points is two phases with one exchange through shared memory:
//
//   phase 1   n = n1 NV + v: R1-point DFT over n1, twiddle W_L^(k1 v)
//   phase 2   R2-point DFT over v, output X[k1 + R1 k2]
//
// What bounds such a pass, and why it is laid out so.  A 16K-point FP16 (8K
// FP32) tile is 64 KB in and 64 KB out, 5.9 K cycles of one SM's share of the
// copy bandwidth.  The tile crosses shared memory six times (TMA in, phase 1
// load and store, phase 2 load and store, TMA out): 3 K wavefronts of 128
// bytes plus 0.6 .. 0.9 K of twiddles, and 2 to 2.6 K cycles of the FP32 pipe.
// The tcgen05 form of the same pass (fft_tile.cuh) crosses it eight times and
// reads its stage operands and twiddle rows on top, 5.6 K wavefronts in
// phases that wait for one another; a 16-point DFT as a real 32 x 32 product
// is too small a contraction to pay for staging its operand.  Measured on a
// B200 (2^20 x 64, FP16 in, FP32 out, whole exec): 512 us with the tcgen05
// split tiles, 375 us here; the same TMA copies without any arithmetic take
// 350 us.  3D 256^3 FP32: 195 -> 141 us.  Plain, where a 64 KB tile holds 16K
// points, 4.3 K cycles of the FP32 pipe that no longer hide behind the copies:
// 2D 1024^2 x 16 70.9 -> 65.6 us, 3D 256^3 92.3 -> 84.3, so 256 to 1024 plain
// points are MmaPass (fft_mma.cuh: 57.1 and 72.4).
//
// Exchange in place.  Phase 1 writes its outputs into the slots its own warp
// has read (k1 in the place of n1, lanes of the warp permuted so that phase 2
// reads without bank conflicts), so no barrier separates a phase's loads from
// its stores.  KIND says where the pass's points lie:
//   RR  rows in and out: a warp owns whole columns (1024 points of them), both
//       phases are warp-local, and no block barrier is needed at all;
//   CC  columns in and out: phase 2 also writes in place; the tile leaves
//       digit-reversed in shared memory and the TMA store's box dimensions
//       (column, k1 low, k2, k1 high) undo that.  One barrier per tile;
//   RC  rows in, columns out: phase 2's output goes to other slots, two
//       barriers per tile.
// Each warp signals the tile's `done` mbarrier; the producer warp stores the
// tile, and refills the buffer once the store has read it.
//
// Number forms: OUT16 (plain): FP16 staging and exchange, packed FP32x2
// arithmetic, 1/R per phase.  Otherwise FP32 staging and exchange, unscaled
// (split form; IN16: FP16 input).
//
// Every wait is bounded.  After a timeout the abort flag makes all later
// waits return at once, so that every warp still takes part in the remaining
// barriers and the block ends; nothing more is stored, and the status word
// reports it.
#pragma once
#include "fft_codelets.cuh"

namespace mcfft {
namespace reg {

enum RegKind { kRR = 0, kCC = 1, kRC = 2 };

// Order in which a warp's column bits are taken: column bit 2 flips the
// upper half of a 128-byte row under the row staging's swizzle, bit 1 the
// quarter, so lanes that share a row position fall in distinct banks.
__host__ __device__ constexpr int s_bit(int i) { return i == 0 ? 2 : i == 1 ? 1 : i == 2 ? 0 : i; }
__host__ __device__ constexpr uint32_t s_deposit(uint32_t x, int from, int cnt) {
  uint32_t c = 0;
  for (int i = 0; i < cnt; ++i) c |= ((x >> i) & 1u) << s_bit(from + i);
  return c;
}
// Bits of x into the column bits below lgc that s_bit(0 .. nc - 1) leave free.
__host__ __device__ constexpr uint32_t s_rest(uint32_t x, int nc, int lgc) {
  uint32_t c = 0;
  int at = 0;
  for (int b = 0; b < lgc; ++b) {
    bool used = false;
    for (int i = 0; i < nc; ++i) used |= s_bit(i) == b;
    if (!used) c |= ((x >> at++) & 1u) << b;
  }
  return c;
}

__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}

// Bounded wait; after a timeout (here or elsewhere in the block) it returns
// at once, leaving the abort flag set.
__device__ __forceinline__ void wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (sm100::mbar_try_wait(bar, parity)) return;
  const uint32_t t0 = sm100::globaltimer_ns();
  while (!sm100::mbar_try_wait(bar, parity)) {
    if (*abort_flag) return;
    if (sm100::globaltimer_ns() - t0 > kWaitLimit) {
      *abort_flag = 1;
      return;
    }
  }
}

// Barrier among the T threads of a group.
template <int T>
struct Sync {
  int bar;
  __device__ __forceinline__ void group() const {
    asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(T) : "memory");
  }
};

template <int L_, int R1_, int R2_, int TP_, bool IN16_, bool OUT16_, int KIND_, bool POST_, bool INV_>
struct RegPass {
  static constexpr int L = L_, R1 = R1_, R2 = R2_, TP = TP_, KIND = KIND_;
  static constexpr bool IN16 = IN16_, OUT16 = OUT16_, POST = POST_, INV = INV_;
  static_assert(L == R1 * R2 && R1 <= 32 && R2 <= 32 && L >= 64 && L <= 1024, "two phases");
  static_assert(!OUT16 || IN16, "FP16 out takes FP16 in");
  static_assert(!POST || KIND == kCC, "four-step twiddle on column passes");
  static constexpr int C = TP / L, NV = R2, T = TP / 32, NW = T / 32;
  static constexpr int V1 = 32 / R1, V2 = 32 / R2;
  static constexpr int EI = IN16 ? 4 : 8, EO = OUT16 ? 4 : 8;  // bytes per point: in, exchange and out
  static constexpr bool PK = OUT16;
  static constexpr int lgC = ilog2c(C), lgNV = ilog2c(NV), lgR1 = ilog2c(R1);
  static constexpr int nc = 10 - ilog2c(L);  // column bits inside a warp (row passes)
  static_assert(T >= 128 && (T >= 256 || KIND == kRR), "small tiles: rows in and out");
  static_assert(C >= 8, "row swizzle and in-warp columns need eight columns");
  // Column staging: bytes of one point row, and the point rows that share a
  // 128-byte line (1 << h of them).
  static constexpr int RBI = C * EI, RB = C * EO;
  static constexpr int h = RB >= 128 ? 0 : ilog2c(128 / RB), m = (1 << h) - 1;
  static constexpr int lc = lgC < 5 ? lgC : 5;  // lanes along columns (column passes)
  static_assert(KIND == kRR || 5 - lc >= h, "rows of one line sit in one warp");
  static constexpr int BUF = TP * (EI > EO ? EI : EO);
  // Twiddle table, k-major, v fastest: one factor doubled for two columns, 16
  // bytes; FP32 form 8 bytes.
  static constexpr int TWB = L * (PK ? 16 : 8);
  static constexpr int NG = T >= 256 ? 512 / T : 1;  // tiles in work at a time
  static constexpr int NBUF = T >= 256 ? 3 : 2;
  // Load barriers: a ring long enough that one group alone waits on each
  // (tile i and tile i + NFULL go to the same group).  A group may run ahead
  // of the other's tile in the same buffer, and a parity wait is only right
  // for a waiter that has seen the phase before.
  static constexpr int NFULL = NG == 1 ? NBUF : NG * NBUF;
  static constexpr bool BIG = NG * T == 512;  // one CTA per SM; else small tiles, several
  static constexpr int THREADS = NG * T + (BIG ? 128 : 32), MINB = BIG ? 1 : 3;
  static constexpr int OFF_TW = NBUF * BUF;
  static constexpr int OFF_BAR = OFF_TW + TWB;
  static constexpr int TABB = TWB;  // all tables
  static constexpr int SMEM_BYTES = OFF_BAR + 128 + 1024;
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");

  // ------------------------------------------------ vectors of this thread
  // Row kinds, phase p (R = the other factor's digit x): x in the low lane
  // bits, columns after it.
  static __host__ __device__ __forceinline__ void row_vec(int t, int j, int lgx, uint32_t& x, uint32_t& c) {
    const uint32_t lane = t & 31, warp = t >> 5;
    x = lane & ((1u << lgx) - 1u);
    c = s_deposit(lane >> lgx, 0, 5 - lgx) | s_deposit(j, 5 - lgx, nc - (5 - lgx)) | s_rest(warp, nc, lgC);
  }
  // Column kinds: columns in the low lane bits, then low bits of the digit x;
  // register vectors take further column bits, the warp the rest.
  template <int LGV>
  static __host__ __device__ __forceinline__ void col_vec(int t, int j, uint32_t& x, uint32_t& c) {
    const uint32_t lane = t & 31, warp = t >> 5;
    constexpr int chi = lgC - lc, cv = chi < LGV ? chi : LGV, cw = chi - cv;  // column bits: vectors, warp
    c = (lane & ((1u << lc) - 1u)) | ((j & ((1u << cv) - 1u)) << lc) | ((warp & ((1u << cw) - 1u)) << (lc + cv));
    const uint32_t xl = lane >> lc, xj = (uint32_t)j >> cv, xw = warp >> cw;
    x = xl | (xj << (5 - lc)) | (xw << (5 - lc + LGV - cv));
  }
  static __host__ __device__ __forceinline__ void vec1(int t, int j, uint32_t& v, uint32_t& c) {
    if constexpr (KIND == kCC) col_vec<ilog2c(V1)>(t, j, v, c);
    else row_vec(t, j, lgNV, v, c);
  }
  static __host__ __device__ __forceinline__ void vec2(int t, int j, uint32_t& k1, uint32_t& c) {
    if constexpr (KIND == kRR) row_vec(t, j, lgR1, k1, c);
    else col_vec<ilog2c(V2)>(t, j, k1, c);
  }

  // ----------------------------------------------------- shared addresses
  // Every access is (base ^ x) + a with x, a known at compile time.  Row
  // staging: 128-byte rows of EL points, row (pos / EL) C + c, 16-byte chunks
  // XORed with c & 7 (the TMA 128-byte swizzle; C is a multiple of eight).
  template <int E8>
  static __host__ __device__ __forceinline__ uint32_t row_base(uint32_t pos, uint32_t c) {
    constexpr uint32_t EL = 128 / E8;
    return ((pos / EL) * C + c) * 128u + (((pos % EL) * E8) ^ ((c & 7u) << 4));
  }
  // Stride S points, i-th step: XOR and add parts.
  template <int E8, int S>
  static __host__ __device__ constexpr uint32_t row_x(int i) {
    return S < 128 / E8 ? (uint32_t)(i % (128 / E8 / S)) * S * E8 : 0u;
  }
  template <int E8, int S>
  static __host__ __device__ constexpr uint32_t row_a(int i) {
    return S < 128 / E8 ? (uint32_t)(i / (128 / E8 / S)) * C * 128u : (uint32_t)i * (S / (128 / E8)) * C * 128u;
  }
  // Extra chunk XOR of exchange vector k1, so that lanes with different k1
  // read (16 bytes each) from distinct banks.
  static constexpr int EM = 128 / EO;                          // points per 128-byte row
  static constexpr int CH = NV * EO / 16 < 8 ? NV * EO / 16 : 8;  // chunks of a vector within a row
  static __host__ __device__ constexpr uint32_t fx(uint32_t k1) {
    return NV >= EM ? (k1 & 7u) : ((k1 / (EM / NV)) & (CH - 1));
  }

  static __host__ __device__ __forceinline__ uint32_t load1_base(uint32_t v, uint32_t c) {
    if constexpr (KIND == kCC) return v * RBI + c * EI;
    else return row_base<EI>(v, c);
  }
  static __host__ __device__ constexpr uint32_t load1_x(int n) { return KIND == kCC ? 0u : row_x<EI, NV>(n); }
  static __host__ __device__ constexpr uint32_t load1_a(int n) {
    return KIND == kCC ? (uint32_t)n * NV * RBI : row_a<EI, NV>(n);
  }
  static __host__ __device__ __forceinline__ uint32_t store1_base(uint32_t v, uint32_t c) {
    if constexpr (KIND == kCC) return v * RB + c * EO;
    else return row_base<EO>(v, c);
  }
  static __host__ __device__ constexpr uint32_t store1_x(int k) {
    return KIND == kCC ? (uint32_t)(k & m) * RB : (row_x<EO, NV>(k) ^ (fx(k) << 4));
  }
  static __host__ __device__ constexpr uint32_t store1_a(int k) {
    return KIND == kCC ? (uint32_t)k * NV * RB : row_a<EO, NV>(k);
  }
  // Phase 2 loads: points (CC) or 16-byte chunks (RR, RC) of vector k1.
  static constexpr int LW2 = KIND == kCC ? 1 : 16 / EO;  // points per load
  static __host__ __device__ __forceinline__ uint32_t load2_base(uint32_t k1, uint32_t c) {
    if constexpr (KIND == kCC) return (k1 * NV + (k1 & m)) * RB + c * EO;
    else return row_base<EO>(k1 * NV, c) ^ (fx(k1) << 4);
  }
  static __host__ __device__ constexpr uint32_t load2_x(int i) {
    return KIND == kCC ? (uint32_t)(i & m) * RB : (uint32_t)(i % 8) << 4;
  }
  static __host__ __device__ constexpr uint32_t load2_a(int i) {
    return KIND == kCC ? (uint32_t)(i - (i & m)) * RB : (uint32_t)(i / 8) * C * 128u;
  }
  static __host__ __device__ __forceinline__ uint32_t store2_base(uint32_t k1, uint32_t c) {
    if constexpr (KIND == kCC) return ((k1 >> h) * (NV << h) + (k1 & m)) * RB + c * EO;
    else if constexpr (KIND == kRC) return k1 * RB + c * EO;
    else return row_base<EO>(k1, c);
  }
  static __host__ __device__ constexpr uint32_t store2_x(int k) { return KIND == kRR ? row_x<EO, R1>(k) : 0u; }
  static __host__ __device__ constexpr uint32_t store2_a(int k) {
    return KIND == kCC ? (uint32_t)(k << h) * RB : KIND == kRC ? (uint32_t)k * R1 * RB : row_a<EO, R1>(k);
  }

  // --------------------------------------------------------- plain, packed
  // R-point DFTs of this thread's 32 points, in FP16 words w[j][n] and out in
  // packed FP32 pairs: pair (j / 2, k) = output k of vectors j and j + 1.
  template <int R>
  static __device__ __forceinline__ void dft_pk(const uint32_t (&w)[32 / R][R], P2 (&re)[16], P2 (&im)[16]) {
    static_assert(R <= 16, "two vectors per thread");
#pragma unroll
    for (int j = 0; j < 32 / R; j += 2) {
      P2 r[R], i[R];
#pragma unroll
      for (int n = 0; n < R; ++n) {
        const float2 a = sm100::unpack_half2(w[j][n]), b = sm100::unpack_half2(w[j + 1][n]);
        r[n] = pack2(a.x, b.x);
        i[n] = pack2(a.y, b.y);
      }
      Dft<R, INV, P2>::run(r, i);
#pragma unroll
      for (int k = 0; k < R; ++k) {
        re[j / 2 * R + k] = r[k];
        im[j / 2 * R + k] = i[k];
      }
    }
  }
  // Pair p of dft_pk's result -> the FP16 words of its two points.
  template <int R>
  static __device__ __forceinline__ void words(int p, P2 re, P2 im, uint32_t (&w)[32 / R][R]) {
    float r0, r1, i0, i1;
    f2u(re.v, r0, r1);
    f2u(im.v, i0, i1);
    w[2 * (p / R)][p % R] = sm100::pack_half2(r0, i0);
    w[2 * (p / R) + 1][p % R] = sm100::pack_half2(r1, i1);
  }

  template <class A>
  static __device__ __forceinline__ float2 post_tab(const A& a, uint64_t e) {
    e &= a.post_mask;
    return cmulf(__ldg(a.post_a + (e & ((1ull << a.post_shift) - 1))), __ldg(a.post_b + (e >> a.post_shift)));
  }
  // W_N^e, plain form: the hardware sine and cosine of the exact angle up to
  // N = 2^24 (absolute error below 1e-6, far under the FP16 rounding), else
  // the FP64-generated two-level table.
  template <class A>
  static __device__ __forceinline__ float2 post_fast(const A& a, uint64_t e) {
    if (a.post_scale == 0.f) return post_tab(a, e);
    float x = (float)(e & a.post_mask) * a.post_scale;  // [0, 2)
    x = x >= 1.f ? x - 2.f : x;
    float sn, cs;
    __sincosf(x * 3.14159265358979f, &sn, &cs);
    return make_float2(cs, INV ? sn : -sn);
  }

  // Row kind: byte in the tile's transforms, one after another, of byte off of
  // the buffer (swizzled 128-byte rows, the columns' side by side).
  template <int E>
  static __host__ __device__ constexpr uint32_t row_map(uint32_t off) {
    return ((off >> 7) % C) * (L * E) + (off >> 7) / C * 128u + ((off ^ off >> 3) & 0x70u) + (off & 15u);
  }
  static __host__ __device__ constexpr uint32_t in_map(uint32_t off) { return row_map<EI>(off); }
  static __host__ __device__ constexpr uint32_t out_map(uint32_t off) { return row_map<EO>(off); }

  // Tables that depend on the plan (none here).
  template <class A>
  static __device__ __forceinline__ void setup(const A&, uint8_t*, int) {}

  // What a thread keeps for the whole launch (nothing here).
  struct State {
    template <class A>
    __device__ __forceinline__ State(const A&, int) {}
  };

  // One tile in buffer sb; t: thread of the group, tws: twiddle table.
  template <class A>
  static __device__ __forceinline__ void run(const A& a, const State&, uint32_t sb, uint32_t tws, int t, uint32_t cb,
                                             const Sync<T>& sync) {
    if constexpr (PK) run_pk(a, sb, tws, t, cb, sync);
    else run_f32(a, sb, tws, t, cb, sync);
  }

  template <class A>
  static __device__ __forceinline__ void run_pk(const A& a, uint32_t sb, uint32_t tws, int t, uint32_t cb,
                                                const Sync<T>& sync) {
    P2 re[16], im[16];
    {  // ------------------------------------------------------- phase 1
      uint32_t w[V1][R1], b[V1], v = 0, c = 0;
#pragma unroll
      for (int j = 0; j < V1; ++j) {
        vec1(t, j, v, c);
        b[j] = sb + load1_base(v, c);
#pragma unroll
        for (int n = 0; n < R1; ++n) w[j][n] = lds32((b[j] ^ load1_x(n)) + load1_a(n));
      }
      __syncwarp();
      dft_pk<R1>(w, re, im);
      const uint32_t tw = tws + v * 16u;  // v is the same for all vectors of a thread
      constexpr float sc = 1.f / R1;
#pragma unroll
      for (int p = 0; p < 16; ++p) {
        if (p % R1 == 0) {
          re[p] = re[p] * num<P2>(sc);
          im[p] = im[p] * num<P2>(sc);
        } else {
          const float4 f = lds128f(tw + p % R1 * (NV * 16));
          cmulv(re[p], im[p], pack2(f.x, f.y), pack2(f.z, f.w));
        }
        words<R1>(p, re[p], im[p], w);
      }
#pragma unroll
      for (int j = 0; j < V1; ++j)
#pragma unroll
        for (int k = 0; k < R1; ++k) tile::sts32((b[j] ^ store1_x(k)) + store1_a(k), w[j][k]);
    }
    if constexpr (KIND == kRR) __syncwarp();
    else sync.group();
    {  // ------------------------------------------------------- phase 2
      uint32_t w[V2][R2], k1[V2], c[V2];
#pragma unroll
      for (int j = 0; j < V2; ++j) {
        vec2(t, j, k1[j], c[j]);
        const uint32_t b = sb + load2_base(k1[j], c[j]);
        if constexpr (KIND == kCC) {
#pragma unroll
          for (int n = 0; n < R2; ++n) w[j][n] = lds32((b ^ load2_x(n)) + load2_a(n));
        } else {
#pragma unroll
          for (int n = 0; n < R2 / 4; ++n) {
            const uint4 q = tile::lds128((b ^ load2_x(n)) + load2_a(n));
            w[j][4 * n] = q.x;
            w[j][4 * n + 1] = q.y;
            w[j][4 * n + 2] = q.z;
            w[j][4 * n + 3] = q.w;
          }
        }
      }
      if constexpr (KIND != kRC) __syncwarp();
      dft_pk<R2>(w, re, im);
      constexpr float sc = 1.f / R2;
      if constexpr (POST) {
        // W_N^((k1 + R1 k2) g) / R2: the first factor of each pair and its
        // step, advanced by an FP32 recurrence of 15 steps at most.
        P2 wr[V2 / 2], wi[V2 / 2], sr[V2 / 2], si[V2 / 2];
#pragma unroll
        for (int q = 0; q < V2 / 2; ++q) {
          float2 f[2], s[2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const uint64_t g = (uint64_t)(cb * C + c[2 * q + u]);
            f[u] = post_fast(a, k1[2 * q + u] * g);
            s[u] = post_fast(a, (uint64_t)R1 * g);
          }
          wr[q] = pack2(f[0].x * sc, f[1].x * sc);
          wi[q] = pack2(f[0].y * sc, f[1].y * sc);
          sr[q] = pack2(s[0].x, s[1].x);
          si[q] = pack2(s[0].y, s[1].y);
        }
#pragma unroll
        for (int p = 0; p < 16; ++p) {
          const int q = p / R2;
          cmulv(re[p], im[p], wr[q], wi[q]);
          if (p % R2 != R2 - 1) cmulv(wr[q], wi[q], sr[q], si[q]);
          words<R2>(p, re[p], im[p], w);
        }
      } else {
#pragma unroll
        for (int p = 0; p < 16; ++p) words<R2>(p, re[p] * num<P2>(sc), im[p] * num<P2>(sc), w);
      }
      if constexpr (KIND == kRC) sync.group();
#pragma unroll
      for (int j = 0; j < V2; ++j) {
        const uint32_t b = sb + store2_base(k1[j], c[j]);
#pragma unroll
        for (int k = 0; k < R2; ++k) tile::sts32((b ^ store2_x(k)) + store2_a(k), w[j][k]);
      }
    }
  }

  // ------------------------------------------------------- FP32 arithmetic
  template <int R>
  static __device__ __forceinline__ void dft_f32(float (&re)[R], float (&im)[R]) {
    if constexpr (R == 32) {
      float er[16], ei[16], dr[16], di[16];
#pragma unroll
      for (int n = 0; n < 16; ++n)
        split32<INV>(re[n], im[n], re[n + 16], im[n + 16], n, er[n], ei[n], dr[n], di[n]);
      Dft<16, INV, float>::run(er, ei);
      Dft<16, INV, float>::run(dr, di);
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        re[2 * k] = er[k];
        im[2 * k] = ei[k];
        re[2 * k + 1] = dr[k];
        im[2 * k + 1] = di[k];
      }
    } else {
      Dft<R, INV, float>::run(re, im);
    }
  }

  template <class A>
  static __device__ __forceinline__ void run_f32(const A& a, uint32_t sb, uint32_t tws, int t, uint32_t cb,
                                                 const Sync<T>& sync) {
    {  // ------------------------------------------------------- phase 1
      float re[V1][R1], im[V1][R1];
      uint32_t v[V1], c[V1];
#pragma unroll
      for (int j = 0; j < V1; ++j) {
        vec1(t, j, v[j], c[j]);
        const uint32_t b = sb + load1_base(v[j], c[j]);
#pragma unroll
        for (int n = 0; n < R1; ++n) {
          if constexpr (IN16) {
            const float2 x = sm100::unpack_half2(lds32((b ^ load1_x(n)) + load1_a(n)));
            re[j][n] = x.x;
            im[j][n] = x.y;
          } else {
            const float2 x = lds64f((b ^ load1_x(n)) + load1_a(n));
            re[j][n] = x.x;
            im[j][n] = x.y;
          }
        }
      }
      // FP16 input and FP32 exchange share the buffer: all loads first
      if constexpr (EI != EO) sync.group();
      else __syncwarp();
#pragma unroll
      for (int j = 0; j < V1; ++j) {
        dft_f32<R1>(re[j], im[j]);
        const uint32_t tw = tws + v[j] * 8u, b = sb + store1_base(v[j], c[j]);
#pragma unroll
        for (int k = 0; k < R1; ++k) {
          if (k > 0) {
            const float2 f = lds64f(tw + k * (NV * 8));
            cmulv(re[j][k], im[j][k], f.x, f.y);
          }
          tile::sts64((b ^ store1_x(k)) + store1_a(k), make_float2(re[j][k], im[j][k]));
        }
      }
    }
    if constexpr (KIND == kRR) __syncwarp();
    else sync.group();
    {  // ------------------------------------------------------- phase 2
      float re[V2][R2], im[V2][R2];
      uint32_t k1[V2], c[V2];
#pragma unroll
      for (int j = 0; j < V2; ++j) {
        vec2(t, j, k1[j], c[j]);
        const uint32_t b = sb + load2_base(k1[j], c[j]);
        if constexpr (KIND == kCC) {
#pragma unroll
          for (int n = 0; n < R2; ++n) {
            const float2 x = lds64f((b ^ load2_x(n)) + load2_a(n));
            re[j][n] = x.x;
            im[j][n] = x.y;
          }
        } else {
#pragma unroll
          for (int n = 0; n < R2 / 2; ++n) {
            const float4 x = lds128f((b ^ load2_x(n)) + load2_a(n));
            re[j][2 * n] = x.x;
            im[j][2 * n] = x.y;
            re[j][2 * n + 1] = x.z;
            im[j][2 * n + 1] = x.w;
          }
        }
      }
      if constexpr (KIND == kRC) sync.group();
      else __syncwarp();
#pragma unroll
      for (int j = 0; j < V2; ++j) {
        dft_f32<R2>(re[j], im[j]);
        const uint32_t b = sb + store2_base(k1[j], c[j]);
        if constexpr (POST) {
          // W_N^((k1 + R1 k2) g), k2 = u + 4 q: four table factors (first,
          // steps 1, 4, 16) and products at most five deep, so the FP32
          // rounding does not grow along a chain of 31 steps
          const uint64_t g = (uint64_t)(cb * C + c[j]);
          float2 w[4];
          w[0] = post_tab(a, k1[j] * g);
          const float2 s1 = post_tab(a, (uint64_t)R1 * g), s4 = post_tab(a, (uint64_t)R1 * 4 * g);
          const float2 s2 = cmulf(s1, s1);
          w[1] = cmulf(w[0], s1);
          w[2] = cmulf(w[0], s2);
          w[3] = cmulf(w[1], s2);
          float2 s16 = make_float2(1.f, 0.f);
          if constexpr (R2 == 32) s16 = post_tab(a, (uint64_t)R1 * 16 * g);
          float2 f = make_float2(1.f, 0.f);
#pragma unroll
          for (int q = 0; q < R2 / 4; ++q) {
            if (q == 1) f = s4;
            else if (q > 1) f = q == 4 ? s16 : cmulf(f, s4);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int k = 4 * q + u;
              const float2 z = q ? cmulf(w[u], f) : w[u];
              cmulv(re[j][k], im[j][k], z.x, z.y);
            }
          }
        }
#pragma unroll
        for (int k = 0; k < R2; ++k)
          tile::sts64((b ^ store2_x(k)) + store2_a(k), make_float2(re[j][k], im[j][k]));
      }
    }
  }
};

template <class P>
__global__ void __launch_bounds__(P::THREADS, P::MINB) fft_reg(const __grid_constant__ TileArgs a) {
  constexpr int NG = P::NG, T = P::T, NW = P::NW, NBUF = P::NBUF;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_u = sm100::smem_u32(smem_raw);
  const uint32_t base_u = (raw_u + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base_u - raw_u);
  constexpr int NFULL = P::NFULL;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + P::OFF_BAR);  // [NFULL]
  uint64_t* done = full + NFULL;                                    // [NBUF]
  volatile int* abort_flag = reinterpret_cast<volatile int*>(done + NBUF);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool producer = warp == NG * NW;
  // 32-bit tile arithmetic (the plan refuses more tiles than that)
  const uint32_t step = gridDim.x, ntiles = (uint32_t)a.ntiles, ncb = (uint32_t)a.col_blocks;
  const uint32_t mine = ntiles > blockIdx.x ? (ntiles - 1 - blockIdx.x) / step + 1 : 0;
  auto load = [&](uint32_t i) {
    const uint32_t t = blockIdx.x + i * step, b = i % NBUF;
    int32_t crd[5];
    tile::tile_coords(a.in_cmul, a.in_omul, t % ncb, t / ncb, crd);
    sm100::mbar_arrive_expect_tx(&full[i % NFULL], a.in_tile_bytes);
    tile::tma_load(&a.tmap_in, a.in_ndims, crd, base_u + b * P::BUF, &full[i % NFULL]);
  };
  // Small tiles: the first loads are issued before the tables are in place.
  // Large ones issue them after the barrier, all from the one loop that holds
  // the copying thread's state: with a second copy of the load before the
  // barrier, and with the copying warps returning early instead of joining the
  // consumers at the end, the consumers' code got slower (1024 x 16384 28.9 ->
  // 32.5 us, 3D 256^3 68.9 -> 74.0, 2^20 x 64 213 -> 224, same registers).
  // Under a programmatic dependent launch the buffers the passes share are
  // touched only after the wait; the tables are this launch's own constants.
  uint32_t loaded = 0;
  if (producer) {
    if (lane == 0) {
      tile::prefetch_tmap(&a.tmap_in);
      tile::prefetch_tmap(&a.tmap_out);
      for (int f = 0; f < NFULL; ++f) sm100::mbar_init(&full[f], 1);
      for (int b = 0; b < NBUF; ++b) sm100::mbar_init(&done[b], NW);
      *abort_flag = 0;
      sm100::fence_mbar_init();
      if constexpr (!P::BIG) {
        sm100::grid_dep_wait();
        for (; loaded < mine && loaded < NBUF; ++loaded) load(loaded);
      }
    }
    __syncwarp();
  } else if (warp < NG * NW) {
    for (int i = tid; i < P::TWB / 16; i += NG * T)
      *reinterpret_cast<float4*>(smem + P::OFF_TW + 16 * i) = __ldg(a.tw + i);
    P::setup(a, smem + P::OFF_TW, tid);
  }
  __syncthreads();
  sm100::grid_dep_wait();
  sm100::grid_dep_launch();
  if (warp >= NG * NW) {
    if constexpr (P::BIG) asm volatile("setmaxnreg.dec.sync.aligned.u32 24;");
    if (producer && lane == 0) {
      uint32_t i = 0;
      if constexpr (P::BIG)
        for (; loaded < mine && loaded < NBUF; ++loaded) load(loaded);
      for (; i < mine; ++i) {
        const uint32_t b = i % NBUF;
        wait_or_abort(&done[b], (i / NBUF) & 1u, abort_flag);
        if (*abort_flag) break;
        const uint32_t t = blockIdx.x + i * step;
        int32_t crd[5];
        tile::tile_coords(a.out_cmul, a.out_omul, t % ncb, t / ncb, crd);
        tile::tma_store(&a.tmap_out, a.out_ndims, crd, base_u + b * P::BUF);
        if (loaded < mine) {
          tile::tma_store_wait_read();
          load(loaded++);
        }
      }
      tile::tma_store_wait_all();
      // after an abort: loads still in flight must land before the shared
      // memory is released
      for (; i < loaded; ++i) sm100::mbar_wait_bounded(&full[i % NFULL], (i / NFULL) & 1u, kWaitLimit);
    }
    __syncwarp();
  } else {
    if constexpr (P::BIG) asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    const int grp = NG == 1 ? 0 : tid / T, t = tid - grp * T;
    const Sync<T> sync{1 + grp};
    const typename P::State st(a, t);
    for (uint32_t i = grp; i < mine; i += NG) {
      const uint32_t b = i % NBUF;
      wait_or_abort(&full[i % NFULL], (i / NFULL) & 1u, abort_flag);
      P::run(a, st, base_u + b * P::BUF, base_u + P::OFF_TW, t, (blockIdx.x + i * step) % ncb, sync);
      sm100::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) tile::mbar_arrive(&done[b]);
    }
  }
  __syncthreads();
  if (tid == 0 && *abort_flag && a.status) atomicExch(a.status, kStatusTimeout);
}

}  // namespace reg
}  // namespace mcfft
