// fft_mma.cuh -- plain-form (FP16) pass of 256, 512 or 1024 points whose
// radix-16 stages run on the tensor cores from register fragments.
//
// L = 16 x 16 x R, R = 1, 2, 4; a 16K-point tile, 16 warps, two phases with
// one exchange (the tile loop, barriers and copies are fft_reg.cuh's):
//
//   phase 1   n = n1 NV + v, v = n2 R + n3: DFT-16 over n1, twiddle W_L^(k1 v)
//   phase 2   DFT-16 over n2, twiddle W_16R^(k2 n3), DFT-R over n3 in
//             registers (FP32), output X[k1 + 16 k2 + 256 k3]
//
// A DFT-16 of eight vectors is four mma.sync.m16n8k16: the A fragments hold
// the real embedding of the DFT-16 matrix (16 registers for the whole launch),
// a B fragment register is one complex FP16 point, so a word read from shared
// memory is an operand as it is, and an accumulator pair is one output of two
// vectors -- the packed FP32x2 operand of the twiddle product.  tcgen05 would
// need its operand staged in shared memory and its result read back from
// tensor memory: eight shared-memory crossings per tile instead of six, for a
// contraction of only 32 x 32.
//
// What bounds it: the copies, then the serial chain of a tile's phases.  2^20 x
// 64, counters of both passes: a sub-partition spends 14 and 26 cycles of the
// FP32 pipe on 32 points (two per packed instruction; the FP32 register form,
// RegPass, 31 and 40), 16 of the tensor pipe (eight per warp-wide m16n8k16)
// and 16 and 29 issue slots, where the copies of the tile alone take about 52.
// Both passes together 213 us, the copies alone 194.
//
// Every shared access moves 16 bytes: a thread's 32 points are eight chunks
// of four, and which digit runs within a chunk, along the lanes and along the
// warps is fixed per kind so that (a) the chunk's four points are four columns
// or vectors of one operand slot, or four operand slots of one vector, (b)
// a quarter warp touches eight distinct banks groups, and (c) phase 1 writes
// only slots its own warp has read.  in_at / ex_at / out_at give the byte of
// each point in the three layouts; all are linear over GF(2) in the index
// bits, and only bits 4..6 of an address mix several of them, so an access is
// (base ^ x) + a with x and a known at compile time.
// tests/reg_layout_check.cu checks all of this on the host.
#pragma once
#include <cmath>
#include <type_traits>

#include "fft_reg.cuh"

namespace mcfft {
namespace reg {

// D = A B + C, m16n8k16, FP16 operands, FP32 accumulators; FIRST: C = 0.
template <bool FIRST>
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (FIRST) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
  } else {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
}

// The A fragments (the same for every pass of a direction): output half mt,
// operand half s.
struct MmaFrags {
  uint32_t a[2][2][4];
  template <class A>
  __device__ __forceinline__ MmaFrags(const A& args, int t) {
    const uint4* f = args.bmat + (t & 31) * 4;
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const uint4 x = __ldg(f + mt * 2 + s);
        a[mt][s][0] = x.x;
        a[mt][s][1] = x.y;
        a[mt][s][2] = x.z;
        a[mt][s][3] = x.w;
      }
  }
};

// TP: 16384 points per tile; 4096 (rows in and out, where a warp needs no
// other) for small batches.
template <int L_, int KIND_, bool POST_, bool INV_, int TP_ = 16384>
struct MmaPass {
  static constexpr int L = L_, KIND = KIND_, TP = TP_, R = L / 256, NV = L / 16, C = TP / L;
  static constexpr bool POST = POST_, INV = INV_;
  static_assert(L == 256 || L == 512 || L == 1024, "16 x 16 x R");
  static_assert(!POST || KIND == kCC, "four-step twiddle on column passes");
  static_assert(TP == 16384 || (TP == 4096 && KIND == kRR), "tile size");
  static constexpr int T = TP / 32, NW = T / 32, NG = 1;
  static constexpr bool BIG = T == 512;
  static constexpr int NBUF = BIG ? 3 : 2, NFULL = NBUF, THREADS = T + (BIG ? 128 : 32), MINB = BIG ? 1 : 3;
  static constexpr int BUF = TP * 4, EI = 4, EO = 4;
  static constexpr bool ROWIN = KIND != kCC;
  // Phase 2 of row-input passes of 256 and 512 points reads the four operand
  // slots of a vector as one chunk (WK); elsewhere a chunk is four vectors.
  static constexpr bool WK = ROWIN && L < 1024;

  using u32 = uint32_t;
  static __host__ __device__ constexpr u32 bit(u32 x, int b) { return (x >> b) & 1u; }
  // x's low bits into the column bits the lanes and registers leave free
  // (row-input passes whose warps own 2 or 4 columns)
  static __host__ __device__ constexpr u32 wcol(u32 w) {
    return L == 1024 ? w : L == 512 ? (w & 3u) | (w >> 2) << 3 : (w & 3u) | (w >> 2) << 4;
  }

  // ------------------------------------------------------ the three layouts
  static __host__ __device__ constexpr u32 in_at(u32 n1, u32 v, u32 c) {
    if (!ROWIN) {
      const u32 row = v * 16 + n1, q = c >> 2;
      if (C == 16) return row * 64 + ((q ^ ((n1 >> 1) & 3u)) << 4) + (c & 3u) * 4;
      return ((c >> 5) << 15) + row * 128 + (((q & 7u) ^ (n1 & 7u)) << 4) + (c & 3u) * 4;
    }
    const u32 pos = n1 * NV + v, row = pos >> 5;
    return c * (L * 4) + row * 128 + ((((pos >> 2) ^ row) & 7u) << 4) + (pos & 3u) * 4;
  }
  static __host__ __device__ constexpr u32 ex_at(u32 k1, u32 v, u32 c) {
    if (!ROWIN) {
      const u32 q = c >> 2, row = v * 16 + k1;
      if (C == 64)
        return ((c >> 5) << 15) + row * 128 +
               (((q & 7u) ^ (bit(v, 0) << 1 | (bit(v, 1) ^ bit(k1, 0)) << 2)) << 4) + (c & 3u) * 4;
      if (C == 32)
        return row * 128 + ((q ^ (bit(v, 1) << 1 | (bit(v, 2) ^ bit(k1, 0)) << 2)) << 4) + (c & 3u) * 4;
      return (row >> 1) * 128 +
             (((q | bit(k1, 0) << 2) ^ (bit(v, 2) | bit(v, 0) << 1 | bit(v, 3) << 2)) << 4) + (c & 3u) * 4;
    }
    if (L == 1024)
      return c * 4096 + (k1 * 2 + bit(v, 5)) * 128 +
             ((((v >> 2) & 7u) ^ (bit(k1, 0) | (bit(k1, 0) ^ bit(c, 0)) << 2)) << 4) + (v & 3u) * 4;
    if (L == 512)
      return c * 2048 + k1 * 128 + (((v & 7u) ^ (bit(c, 2) | bit(k1, 0) << 1)) << 4) + (v >> 3) * 4;
    return c * 1024 + (k1 >> 1) * 128 +
           ((((v & 3u) | bit(k1, 0) << 2) ^ (bit(c, 2) | bit(c, 3) << 1 | bit(c, 0) << 2)) << 4) + (v >> 2) * 4;
  }
  static __host__ __device__ constexpr u32 out_at(u32 k1, u32 k2, u32 k3, u32 c) {
    if (KIND == kRR) {
      const u32 pos = k1 + 16 * k2 + 256 * k3, row = pos >> 5;
      return c * (L * 4) + row * 128 + ((((pos >> 2) ^ row) & 7u) << 4) + (pos & 3u) * 4;
    }
    const u32 q = c >> 2;
    const u32 row = (k1 * R + k3) * 16 + k2;
    if (C == 16) return row * 64 + ((q ^ ((k2 >> 1) & 3u)) << 4) + (c & 3u) * 4;
    return ((c >> 5) << 15) + row * 128 + (((q & 7u) ^ (k2 & 7u)) << 4) + (c & 3u) * 4;
  }

  // -------------------------------------------------- who handles which point
  // Phase 1 vector (v, c) of vector bits g (three), register bits h (one), w
  // (two) and the warp; operand slot n1 = q + 4 i.
  struct VC {
    u32 v, c;
  };
  static __host__ __device__ constexpr VC p1(u32 g, u32 h, u32 w, u32 warp) {
    const u32 g0 = bit(g, 0), g1 = bit(g, 1), g2 = bit(g, 2);
    if (!ROWIN) {
      if (C == 64) return {warp, w | g1 << 2 | g2 << 3 | g0 << 4 | h << 5};
      if (C == 32) return {h | warp << 1, w | g1 << 2 | g2 << 3 | g0 << 4};
      return {g2 | h << 1 | warp << 2, w | g1 << 2 | g0 << 3};
    }
    if (L == 1024) return {w | g0 << 2 | g1 << 3 | g2 << 4 | h << 5, warp};
    if (L == 512) return {w | g1 << 2 | h << 3 | g0 << 4, g2 << 2 | wcol(warp)};
    return {w | h << 2 | g0 << 3, g1 << 2 | g2 << 3 | wcol(warp)};
  }
  // Phase 2 vector (k1, n3, c) of vector bits g, register unit u (three bits:
  // w + 4 h, or the load's index where a chunk is one vector) and the warp.
  struct KNC {
    u32 k1, n3, c;
  };
  static __host__ __device__ constexpr KNC p2(u32 g, u32 u, u32 warp) {
    const u32 g0 = bit(g, 0), g1 = bit(g, 1), g2 = bit(g, 2), w = u & 3u, h = u >> 2;
    const u32 u0 = bit(u, 0), u1 = bit(u, 1), u2 = bit(u, 2);
    if (!ROWIN) {
      if (C == 64) return {warp, 0, w | g << 2 | h << 5};
      if (C == 32) return {warp, h, w | g << 2};
      return {warp, g0 | h << 1, w | g1 << 2 | g2 << 3};
    }
    if (L == 1024) {
      const u32 x = g0 | h << 1 | g1 << 2 | g2 << 3;
      return KIND == kRR ? KNC{x, w, warp} : KNC{warp, w, x};
    }
    if (L == 512)
      return KIND == kRR ? KNC{u1 | u2 << 1 | g1 << 2 | g2 << 3, u0, g0 << 2 | wcol(warp)}
                         : KNC{warp, u0, u1 | u2 << 1 | g << 2};
    return KIND == kRR ? KNC{g0 | u0 << 1 | g1 << 2 | g2 << 3, 0, u1 << 2 | u2 << 3 | wcol(warp)}
                       : KNC{warp, 0, g0 | u0 << 1 | u1 << 2 | g1 << 3 | g2 << 4 | u2 << 5};
  }
  static __host__ __device__ constexpr u32 v_of(u32 n2, u32 n3) { return n2 * R + n3; }

  // Row kinds: byte in the tile's transforms, one after another, of byte off
  // of the buffer.
  static __host__ __device__ constexpr u32 in_map(u32 off) { return off ^ ((off >> 3) & 0x70u); }
  static __host__ __device__ constexpr u32 out_map(u32 off) { return in_map(off); }

  // Offsets of a thread's chunks: thread part, and register part (linear).
  static constexpr u32 XM = 0x70u;
  static __host__ __device__ constexpr u32 load1_t(u32 lane, u32 warp) {
    const VC a = p1(lane >> 2, 0, 0, warp);
    return in_at(lane & 3u, a.v, a.c);
  }
  static __host__ __device__ constexpr u32 load1_r(u32 h, u32 i) {
    const VC a = p1(0, h, 0, 0);
    return in_at(4 * i, a.v, a.c);
  }
  // Output lanes: q = vector bits 1, 2, g = low output bits; p = vector bit 0.
  static __host__ __device__ constexpr u32 store1_t(u32 lane, u32 warp) {
    const VC a = p1((lane & 3u) << 1, 0, 0, warp);
    return ex_at(lane >> 2, a.v, a.c);
  }
  static __host__ __device__ constexpr u32 store1_r(u32 mt, u32 p, u32 h, u32 w) {
    const VC a = p1(p, h, w, 0);
    return ex_at(8 * mt, a.v, a.c);
  }
  static __host__ __device__ constexpr u32 load2_t(u32 lane, u32 warp) {
    const KNC a = p2(lane >> 2, 0, warp);
    return ex_at(a.k1, v_of(lane & 3u, a.n3), a.c);
  }
  // load j: WK: unit j; else (h, i) = (j >> 2, j & 3)
  static __host__ __device__ constexpr u32 load2_r(u32 j) {
    if (WK) {
      const KNC a = p2(0, j, 0);
      return ex_at(a.k1, v_of(0, a.n3), a.c);
    }
    const KNC a = p2(0, (j >> 2) << 2, 0);
    return ex_at(a.k1, v_of(4 * (j & 3u), a.n3), a.c);
  }
  static __host__ __device__ constexpr u32 store2_t(u32 lane, u32 warp) {
    const KNC a = p2((lane & 3u) << 1, 0, warp);
    return out_at(a.k1, lane >> 2, 0, a.c);
  }
  // unit u's column / k1 bits and vector bit p, output digit bits mt and k3
  static __host__ __device__ constexpr u32 store2_r(u32 mt, u32 p, u32 u, u32 k3) {
    const KNC a = p2(p, u, 0);
    return out_at(a.k1, 8 * mt, k3, a.c);
  }

  // -------------------------------------------------------- twiddle tables
  // Phase 1, 16-byte pairs (vector bit p = 0, 1), index ((class * N1) + entry)
  // * LC + lane class; entries (mt, h, w) of row kinds, (mt, h) or (mt) of
  // column kinds (whose w, and at C = 64 also h, are columns).  Phase 2 (R >
  // 1, scaled by 1 / R): see tw2_n3.
  static constexpr int N1 = ROWIN ? 16 : C == 64 ? 2 : 4;
  static constexpr int LC = ROWIN ? (L == 1024 ? 32 : L == 512 ? 16 : 8) : (C == 16 ? 16 : 8);
  static constexpr int NCL = ROWIN ? 1 : 16;  // warp classes
  static __host__ __device__ constexpr u32 lane_class(u32 lane) {
    const u32 q = lane & 3u, g = lane >> 2;
    if (LC == 32) return lane;
    if (LC == 16) return g + 8 * (ROWIN ? q & 1u : q >> 1);
    return g;
  }
  static constexpr int N2 = R == 1 ? 0 : R == 2 ? 2 : ROWIN ? 6 : 4;
  static constexpr int TW1B = NCL * N1 * LC * 16, TWB = TW1B + N2 * 8 * 16;
  // Four-step twiddles W_N^(k col): a thread's outputs are four packed chains
  // (mt, z) over its four columns w, z = h (L = 256), k3 (512) or the pair
  // (2 z, 2 z + 1) of k3 (1024), each started once per tile and advanced by
  // its step W_N^k from one column to the next.  Step table: 16 bytes at
  // ((k1 * 4 + mt * 2 + z) * 8 + g) * 16; L < 1024 also W_N^(4 k), 8 bytes,
  // and L = 256 W_N^(32 k), in the same order.  Filled by the kernel itself
  // (N is the plan's).
  static constexpr int PSTEPB = POST ? 512 * 16 : 0, PQB = POST && L < 1024 ? 512 * 8 : 0;
  static constexpr int PHB = POST && L == 256 ? 512 * 8 : 0;
  static constexpr int OFF_PSTEP = TWB, OFF_PQ = OFF_PSTEP + PSTEPB, OFF_PH = OFF_PQ + PQB;
  // Entry e of the phase-2 table: output half mt and the n3 of the pair's two
  // lanes: one n3 for both (doubled), or n3 = 2 h + p (column kind, R = 4).
  static __host__ __device__ constexpr u32 tw2_mt(int e) { return R == 2 ? e : ROWIN ? e / 3 : e / 2; }
  static __host__ __device__ constexpr u32 tw2_n3(int e, int p) {
    return R == 2 ? 1 : ROWIN ? e % 3 + 1 : 2 * (e % 2) + p;
  }

  static constexpr int OFF_TW = NBUF * BUF;
  static constexpr int OFF_BAR = OFF_TW + TWB + PSTEPB + PQB + PHB;
  static constexpr int SMEM_BYTES = OFF_BAR + 128 + 1024;
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");

  static constexpr int TABB = OFF_BAR - OFF_TW;  // all tables
  using State = MmaFrags;

  // DFT-16 of the unit whose operand slots are b0 .. b3: pairs re[mt], im[mt].
  static __device__ __forceinline__ void unit(const State& st, u32 b0, u32 b1, u32 b2, u32 b3, P2 (&re)[2],
                                              P2 (&im)[2]) {
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
      float d[4];
      mma16816<true>(d, st.a[mt][0], b0, b1);
      mma16816<false>(d, st.a[mt][1], b2, b3);
      re[mt] = pack2(d[0], d[1]);
      im[mt] = pack2(d[2], d[3]);
    }
  }
  static __device__ __forceinline__ void to_words(P2 re, P2 im, u32& w0, u32& w1) {
    float r0, r1, i0, i1;
    f2u(re.v, r0, r1);
    f2u(im.v, i0, i1);
    w0 = sm100::pack_half2(r0, i0);
    w1 = sm100::pack_half2(r1, i1);
  }
  static __device__ __forceinline__ void put(u32 base, u32 d, const u32 (&w)[4]) {
    tile::sts128((base ^ (d & XM)) + (d & ~XM), make_uint4(w[0], w[1], w[2], w[3]));
  }

  static __device__ __forceinline__ P2 dup(float x) { return pack2(x, x); }

  // W_N^e; e may wrap modulo 2^32, which N divides.
  template <class A>
  static __device__ __forceinline__ float2 post(const A& a, u32 e) {
    e &= (u32)a.post_mask;
    if (a.post_scale == 0.f)
      return cmulf(__ldg(a.post_a + (e & ((1u << a.post_shift) - 1))), __ldg(a.post_b + (e >> a.post_shift)));
    float x = (float)e * a.post_scale;  // [0, 2)
    x = x >= 1.f ? x - 2.f : x;
    float sn, cs;
    __sincosf(x * 3.14159265358979f, &sn, &cs);
    return make_float2(cs, INV ? sn : -sn);
  }
  // Fills the step tables (threads t of T).
  template <class A>
  static __device__ __forceinline__ void setup(const A& a, uint8_t* tw, int t) {
    if constexpr (POST) {
      const u32 g = t & 7, z = (t >> 3) & 1, mt = (t >> 4) & 1, k1 = t >> 5;
      const u32 kb = k1 + 16 * (g + 8 * mt);
      float4 st;
      if constexpr (L == 1024) {
        const float2 s0 = post(a, kb + 512 * z), s1 = post(a, kb + 512 * z + 256);
        st = make_float4(s0.x, s1.x, s0.y, s1.y);
      } else {
        const u32 k = kb + (L == 512 ? 256 * z : 0);
        const float2 s0 = post(a, k);
        st = make_float4(s0.x, s0.x, s0.y, s0.y);
        *reinterpret_cast<float2*>(tw + OFF_PQ + 8 * t) = post(a, 4 * k);
        if constexpr (L == 256) *reinterpret_cast<float2*>(tw + OFF_PH + 8 * t) = post(a, 32 * k * z);
      }
      *reinterpret_cast<float4*>(tw + OFF_PSTEP + 16 * t) = st;
    }
  }
  // The four chains of a tile.
  struct Chains {
    P2 r[2][2], i[2][2];
    u32 tab;
    template <class A>
    __device__ __forceinline__ Chains(const A& a, u32 tws, u32 cb, u32 lane, u32 warp) {
      const u32 g = lane >> 2, q = lane & 3u, kb = warp + 16 * g;
      const u32 col = cb * C + (C == 16 ? 4 : 8) * q;  // of w = p = h = 0
      tab = tws + OFF_PSTEP + (warp * 32 + g) * 16;
      float2 tt = make_float2(1.f, 0.f), tq = tt;
      if constexpr (L > 256) tt = post(a, 256 * col);
      if constexpr (L == 1024) tq = cmulf(tt, tt);
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        const float2 e = post(a, (kb + 128 * mt) * col);
        if constexpr (L == 1024) {
          const float2 et = cmulf(e, tt);
          r[mt][0] = r[mt][1] = pack2(e.x, et.x);
          i[mt][0] = i[mt][1] = pack2(e.y, et.y);
          cmulv(r[mt][1], i[mt][1], dup(tq.x), dup(tq.y));
        } else {
#pragma unroll
          for (int z = 0; z < 2; ++z) {
            const u32 at = (warp * 32 + (mt * 2 + z) * 8 + g) * 8;
            const float2 s4 = lds64f(tws + OFF_PQ + at);
            const float2 e0 = z == 0 ? e : cmulf(e, L == 512 ? tt : lds64f(tws + OFF_PH + at));
            const float2 e4 = cmulf(e0, s4);
            r[mt][z] = pack2(e0.x, e4.x);
            i[mt][z] = pack2(e0.y, e4.y);
          }
        }
      }
    }
    // (re, im) times chain (mt, z)
    __device__ __forceinline__ void apply(int mt, int z, P2& re, P2& im) const { cmulv(re, im, r[mt][z], i[mt][z]); }
    __device__ __forceinline__ void step(int mt, int z) {
      const float4 f = lds128f(tab + (mt * 2 + z) * 128);
      cmulv(r[mt][z], i[mt][z], pack2(f.x, f.y), pack2(f.z, f.w));
    }
  };
  struct NoChains {
    template <class A>
    __device__ __forceinline__ NoChains(const A&, u32, u32, u32, u32) {}
    __device__ __forceinline__ void apply(int, int, P2&, P2&) const {}
    __device__ __forceinline__ void step(int, int) {}
  };

  template <class A>
  static __device__ __forceinline__ void run(const A& a, const State& st, u32 sb, u32 tws, int t, u32 cb,
                                             const Sync<T>& sync) {
    const u32 lane = t & 31, warp = t >> 5;
    u32 x[8][4];  // this thread's chunks
    {             // --------------------------------------------------- phase 1
      const u32 lb = sb + load1_t(lane, warp), sp = sb + store1_t(lane, warp);
      const u32 tw = tws + ((ROWIN ? 0 : warp) * (N1 * LC) + lane_class(lane)) * 16;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const u32 d = load1_r(j >> 2, j & 3);
        const uint4 v = tile::lds128((lb ^ (d & XM)) + (d & ~XM));
        x[j][0] = v.x;
        x[j][1] = v.y;
        x[j][2] = v.z;
        x[j][3] = v.w;
      }
      __syncwarp();
      auto one = [&](int h, int w, u32 (&o)[2][2]) {  // [mt][p]
        P2 re[2], im[2];
        unit(st, x[4 * h][w], x[4 * h + 1][w], x[4 * h + 2][w], x[4 * h + 3][w], re, im);
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
          const int e = ROWIN ? mt * 8 + h * 4 + w : C == 64 ? mt : mt * 2 + h;
          const float4 f = lds128f(tw + e * (LC * 16));
          cmulv(re[mt], im[mt], pack2(f.x, f.y), pack2(f.z, f.w));
          to_words(re[mt], im[mt], o[mt][0], o[mt][1]);
        }
      };
      if constexpr (!WK) {  // a chunk holds the four w
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          u32 o[2][2][4];
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            u32 z[2][2];
            one(h, w, z);
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
              o[mt][0][w] = z[mt][0];
              o[mt][1][w] = z[mt][1];
            }
          }
#pragma unroll
          for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int p = 0; p < 2; ++p) put(sp, store1_r(mt, p, h, 0), o[mt][p]);
        }
      } else {  // a chunk holds (h, p): the operand slots of phase 2
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          u32 o[2][4];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            u32 z[2][2];
            one(h, w, z);
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
              o[mt][h] = z[mt][0];
              o[mt][h + 2] = z[mt][1];
            }
          }
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) put(sp, store1_r(mt, 0, 0, w), o[mt]);
        }
      }
    }
    if constexpr (KIND == kRR) __syncwarp();
    else sync.group();
    {  // --------------------------------------------------------------- phase 2
      const u32 lb = sb + load2_t(lane, warp), sp = sb + store2_t(lane, warp);
      const u32 tw2 = tws + TW1B + (lane >> 2) * 16;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const u32 d = load2_r(j);
        const uint4 v = tile::lds128((lb ^ (d & XM)) + (d & ~XM));
        x[j][0] = v.x;
        x[j][1] = v.y;
        x[j][2] = v.z;
        x[j][3] = v.w;
      }
      // the chains' starts overlap the loads
      typename std::conditional<POST, Chains, NoChains>::type ch(a, tws, cb, lane, warp);
      if constexpr (KIND == kRR) __syncwarp();
      else sync.group();
      auto dft = [&](int u, P2 (&re)[2], P2 (&im)[2]) {
        if constexpr (WK) unit(st, x[u][0], x[u][1], x[u][2], x[u][3], re, im);
        else unit(st, x[(u & 4)][u & 3], x[(u & 4) + 1][u & 3], x[(u & 4) + 2][u & 3], x[(u & 4) + 3][u & 3], re, im);
      };
      auto twid = [&](int e, P2& re, P2& im) {
        const float4 f = lds128f(tw2 + e * 128);
        cmulv(re, im, pack2(f.x, f.y), pack2(f.z, f.w));
      };
      if constexpr (L == 256 && KIND == kCC) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          u32 o[2][2][4];
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            P2 re[2], im[2];
            dft(w + 4 * h, re, im);
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
              ch.apply(mt, h, re[mt], im[mt]);
              if (w < 3) ch.step(mt, h);
              to_words(re[mt], im[mt], o[mt][0][w], o[mt][1][w]);
            }
          }
#pragma unroll
          for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int p = 0; p < 2; ++p) put(sp, store2_r(mt, p, 4 * h, 0), o[mt][p]);
        }
      } else if constexpr (L == 256) {  // chunk = (p, u0)
#pragma unroll
        for (int uu = 0; uu < 8; uu += 2) {
          u32 o[2][4];
#pragma unroll
          for (int u0 = 0; u0 < 2; ++u0) {
            P2 re[2], im[2];
            dft(uu + u0, re, im);
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) to_words(re[mt], im[mt], o[mt][2 * u0], o[mt][2 * u0 + 1]);
          }
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) put(sp, store2_r(mt, 0, uu, 0), o[mt]);
        }
      } else if constexpr (L == 512) {
        // n3 = h (column kind, chunk = w) or u0 (row kinds, chunk = (u1, u2))
        u32 o[2][2][2][4];  // [mt][p][k3][word]
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          P2 zr[2], zi[2], yr[2], yi[2];
          dft(KIND == kCC ? w : 2 * w, zr, zi);
          dft(KIND == kCC ? w + 4 : 2 * w + 1, yr, yi);
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) {
            twid(mt, yr[mt], yi[mt]);
            const P2 hr = zr[mt] * dup(0.5f), hi = zi[mt] * dup(0.5f);
            P2 ar = hr + yr[mt], ai = hi + yi[mt], br = hr - yr[mt], bi = hi - yi[mt];
            ch.apply(mt, 0, ar, ai);
            ch.apply(mt, 1, br, bi);
            if (w < 3) {
              ch.step(mt, 0);
              ch.step(mt, 1);
            }
            to_words(ar, ai, o[mt][0][0][w], o[mt][1][0][w]);
            to_words(br, bi, o[mt][0][1][w], o[mt][1][1][w]);
          }
        }
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
          for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int k3 = 0; k3 < 2; ++k3) put(sp, store2_r(mt, p, 0, k3), o[mt][p][k3]);
      } else if constexpr (KIND != kCC) {
        // L = 1024, rows in: n3 = w, chunk = (p, h)
        u32 o[2][4][4];  // [mt][k3][word]
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          P2 zr[4][2], zi[4][2];
#pragma unroll
          for (int w = 0; w < 4; ++w) dft(w + 4 * h, zr[w], zi[w]);
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) {
            zr[0][mt] = zr[0][mt] * dup(0.25f);
            zi[0][mt] = zi[0][mt] * dup(0.25f);
#pragma unroll
            for (int w = 1; w < 4; ++w) twid(mt * 3 + w - 1, zr[w][mt], zi[w][mt]);
            dft4<INV>(zr[0][mt], zi[0][mt], zr[1][mt], zi[1][mt], zr[2][mt], zi[2][mt], zr[3][mt], zi[3][mt]);
#pragma unroll
            for (int k3 = 0; k3 < 4; ++k3)
              to_words(zr[k3][mt], zi[k3][mt], o[mt][k3][2 * h], o[mt][k3][2 * h + 1]);
          }
        }
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
          for (int k3 = 0; k3 < 4; ++k3) put(sp, store2_r(mt, 0, 0, k3), o[mt][k3]);
      } else {
        // L = 1024, columns: n3 = 2 h + p: the first radix-2 step is packed
        // (over h), the second runs across the pair; chunk = w
        u32 o[2][4][4];  // [mt][k3][word]
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          P2 zr[2], zi[2], yr[2], yi[2];
          dft(w, zr, zi);
          dft(w + 4, yr, yi);
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) {
            twid(mt * 2, zr[mt], zi[mt]);
            twid(mt * 2 + 1, yr[mt], yi[mt]);
            const P2 ar = zr[mt] + yr[mt], ai = zi[mt] + yi[mt], br = zr[mt] - yr[mt], bi = zi[mt] - yi[mt];
            float a0r, a1r, a0i, a1i, b0r, b1r, b0i, b1i;
            f2u(ar.v, a0r, a1r);
            f2u(ai.v, a0i, a1i);
            f2u(br.v, b0r, b1r);
            f2u(bi.v, b0i, b1i);
            // X0, X2 = a0 +- a1, X1, X3 = b0 +- (SGN i) b1; pairs (0, 1), (2, 3)
            P2 r01 = pack2(a0r + a1r, INV ? b0r - b1i : b0r + b1i);
            P2 i01 = pack2(a0i + a1i, INV ? b0i + b1r : b0i - b1r);
            P2 r23 = pack2(a0r - a1r, INV ? b0r + b1i : b0r - b1i);
            P2 i23 = pack2(a0i - a1i, INV ? b0i - b1r : b0i + b1r);
            ch.apply(mt, 0, r01, i01);
            ch.apply(mt, 1, r23, i23);
            if (w < 3) {
              ch.step(mt, 0);
              ch.step(mt, 1);
            }
            to_words(r01, i01, o[mt][0][w], o[mt][1][w]);
            to_words(r23, i23, o[mt][2][w], o[mt][3][w]);
          }
        }
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
          for (int k3 = 0; k3 < 4; ++k3) put(sp, store2_r(mt, 0, 0, k3), o[mt][k3]);
      }
    }
  }

  // ------------------------------------------------------ host-side tables
  // The twiddle table (TWB bytes), FP64 rounded once.
  static void fill_twiddles(float* out) {
    constexpr double pi2 = 6.283185307179586476925286766559, sgn = INV ? 1.0 : -1.0;
    auto set = [&](u32 at, int p, u32 e, u32 mod, double scale) {
      const double x = pi2 * (double)(e % mod) / (double)mod;
      out[at * 4 + p] = (float)(scale * std::cos(x));
      out[at * 4 + 2 + p] = (float)(scale * sgn * std::sin(x));
    };
    for (u32 wc = 0; wc < (u32)NCL; ++wc)
      for (u32 e = 0; e < (u32)N1; ++e)
        for (u32 lane = 0; lane < 32; ++lane)
          for (u32 p = 0; p < 2; ++p) {
            const u32 mt = ROWIN ? e >> 3 : C == 64 ? e : e >> 1;
            const u32 h = ROWIN ? (e >> 2) & 1u : C == 64 ? 0 : e & 1u, w = ROWIN ? e & 3u : 0;
            const VC a = p1((lane & 3u) << 1 | p, h, w, wc);
            set((wc * N1 + e) * LC + lane_class(lane), p, ((lane >> 2) + 8 * mt) * a.v, L, 1.0);
          }
    for (int e = 0; e < N2; ++e)
      for (u32 g = 0; g < 8; ++g)
        for (u32 p = 0; p < 2; ++p)
          set(TW1B / 16 + e * 8 + g, p, (g + 8 * tw2_mt(e)) * tw2_n3(e, p), 16 * R, 1.0 / R);
  }
  // The A fragments (32 lanes x 16 words): the real embedding of the DFT-16
  // matrix times 1 / 16 (exact) in FP16, operand column (slot, re / im) of
  // lane q's slots q + 4 i, output row g + 8 mt (real part, then imaginary).
  static void fill_fragments(uint32_t* out) {
    constexpr double pi2 = 6.283185307179586476925286766559, sgn = INV ? 1.0 : -1.0;
    auto half_bits = [](double x) {
      const __half_raw r = static_cast<__half_raw>(__double2half(x));
      return (u32)r.x;
    };
    for (u32 lane = 0; lane < 32; ++lane)
      for (u32 mt = 0; mt < 2; ++mt)
        for (u32 s = 0; s < 2; ++s)
          for (u32 i = 0; i < 4; ++i) {
            const u32 k = (lane >> 2) + 8 * mt, n = (lane & 3u) + 4 * (2 * s + (i >> 1));
            // sines and cosines of multiples of pi / 8, exact where they are 0 or 1
            const u32 e = (k * n) % 16;
            const double c = e % 8 == 4 ? 0.0 : std::cos(pi2 * e / 16.0), sn = e % 8 == 0 ? 0.0 : std::sin(pi2 * e / 16.0);
            const double re = i & 1 ? sgn * sn : c, im = i & 1 ? c : -sgn * sn;
            out[lane * 16 + (mt * 2 + s) * 4 + i] = half_bits(re / 16.0) | half_bits(im / 16.0) << 16;
          }
  }
};

}  // namespace reg
}  // namespace mcfft
