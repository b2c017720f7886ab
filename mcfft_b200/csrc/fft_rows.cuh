// fft_rows.cuh -- row passes of 4096 and 2048 points (1D transforms of these
// lengths in one pass), a transform to four (two) warps.
//
// 4096 points: three radix-16 phases,
//   n = 256 n1 + 16 n2 + n3, X[k1 + 16 k2 + 256 k3]
//   phase 1  DFT-16 over n1, twiddle W_4096^(k1 (16 n2 + n3))
//   phase 2  DFT-16 over n2, twiddle W_256^(k2 n3)
//   phase 3  DFT-16 over n3
//
// Phases 1 and 2 write in place (slots of the writing warp); phase 3 puts the
// result into natural order.  Three barriers of four warps per transform
// (FP16 input with FP32 exchange: four), three or four CTAs per SM so that
// their phases overlap: such batches are small more often than not, and a
// 16K-point tile of four transforms (fft_tile.cuh) leaves most SMs idle and
// takes four times as long per tile.  The one-launch kernel of uneven batches
// runs four transforms per 16K-point tile.
//
// 2048 points (plain form): 16 x 16 x 8, two phases as MmaPass with the
// radix-8 step in registers, eight transforms per 16K-point tile.  Bound by
// HBM from a few thousand transforms: 20000 in 61 us (5.4 TB/s), 80 on the
// tcgen05 tile of eight columns; 3000 in 15 against 24 us; as the rows of
// 2048^2 x 4, 64 against 74 us in all.
#pragma once
#include "fft_mma.cuh"

namespace mcfft {
namespace reg {

// Barrier of the N threads of one transform (id: one per transform in work).
template <int N>
__device__ __forceinline__ void col_bar(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(N) : "memory");
}

// Plain form: the phases of MmaPass, every shared access 16 bytes wide and
// free of bank conflicts (tests/reg_layout_check.cu).
template <bool INV_, int TP_ = 4096>
struct Mma4096 {
  using u32 = uint32_t;
  static constexpr int L = 4096, KIND = kRR, TP = TP_, R = 16, C = TP / L, EI = 4, EO = 4;
  static constexpr bool POST = false, INV = INV_, BIG = C == 4;
  static_assert(C == 1 || C == 4, "tile size");
  static constexpr int T = TP / 32, NW = T / 32, NG = 1, NBUF = BIG ? 3 : 2, NFULL = NBUF;
  static constexpr int THREADS = T + (BIG ? 128 : 32), MINB = BIG ? 1 : 4;
  static constexpr int BUF = TP * 4;
  using State = MmaFrags;
  static __host__ __device__ constexpr u32 bit(u32 x, int b) { return (x >> b) & 1u; }

  // ------------------------------------------------------------ the layouts
  // 128-byte rows of 32 points; rows 16 (n2 >> 1) + n1, so that the 128-byte
  // swizzle (row & 7) runs along n1 (output: along k3).
  static __host__ __device__ constexpr u32 in_at(u32 n1, u32 n2, u32 n3) {
    return ((n2 >> 1) * 16 + n1) * 128 + ((((n2 & 1u) << 2 | n3 >> 2) ^ (n1 & 7u)) << 4) + (n3 & 3u) * 4;
  }
  static __host__ __device__ constexpr u32 ex1_at(u32 k1, u32 n2, u32 n3) {
    return ((n2 >> 1) * 16 + k1) * 128 +
           ((((n2 & 1u) << 2 | n3 >> 2) ^ (bit(n2, 1) << 1 | bit(k1, 0) << 2)) << 4) + (n3 & 3u) * 4;
  }
  static __host__ __device__ constexpr u32 ex2_at(u32 k1, u32 k2, u32 n3) {
    return ((k2 >> 1) * 16 + k1) * 128 +
           ((((k2 & 1u) << 2 | (n3 & 3u)) ^ (bit(k1, 2) | bit(k1, 3) << 1 | bit(k1, 0) << 2)) << 4) + (n3 >> 2) * 4;
  }
  static __host__ __device__ constexpr u32 out_at(u32 k1, u32 k2, u32 k3) {
    return ((k2 >> 1) * 16 + k3) * 128 + ((((k2 & 1u) << 2 | k1 >> 2) ^ (k3 & 7u)) << 4) + (k1 & 3u) * 4;
  }
  // byte in the transforms, one after another, of byte off of the buffer
  static __host__ __device__ constexpr u32 in_map(u32 off) {
    return (off & ~0x3fffu) + ((off >> 7) & 15u) * 1024 + ((off >> 11) & 7u) * 128 + ((off ^ off >> 3) & 0x70u) + (off & 15u);
  }
  static __host__ __device__ constexpr u32 out_map(u32 off) { return in_map(off); }
  // ------------------------------------------------- who handles which point
  struct XY {
    u32 x, y;
  };
  // phase 1: (n2, n3); phase 2: (k1, n3); phase 3: (k1, k2), u the load index
  static __host__ __device__ constexpr XY p1(u32 g, u32 h, u32 w, u32 warp) {
    return {bit(g, 0) | bit(g, 1) << 1 | warp << 2, w | bit(g, 2) << 2 | h << 3};
  }
  static __host__ __device__ constexpr XY p2(u32 g, u32 h, u32 w, u32 warp) {
    return {warp | bit(g, 1) << 2 | bit(g, 2) << 3, w | bit(g, 0) << 2 | h << 3};
  }
  static __host__ __device__ constexpr XY p3(u32 g, u32 u, u32 warp) {
    return {bit(g, 0) | bit(u, 0) << 1 | bit(u, 1) << 2 | bit(g, 1) << 3,
            bit(g, 2) | bit(u, 2) << 1 | warp << 2};
  }
  static constexpr u32 XM = 0x70u;
  static __host__ __device__ constexpr u32 load1_t(u32 lane, u32 warp) {
    const XY a = p1(lane >> 2, 0, 0, warp);
    return in_at(lane & 3u, a.x, a.y);
  }
  static __host__ __device__ constexpr u32 load1_r(u32 h, u32 i) {
    const XY a = p1(0, h, 0, 0);
    return in_at(4 * i, a.x, a.y);
  }
  static __host__ __device__ constexpr u32 store1_t(u32 lane, u32 warp) {
    const XY a = p1((lane & 3u) << 1, 0, 0, warp);
    return ex1_at(lane >> 2, a.x, a.y);
  }
  static __host__ __device__ constexpr u32 store1_r(u32 mt, u32 p, u32 h) {
    const XY a = p1(p, h, 0, 0);
    return ex1_at(8 * mt, a.x, a.y);
  }
  static __host__ __device__ constexpr u32 load2_t(u32 lane, u32 warp) {
    const XY a = p2(lane >> 2, 0, 0, warp);
    return ex1_at(a.x, lane & 3u, a.y);
  }
  static __host__ __device__ constexpr u32 load2_r(u32 h, u32 i) {
    const XY a = p2(0, h, 0, 0);
    return ex1_at(a.x, 4 * i, a.y);
  }
  static __host__ __device__ constexpr u32 store2_t(u32 lane, u32 warp) {
    const XY a = p2((lane & 3u) << 1, 0, 0, warp);
    return ex2_at(a.x, lane >> 2, a.y);
  }
  static __host__ __device__ constexpr u32 store2_r(u32 mt, u32 w) {
    const XY a = p2(0, 0, w, 0);
    return ex2_at(a.x, 8 * mt, a.y);
  }
  static __host__ __device__ constexpr u32 load3_t(u32 lane, u32 warp) {
    const XY a = p3(lane >> 2, 0, warp);
    return ex2_at(a.x, a.y, lane & 3u);
  }
  static __host__ __device__ constexpr u32 load3_r(u32 u) {
    const XY a = p3(0, u, 0);
    return ex2_at(a.x, a.y, 0);
  }
  static __host__ __device__ constexpr u32 store3_t(u32 lane, u32 warp) {
    const XY a = p3((lane & 3u) << 1, 0, warp);
    return out_at(a.x, a.y, lane >> 2);
  }
  static __host__ __device__ constexpr u32 store3_r(u32 mt, u32 u) {
    const XY a = p3(0, u, 0);
    return out_at(a.x, a.y, 8 * mt);
  }

  // ---------------------------------------------------------------- tables
  // Phase 1: a chain per (mt, h) over the chunk words w, its start (pairs
  // over vector bit 0) at ((warp * 4 + mt * 2 + h) * 32 + lane), its step
  // W_4096^k1 (doubled) at 512 + k1; phase 2: pairs at 528 + (mt * 8 + h * 4 +
  // w) * 8 + g.  16-byte entries.
  static constexpr int TWB = (512 + 16 + 128) * 16, TABB = TWB;
  static constexpr int OFF_TW = NBUF * BUF, OFF_BAR = OFF_TW + TWB;
  static constexpr int SMEM_BYTES = OFF_BAR + 128 + 1024;
  static void fill_twiddles(float* out) {
    constexpr double pi2 = 6.283185307179586476925286766559, sgn = INV ? 1.0 : -1.0;
    auto set = [&](u32 at, u32 p, u32 e, u32 mod) {
      const double x = pi2 * (double)(e % mod) / (double)mod;
      out[at * 4 + p] = (float)std::cos(x);
      out[at * 4 + 2 + p] = (float)(sgn * std::sin(x));
    };
    for (u32 p = 0; p < 2; ++p) {
      for (u32 warp = 0; warp < 4; ++warp)
        for (u32 mh = 0; mh < 4; ++mh)
          for (u32 lane = 0; lane < 32; ++lane) {
            const XY a = p1((lane & 3u) << 1 | p, mh & 1u, 0, warp);
            set((warp * 4 + mh) * 32 + lane, p, ((lane >> 2) + 8 * (mh >> 1)) * (16 * a.x + a.y), 4096);
          }
      for (u32 k1 = 0; k1 < 16; ++k1) set(512 + k1, p, k1, 4096);
      for (u32 e = 0; e < 16; ++e)
        for (u32 g = 0; g < 8; ++g)
          set(528 + e * 8 + g, p, (g + 8 * (e >> 3)) * p2(p, (e >> 2) & 1u, e & 3u, 0).y, 256);
    }
  }
  static void fill_fragments(uint32_t* out) { MmaPass<256, kRR, false, INV>::fill_fragments(out); }

  template <class A>
  static __device__ __forceinline__ void setup(const A&, uint8_t*, int) {}

  static __device__ __forceinline__ void get(u32 base, u32 d, u32 (&x)[4]) {
    const uint4 v = tile::lds128((base ^ (d & XM)) + (d & ~XM));
    x[0] = v.x;
    x[1] = v.y;
    x[2] = v.z;
    x[3] = v.w;
  }
  using M = MmaPass<256, kRR, false, INV>;

  template <class A>
  static __device__ __forceinline__ void run(const A&, const State& st, u32 sb, u32 tws, int t, u32,
                                             const Sync<T>&) {
    const u32 lane = t & 31, warp = (t >> 5) & 3u, g = lane >> 2;
    const int bar = 4 + (t >> 7);
    sb += (t >> 7) * 16384;
    u32 x[8][4];
    {
      const u32 lb = sb + load1_t(lane, warp), sp = sb + store1_t(lane, warp);
#pragma unroll
      for (int j = 0; j < 8; ++j) get(lb, load1_r(j >> 2, j & 3), x[j]);
      __syncwarp();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        P2 cr[2], ci[2];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
          const float4 f = lds128f(tws + ((warp * 4 + mt * 2 + h) * 32 + lane) * 16);
          cr[mt] = pack2(f.x, f.y);
          ci[mt] = pack2(f.z, f.w);
        }
        u32 o[2][2][4];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          P2 re[2], im[2];
          M::unit(st, x[4 * h][w], x[4 * h + 1][w], x[4 * h + 2][w], x[4 * h + 3][w], re, im);
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) {
            cmulv(re[mt], im[mt], cr[mt], ci[mt]);
            if (w < 3) {
              const float4 f = lds128f(tws + (512 + g + 8 * mt) * 16);
              cmulv(cr[mt], ci[mt], pack2(f.x, f.y), pack2(f.z, f.w));
            }
            M::to_words(re[mt], im[mt], o[mt][0][w], o[mt][1][w]);
          }
        }
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
          for (int p = 0; p < 2; ++p) M::put(sp, store1_r(mt, p, h), o[mt][p]);
      }
    }
    col_bar<128>(bar);
    {
      const u32 lb = sb + load2_t(lane, warp), sp = sb + store2_t(lane, warp);
#pragma unroll
      for (int j = 0; j < 8; ++j) get(lb, load2_r(j >> 2, j & 3), x[j]);
      __syncwarp();
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        u32 o[2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          P2 re[2], im[2];
          M::unit(st, x[4 * h][w], x[4 * h + 1][w], x[4 * h + 2][w], x[4 * h + 3][w], re, im);
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) {
            const float4 f = lds128f(tws + (528 + (mt * 8 + h * 4 + w) * 8 + g) * 16);
            cmulv(re[mt], im[mt], pack2(f.x, f.y), pack2(f.z, f.w));
            M::to_words(re[mt], im[mt], o[mt][2 * h], o[mt][2 * h + 1]);
          }
        }
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) M::put(sp, store2_r(mt, w), o[mt]);
      }
    }
    col_bar<128>(bar);
    {
      const u32 lb = sb + load3_t(lane, warp), sp = sb + store3_t(lane, warp);
#pragma unroll
      for (int u = 0; u < 8; ++u) get(lb, load3_r(u), x[u]);
      col_bar<128>(bar);
#pragma unroll
      for (int uu = 0; uu < 8; uu += 2) {
        u32 o[2][4];
#pragma unroll
        for (int u0 = 0; u0 < 2; ++u0) {
          P2 re[2], im[2];
          M::unit(st, x[uu + u0][0], x[uu + u0][1], x[uu + u0][2], x[uu + u0][3], re, im);
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) M::to_words(re[mt], im[mt], o[mt][2 * u0], o[mt][2 * u0 + 1]);
        }
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) M::put(sp, store3_r(mt, uu), o[mt]);
      }
    }
  }
};

// FP32 exchange and output (split form), FP16 or FP32 input; points in
// natural order in shared memory, no swizzle by TMA.
template <bool IN16_, bool INV_>
struct Reg4096 {
  using u32 = uint32_t;
  static constexpr int L = 4096, KIND = kRR, TP = 4096, R = 16, C = 1, EI = IN16_ ? 4 : 8, EO = 8;
  static constexpr bool POST = false, INV = INV_, BIG = false;
  static constexpr int T = 128, NW = 4, NG = 1, NBUF = 2, NFULL = 2, THREADS = T + 32, MINB = 3;
  static constexpr int BUF = TP * 8;
  struct State {
    template <class A>
    __device__ __forceinline__ State(const A&, int) {}
  };
  // A lane runs along one digit x of 16 and the lowest bit of another, y;
  // vector j and the warp give y's other bits.  Phases 1, 2: x = n3, y = n2,
  // k1; phase 3: x = k1, y = k2.
  static __host__ __device__ constexpr u32 xd(u32 t) { return t & 15u; }
  static __host__ __device__ constexpr u32 yd(u32 t, u32 j) { return ((t >> 4) & 1u) | j << 1 | (t >> 5) << 2; }
  static __host__ __device__ constexpr u32 in_map(u32 off) { return off; }
  static __host__ __device__ constexpr u32 out_map(u32 off) { return off; }
  // Slot of phase 2's output: 16-byte chunks of row (k1, k2) XORed with k1.
  static __host__ __device__ constexpr u32 ex2_at(u32 k1, u32 k2, u32 n3) {
    return (k1 * 256 + k2 * 16 + (n3 ^ ((k1 & 7u) << 1))) * 8;
  }
  // Twiddles W_256^(k n) at 16 k + n, then W_4096^(k n): phase 1's factor is
  // their product W_256^(k1 n2) W_4096^(k1 n3), a sixteenth of the one table.
  static constexpr int TWB = 512 * 8;
  static constexpr int OFF_TW = NBUF * BUF, OFF_BAR = OFF_TW + TWB;
  static constexpr int SMEM_BYTES = OFF_BAR + 128 + 1024;
  static void fill_twiddles(float* out) {
    constexpr double pi2 = 6.283185307179586476925286766559, sgn = INV ? 1.0 : -1.0;
    for (u32 h = 0; h < 2; ++h)
      for (u32 e = 0; e < 256; ++e) {
        const double x = pi2 * (double)((e >> 4) * (e & 15u)) / (h ? 4096.0 : 256.0);
        out[(h * 256 + e) * 2] = (float)std::cos(x);
        out[(h * 256 + e) * 2 + 1] = (float)(sgn * std::sin(x));
      }
  }
  template <class A>
  static __device__ __forceinline__ void setup(const A&, uint8_t*, int) {}

  template <class A>
  static __device__ __forceinline__ void run(const A&, const State&, u32 sb, u32 tws, int t, u32,
                                             const Sync<T>&) {
    phases<false>(sb, tws, t, nullptr, nullptr);
  }
  // G: the transform read from and written to global memory (every access of
  // a half warp is a line), the tables complete after the wait.
  template <bool G>
  static __device__ __forceinline__ void phases(u32 sb, u32 tws, int t, const uint8_t* gin, uint8_t* gout) {
    const u32 x = xd(t);
    {
      float re[2][16], im[2][16];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const u32 b = sb + (yd(t, j) * 16 + x) * EI;
#pragma unroll
        for (int n = 0; n < 16; ++n) {
          float2 z;
          if constexpr (G && IN16_)
            z = sm100::unpack_half2(*reinterpret_cast<const u32*>(gin + (yd(t, j) * 16 + x) * 4 + n * 1024));
          else if constexpr (G) z = *reinterpret_cast<const float2*>(gin + (yd(t, j) * 16 + x) * 8 + n * 2048);
          else if constexpr (IN16_) z = sm100::unpack_half2(lds32(b + n * 256 * EI));
          else z = lds64f(b + n * 256 * EI);
          re[j][n] = z.x;
          im[j][n] = z.y;
        }
      }
      if constexpr (G) asm volatile("cp.async.wait_all;" ::: "memory");
      if constexpr (G || EI != EO) col_bar<128>(4);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const u32 y = yd(t, j), b = sb + (y * 16 + x) * 8;
        Dft<16, INV, float>::run(re[j], im[j]);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          if (k > 0) {
            const float2 f = cmulf(lds64f(tws + (k * 16 + y) * 8), lds64f(tws + (256 + k * 16 + x) * 8));
            cmulv(re[j][k], im[j][k], f.x, f.y);
          }
          tile::sts64(b + k * 256 * 8, make_float2(re[j][k], im[j][k]));
        }
      }
    }
    col_bar<128>(4);
    {
      float re[2][16], im[2][16];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const u32 b = sb + (yd(t, j) * 256 + x) * 8;
#pragma unroll
        for (int n = 0; n < 16; ++n) {
          const float2 z = lds64f(b + n * 128);
          re[j][n] = z.x;
          im[j][n] = z.y;
        }
      }
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const u32 b = sb + ex2_at(yd(t, j), 0, x);
        Dft<16, INV, float>::run(re[j], im[j]);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          if (k > 0) {
            const float2 f = lds64f(tws + (k * 16 + x) * 8);
            cmulv(re[j][k], im[j][k], f.x, f.y);
          }
          tile::sts64(b + k * 128, make_float2(re[j][k], im[j][k]));
        }
      }
    }
    col_bar<128>(4);
    {
      float re[2][16], im[2][16];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const u32 b = sb + ex2_at(x, yd(t, j), 0);
#pragma unroll
        for (int n = 0; n < 8; ++n) {
          const float4 z = lds128f(b ^ (n << 4));
          re[j][2 * n] = z.x;
          im[j][2 * n] = z.y;
          re[j][2 * n + 1] = z.z;
          im[j][2 * n + 1] = z.w;
        }
      }
      if constexpr (!G) col_bar<128>(4);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const u32 o = (yd(t, j) * 16 + x) * 8;
        Dft<16, INV, float>::run(re[j], im[j]);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const float2 z = make_float2(re[j][k], im[j][k]);
          if constexpr (G) *reinterpret_cast<float2*>(gout + o + k * 256 * 8) = z;
          else tile::sts64(sb + o + k * 256 * 8, z);
        }
      }
    }
  }
};

// 2048 points, plain form.
template <bool INV_>
struct Mma2048 {
  using u32 = uint32_t;
  static constexpr int L = 2048, KIND = kRR, TP = 16384, R = 8, C = 8, EI = 4, EO = 4;
  static constexpr bool POST = false, INV = INV_, BIG = true;
  static constexpr int T = 512, NW = 16, NG = 1, NBUF = 3, NFULL = 3, THREADS = T + 128, MINB = 1;
  static constexpr int BUF = TP * 4;
  using State = MmaFrags;
  static __host__ __device__ constexpr u32 bit(u32 x, int b) { return (x >> b) & 1u; }

  // n = 128 n1 + 8 n2 + n3; 128-byte rows of 32 points, rows 16 (n2 >> 2) + n1
  // within a transform; the output in natural order.
  static __host__ __device__ constexpr u32 in_at(u32 n1, u32 n2, u32 n3) {
    return ((n2 >> 2) * 16 + n1) * 128 + ((((n2 & 3u) << 1 | n3 >> 2) ^ (n1 & 7u)) << 4) + (n3 & 3u) * 4;
  }
  static __host__ __device__ constexpr u32 ex_at(u32 k1, u32 n2, u32 n3) {
    return ((n2 >> 2) * 16 + k1) * 128 + ((((n2 & 3u) << 1 | n3 >> 2) ^ (bit(k1, 0) * 5u)) << 4) + (n3 & 3u) * 4;
  }
  static __host__ __device__ constexpr u32 out_at(u32 k1, u32 k2, u32 k3) {
    const u32 pos = k1 + 16 * k2 + 256 * k3, row = pos >> 5;
    return row * 128 + ((((pos >> 2) ^ row) & 7u) << 4) + (pos & 3u) * 4;
  }
  struct XY {
    u32 x, y;
  };
  // phase 1: (n2, n3); phase 2: (k1, n3)
  static __host__ __device__ constexpr XY p1(u32 g, u32 h, u32 w, u32 warp) {
    return {bit(g, 1) | bit(g, 0) << 1 | h << 2 | warp << 3, w | bit(g, 2) << 2};
  }
  static __host__ __device__ constexpr XY p2(u32 g, u32 h, u32 w, u32 warp) {
    return {bit(g, 0) | bit(g, 1) << 1 | warp << 2 | bit(g, 2) << 3, w | h << 2};
  }
  static constexpr u32 XM = 0x70u;
  static __host__ __device__ constexpr u32 load1_t(u32 lane, u32 warp) {
    const XY a = p1(lane >> 2, 0, 0, warp);
    return in_at(lane & 3u, a.x, a.y);
  }
  static __host__ __device__ constexpr u32 load1_r(u32 h, u32 i) {
    const XY a = p1(0, h, 0, 0);
    return in_at(4 * i, a.x, a.y);
  }
  static __host__ __device__ constexpr u32 store1_t(u32 lane, u32 warp) {
    const XY a = p1((lane & 3u) << 1, 0, 0, warp);
    return ex_at(lane >> 2, a.x, a.y);
  }
  static __host__ __device__ constexpr u32 store1_r(u32 mt, u32 p, u32 h) {
    const XY a = p1(p, h, 0, 0);
    return ex_at(8 * mt, a.x, a.y);
  }
  static __host__ __device__ constexpr u32 load2_t(u32 lane, u32 warp) {
    const XY a = p2(lane >> 2, 0, 0, warp);
    return ex_at(a.x, lane & 3u, a.y);
  }
  static __host__ __device__ constexpr u32 load2_r(u32 h, u32 i) {
    const XY a = p2(0, h, 0, 0);
    return ex_at(a.x, 4 * i, a.y);
  }
  static __host__ __device__ constexpr u32 store2_t(u32 lane, u32 warp) {
    const XY a = p2((lane & 3u) << 1, 0, 0, warp);
    return out_at(a.x, lane >> 2, 0);
  }
  static __host__ __device__ constexpr u32 store2_r(u32 mt, u32 k3) { return out_at(0, 8 * mt, k3); }

  // Phase 1: chain starts (pairs over vector bit 0) at ((warp * 4 + mt * 2 + h)
  // * 32 + lane), steps W_2048^k1 at 256 + k1; phase 2: W_128^(k2 n3) / 8,
  // doubled, at 272 + ((n3 - 1) * 2 + mt) * 8 + g.
  static constexpr int TWB = (256 + 16 + 112) * 16, TABB = TWB;
  static constexpr int OFF_TW = NBUF * BUF, OFF_BAR = OFF_TW + TWB;
  static constexpr int SMEM_BYTES = OFF_BAR + 128 + 1024;
  static void fill_twiddles(float* out) {
    constexpr double pi2 = 6.283185307179586476925286766559, sgn = INV ? 1.0 : -1.0;
    auto set = [&](u32 at, u32 p, u32 e, u32 mod, double scale) {
      const double x = pi2 * (double)(e % mod) / (double)mod;
      out[at * 4 + p] = (float)(scale * std::cos(x));
      out[at * 4 + 2 + p] = (float)(scale * sgn * std::sin(x));
    };
    for (u32 p = 0; p < 2; ++p) {
      for (u32 warp = 0; warp < 2; ++warp)
        for (u32 mh = 0; mh < 4; ++mh)
          for (u32 lane = 0; lane < 32; ++lane) {
            const XY a = p1((lane & 3u) << 1 | p, mh & 1u, 0, warp);
            set((warp * 4 + mh) * 32 + lane, p, ((lane >> 2) + 8 * (mh >> 1)) * (8 * a.x + a.y), 2048, 1.0);
          }
      for (u32 k1 = 0; k1 < 16; ++k1) set(256 + k1, p, k1, 2048, 1.0);
      for (u32 n3 = 1; n3 < 8; ++n3)
        for (u32 mt = 0; mt < 2; ++mt)
          for (u32 g = 0; g < 8; ++g) set(272 + ((n3 - 1) * 2 + mt) * 8 + g, p, (g + 8 * mt) * n3, 128, 0.125);
    }
  }
  static void fill_fragments(uint32_t* out) { MmaPass<256, kRR, false, INV>::fill_fragments(out); }
  template <class A>
  static __device__ __forceinline__ void setup(const A&, uint8_t*, int) {}
  using M = MmaPass<256, kRR, false, INV>;

  template <class A>
  static __device__ __forceinline__ void run(const A&, const State& st, u32 sb, u32 tws, int t, u32,
                                             const Sync<T>&) {
    const u32 lane = t & 31, warp = (t >> 5) & 1u, g = lane >> 2;
    const int bar = 8 + (t >> 6);
    sb += (t >> 6) * 8192;
    u32 x[8][4];
    {
      const u32 lb = sb + load1_t(lane, warp), sp = sb + store1_t(lane, warp);
#pragma unroll
      for (int j = 0; j < 8; ++j) Mma4096<INV>::get(lb, load1_r(j >> 2, j & 3), x[j]);
      __syncwarp();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        P2 cr[2], ci[2];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
          const float4 f = lds128f(tws + ((warp * 4 + mt * 2 + h) * 32 + lane) * 16);
          cr[mt] = pack2(f.x, f.y);
          ci[mt] = pack2(f.z, f.w);
        }
        u32 o[2][2][4];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          P2 re[2], im[2];
          M::unit(st, x[4 * h][w], x[4 * h + 1][w], x[4 * h + 2][w], x[4 * h + 3][w], re, im);
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) {
            cmulv(re[mt], im[mt], cr[mt], ci[mt]);
            if (w < 3) {
              const float4 f = lds128f(tws + (256 + g + 8 * mt) * 16);
              cmulv(cr[mt], ci[mt], pack2(f.x, f.y), pack2(f.z, f.w));
            }
            M::to_words(re[mt], im[mt], o[mt][0][w], o[mt][1][w]);
          }
        }
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
          for (int p = 0; p < 2; ++p) M::put(sp, store1_r(mt, p, h), o[mt][p]);
      }
    }
    col_bar<64>(bar);
    {
      const u32 lb = sb + load2_t(lane, warp), sp = sb + store2_t(lane, warp);
#pragma unroll
      for (int j = 0; j < 8; ++j) Mma4096<INV>::get(lb, load2_r(j >> 2, j & 3), x[j]);
      col_bar<64>(bar);
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        P2 zr[8], zi[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int j = u & 4, w = u & 3;  // n3 = w + 4 h
          float d[4];
          mma16816<true>(d, st.a[mt][0], x[j][w], x[j + 1][w]);
          mma16816<false>(d, st.a[mt][1], x[j + 2][w], x[j + 3][w]);
          zr[u] = pack2(d[0], d[1]);
          zi[u] = pack2(d[2], d[3]);
          if (u == 0) {
            zr[0] = zr[0] * num<P2>(0.125f);
            zi[0] = zi[0] * num<P2>(0.125f);
          } else {
            const float4 f = lds128f(tws + (272 + ((u - 1) * 2 + mt) * 8 + g) * 16);
            cmulv(zr[u], zi[u], pack2(f.x, f.y), pack2(f.z, f.w));
          }
        }
        Dft<8, INV, P2>::run(zr, zi);
#pragma unroll
        for (int k3 = 0; k3 < 8; ++k3) {
          u32 w0, w1;
          M::to_words(zr[k3], zi[k3], w0, w1);
          const u32 d = store2_r(mt, k3);
          tile::sts64((sp ^ (d & XM)) + (d & ~XM), make_float2(__uint_as_float(w0), __uint_as_float(w1)));
        }
      }
    }
  }
};

}  // namespace reg
}  // namespace mcfft
