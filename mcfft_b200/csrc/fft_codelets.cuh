// fft_codelets.cuh -- register-resident DFTs of 8 and 16 points in FP32, the
// radix-4 step they share and the first step of a 32-point one: the arithmetic
// of the register pass kernels (fft_reg.cuh).
//
// One source serves two number types: `float` (one transform per thread at a
// time) and P2, a pair of FP32 lanes in one 64-bit register on which the
// sm_100 packed instructions (add / mul / fma .f32x2) work: two transforms
// at once, half the issue slots of scalar code for the same FP32 pipe time
// (measured on a B200: one warp-wide f32x2 instruction takes two cycles of a
// sub-partition, a scalar one takes one).
//
// Every codelet computes X[k] = sum_n x[n] exp(SGN 2 pi i n k / R), SGN = +1
// for INV, -1 otherwise, input and output in natural order.  The direction
// is a template argument, so a product with +-i is a choice of add and
// subtract and the internal twiddles are immediates.
#pragma once
#include <cstdint>

#include "fft_tile.cuh"

namespace mcfft {
namespace reg {

struct P2 {
  uint64_t v;
};
__device__ __forceinline__ P2 pack2(float lo, float hi) { return P2{f2p(lo, hi)}; }
__device__ __forceinline__ P2 operator+(P2 a, P2 b) { return P2{add2(a.v, b.v)}; }
__device__ __forceinline__ P2 operator-(P2 a, P2 b) { return P2{sub2(a.v, b.v)}; }
__device__ __forceinline__ P2 operator*(P2 a, P2 b) { return P2{mul2(a.v, b.v)}; }
__device__ __forceinline__ P2 fmad(P2 a, P2 b, P2 c) { return P2{fma2(a.v, b.v, c.v)}; }
__device__ __forceinline__ float fmad(float a, float b, float c) { return fmaf(a, b, c); }
template <class T>
__device__ __forceinline__ T num(float c);
template <>
__device__ __forceinline__ float num<float>(float c) {
  return c;
}
template <>
__device__ __forceinline__ P2 num<P2>(float c) {
  return pack2(c, c);
}

// (re, im) *= c + i s
template <class T>
__device__ __forceinline__ void cmulc(T& re, T& im, float c, float s) {
  const T r = re * num<T>(c), i = im * num<T>(c);
  const T nr = fmad(im, num<T>(-s), r), ni = fmad(re, num<T>(s), i);
  re = nr;
  im = ni;
}
// (re, im) *= c + i s for variable c, s
template <class T>
__device__ __forceinline__ void cmulv(T& re, T& im, T c, T s) {
  const T a = re * c - im * s;
  im = fmad(re, s, im * c);
  re = a;
}
__device__ __forceinline__ void cmulv(float& re, float& im, float c, float s) {
  const float a = fmaf(re, c, -(im * s));
  im = fmaf(re, s, im * c);
  re = a;
}
// Radix-4 on (a, b, c, d) in place: outputs X[0..3] in a, b, c, d.  ROTC:
// c enters multiplied by SGN i (the middle twiddle of the 8- and 16-point
// DFTs), which only exchanges its parts and their signs.
template <bool INV, bool ROTC = false, class T>
__device__ __forceinline__ void dft4(T& ar, T& ai, T& br, T& bi, T& cr, T& ci, T& dr, T& di) {
  const bool neg = ROTC && INV, pos = ROTC && !INV;
  const T s0r = neg ? ar - ci : pos ? ar + ci : ar + cr;
  const T s0i = neg ? ai + cr : pos ? ai - cr : ai + ci;
  const T d0r = neg ? ar + ci : pos ? ar - ci : ar - cr;
  const T d0i = neg ? ai - cr : pos ? ai + cr : ai - ci;
  const T s1r = br + dr, s1i = bi + di, d1r = br - dr, d1i = bi - di;
  ar = s0r + s1r;
  ai = s0i + s1i;
  cr = s0r - s1r;
  ci = s0i - s1i;
  if (INV) {  // X1 = d0 + i d1, X3 = d0 - i d1
    br = d0r - d1i;
    bi = d0i + d1r;
    dr = d0r + d1i;
    di = d0i - d1r;
  } else {
    br = d0r + d1i;
    bi = d0i - d1r;
    dr = d0r - d1i;
    di = d0i + d1r;
  }
}

template <int R, bool INV, class T>
struct Dft;

template <bool INV, class T>
struct Dft<8, INV, T> {
  // n = 4 m + j: radix 2 over m, twiddle W8^(j q), radix 4 over j
  static __device__ __forceinline__ void run(T (&re)[8], T (&im)[8]) {
    constexpr float h = 0.70710678118654752440f;
    constexpr float s = INV ? 1.f : -1.f;
    T er[4], ei[4], orr[4], oi[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      er[j] = re[j] + re[j + 4];
      ei[j] = im[j] + im[j + 4];
      orr[j] = re[j] - re[j + 4];
      oi[j] = im[j] - im[j + 4];
    }
    {  // W8 = h (1 + s i): (re, im) -> h (re - s im, im + s re)
      const T a = INV ? orr[1] - oi[1] : orr[1] + oi[1], b = INV ? oi[1] + orr[1] : oi[1] - orr[1];
      orr[1] = a * num<T>(h);
      oi[1] = b * num<T>(h);
    }
    {  // W8^3 = h (-1 + s i): (re, im) -> h (-re - s im, -im + s re)
      const T a = INV ? orr[3] + oi[3] : orr[3] - oi[3], b = INV ? orr[3] - oi[3] : orr[3] + oi[3];
      orr[3] = a * num<T>(-h);
      oi[3] = b * num<T>(s * h);
    }
    dft4<INV>(er[0], ei[0], er[1], ei[1], er[2], ei[2], er[3], ei[3]);
    dft4<INV, true>(orr[0], oi[0], orr[1], oi[1], orr[2], oi[2], orr[3], oi[3]);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      re[2 * k] = er[k];
      im[2 * k] = ei[k];
      re[2 * k + 1] = orr[k];
      im[2 * k + 1] = oi[k];
    }
  }
};

template <bool INV, class T>
struct Dft<16, INV, T> {
  // n = 4 m + j: radix 4 over m for each j, twiddle W16^(j q), radix 4 over j
  static __device__ __forceinline__ void run(T (&re)[16], T (&im)[16]) {
    constexpr float s = INV ? 1.f : -1.f;
    constexpr float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f, h = 0.70710678118654752440f;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      dft4<INV>(re[j], im[j], re[j + 4], im[j + 4], re[j + 8], im[j + 8], re[j + 12], im[j + 12]);
    // re[j + 4 q] = Y_j[q]; times W16^(j q)
    cmulc(re[5], im[5], c1, s * s1);       // j 1 q 1
    cmulc(re[13], im[13], s1, s * c1);     // j 1 q 3
    cmulc(re[7], im[7], s1, s * c1);       // j 3 q 1
    cmulc(re[15], im[15], -c1, -s * s1);   // j 3 q 3: W16^9
    auto w2 = [](T& a, T& b) {  // W16^2 = h (1 + s i)
      const T x = INV ? a - b : a + b, y = INV ? b + a : b - a;
      a = x * num<T>(h);
      b = y * num<T>(h);
    };
    auto w6 = [](T& a, T& b) {  // W16^6 = h (-1 + s i)
      const T x = INV ? a + b : a - b, y = INV ? a - b : a + b;
      a = x * num<T>(-h);
      b = y * num<T>((INV ? 1.f : -1.f) * h);
    };
    w2(re[9], im[9]);    // j 1 q 2
    w2(re[6], im[6]);    // j 2 q 1
    w6(re[14], im[14]);  // j 2 q 3
    w6(re[11], im[11]);  // j 3 q 2
    // j 2 q 2: W16^4 = s i, taken by the radix 4
    dft4<INV>(re[0], im[0], re[1], im[1], re[2], im[2], re[3], im[3]);
    dft4<INV>(re[4], im[4], re[5], im[5], re[6], im[6], re[7], im[7]);
    dft4<INV, true>(re[8], im[8], re[9], im[9], re[10], im[10], re[11], im[11]);
    dft4<INV>(re[12], im[12], re[13], im[13], re[14], im[14], re[15], im[15]);
    // X[q + 4 p] sits at 4 q + p: transpose the 4 x 4 (register renaming)
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int p = q + 1; p < 4; ++p) {
        const T a = re[4 * q + p], b = im[4 * q + p];
        re[4 * q + p] = re[4 * p + q];
        im[4 * q + p] = im[4 * p + q];
        re[4 * p + q] = a;
        im[4 * p + q] = b;
      }
  }
};

// cos(pi n / 16), n = 0..8, and the cosine and sine for n = 0..16
__device__ __forceinline__ constexpr float cos16q(int n) {
  return n == 0   ? 1.f
         : n == 1 ? 0.98078528040323044913f
         : n == 2 ? 0.92387953251128675613f
         : n == 3 ? 0.83146961230254523708f
         : n == 4 ? 0.70710678118654752440f
         : n == 5 ? 0.55557023301960222474f
         : n == 6 ? 0.38268343236508977173f
         : n == 7 ? 0.19509032201612826785f
                  : 0.f;
}
__device__ __forceinline__ constexpr float cos16(int n) { return n <= 8 ? cos16q(n) : -cos16q(16 - n); }
__device__ __forceinline__ constexpr float sin16(int n) { return n <= 8 ? cos16q(8 - n) : cos16q(n - 8); }

// First step of a 32-point DFT (decimation in frequency): even outputs are
// the 16-point DFT of x[n] + x[n + 16], odd ones that of (x[n] - x[n + 16])
// W32^n.  (er, ei) and (odr, odi) receive the two inputs.
template <bool INV>
__device__ __forceinline__ void split32(float x0r, float x0i, float x1r, float x1i, int n, float& er,
                                        float& ei, float& odr, float& odi) {
  er = x0r + x1r;
  ei = x0i + x1i;
  if (n == 8) {  // W32^8 = SGN i
    odr = INV ? x1i - x0i : x0i - x1i;
    odi = INV ? x0r - x1r : x1r - x0r;
    return;
  }
  odr = x0r - x1r;
  odi = x0i - x1i;
  if (n != 0) cmulc(odr, odi, cos16(n), (INV ? 1.f : -1.f) * sin16(n));
}

}  // namespace reg
}  // namespace mcfft
