// FP64 DFTs in block fixed point.
//
// GB300's FP64 pipe adds or multiplies 2 numbers a cycle on each SM, its
// integer pipes add some 57 64-bit integers (measured; a 32 x 32 -> 64
// multiply-add: 15).  A codelet therefore runs on 64-bit integers: the R
// complex doubles one thread holds are scaled by the exponent of the largest,
//   X = x 2^(B - 1023 - e),  |X| < 2^B,
// transformed and twiddled with integer additions and multiplications, and
// converted back, each output rounded once to a double.  B leaves room for the
// growth of the transform (|.| < 2^61 throughout), so the integers carry 56 to
// 60 bits of the block's largest value: their rounding stays below that of one
// double operation, where the FP64 codelet rounds at every addition.  The
// exponent is the thread's own, so nothing is shared between threads.
//
// Measured on a 32-band block of si64 (96^3; FP64 pipe before, this after):
// x-pass 2480 -> 596 us, inverse y/z 717 -> 274, forward y/z 740 -> 297 (of which
// not running on integers, but the folded x-pass and CTA sizes of
// local_kernels.cuh, give some 370 us).  The x-pass issues on 42% of cycles with
// its integer pipes 50% and the converting FP64 pipe 39% busy: what is left is
// latency, at 128 registers a thread and 16 warps an SM.
//
// A block with a NaN or an infinity gives NaN (any DFT of it is non-finite in FP64
// too), and so does one that holds 2^1018 or more: keeping outputs between that and
// the largest double took a branch a block, 5% of every FP64 pass.  Numbers are kept
// to a multiple of 2^-1022.
#pragma once

#include "codelets.cuh"
#include "qgb_common.cuh"

namespace qgb {

__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
  long long r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}

// A fixed-point factor |c| <= 1 as h 2^32 + l in units of 2^-62, both halves signed.
struct FxConst {
  int l, h;
};
__host__ __device__ constexpr FxConst fx_const(double c) {
  const long long v = static_cast<long long>(c * 4611686018427387904.0);
  const int l = static_cast<int>(static_cast<unsigned>(v & 0xFFFFFFFFll));
  // (the low half moves by one unit where it could not be negated, the high half is its own)
  return FxConst{l == -2147483647 - 1 ? -2147483647 : l, static_cast<int>((v - l) >> 32)};
}

// A 64-bit integer of a block, |v| < 2^61 where it is multiplied.  Fx(c) is a
// codelet's constant factor.
struct Fx {
  long long v;
  Fx() = default;
  __host__ __device__ explicit constexpr Fx(double c) : v(static_cast<long long>(c * 4611686018427387904.0)) {}
};
__device__ __forceinline__ Fx fx_raw(long long v) {
  Fx r;
  r.v = v;
  return r;
}
__device__ __forceinline__ Fx operator+(Fx a, Fx b) { return fx_raw(a.v + b.v); }
__device__ __forceinline__ Fx operator-(Fx a, Fx b) { return fx_raw(a.v - b.v); }
__device__ __forceinline__ Fx operator-(Fx a) { return fx_raw(-a.v); }

// x = h 2^32 + l with both halves signed.
__device__ __forceinline__ void fx_split(Fx x, int& h, int& l) {
  l = static_cast<int>(x.v);
  h = static_cast<int>(x.v >> 32) - (l >> 31);
}
// round(x c): the products of the low halves are below the rounding.
__device__ __forceinline__ Fx fx_mul(Fx x, FxConst c) {
  int h, l;
  fx_split(x, h, l);
  const long long acc = mad_wide(l, c.h, mad_wide(h, c.l, 1ll << 29));
  return fx_raw(mad_wide(h << 2, c.h, acc >> 30));
}
// Codelet constant times value; the constant folds at compile time.
__device__ __forceinline__ Fx operator*(Fx c, Fx x) {
  if (c.v == (1ll << 61)) return fx_raw(x.v >> 1);
  const int l = static_cast<int>(c.v);
  return fx_mul(x, FxConst{l, static_cast<int>((c.v - l) >> 32)});
}

// (a + i b) (wx + i s wy), w from the packed twiddle table (s = -1: conjugated).
template <int S>
__device__ __forceinline__ void fx_twiddle(Fx& a, Fx& b, FxConst wx, FxConst wy) {
  int ah, al, bh, bl;
  fx_split(a, ah, al);
  fx_split(b, bh, bl);
  if (S < 0) wy = FxConst{-wy.l, -wy.h};
  const FxConst nwy{-wy.l, -wy.h};
  long long re = mad_wide(ah, wx.l, 1ll << 29), im = mad_wide(ah, wy.l, 1ll << 29);
  re = mad_wide(al, wx.h, re);
  im = mad_wide(al, wy.h, im);
  re = mad_wide(bh, nwy.l, re);
  im = mad_wide(bh, wx.l, im);
  re = mad_wide(bl, nwy.h, re);
  im = mad_wide(bl, wx.h, im);
  ah <<= 2;
  bh <<= 2;
  a.v = mad_wide(bh, nwy.h, mad_wide(ah, wx.h, re >> 30));
  b.v = mad_wide(bh, wx.h, mad_wide(ah, wy.h, im >> 30));
}

// Bits of a block's largest input: R sqrt(2) 2^B <= 2^61.
template <int R> constexpr int fx_bits() {
  int g = 0;
  while ((1 << g) * (1 << g) < 2 * R * R) ++g;  // 2^g >= R sqrt(2)
  return 61 - g;
}

// Largest exponent field of a block of doubles, at least `least`.
template <int R>
__device__ __forceinline__ int fx_exponent(const double (&re)[R], const double (&im)[R], int least) {
  unsigned m = static_cast<unsigned>(least) << 20;
#pragma unroll
  for (int j = 0; j < R; ++j) {
    m = max(m, static_cast<unsigned>(__double2hiint(re[j])) & 0x7FFFFFFFu);
    m = max(m, static_cast<unsigned>(__double2hiint(im[j])) & 0x7FFFFFFFu);
  }
  return static_cast<int>(m >> 20);
}

// x 2^(bits - 1 - (e - 1023)) truncated toward zero, for an exponent field <= e.
template <int BITS>
__device__ __forceinline__ long long fx_from_double(double x, int e) {
  const unsigned hi = static_cast<unsigned>(__double2hiint(x));
  const int s = e - static_cast<int>((hi >> 20) & 0x7FFu);
  unsigned long long m = (static_cast<unsigned long long>((hi & 0xFFFFFu) | 0x100000u) << 32) |
                         static_cast<unsigned>(__double2loint(x));
  m <<= BITS - 53;
  asm("shr.u64 %0, %1, %2;" : "=l"(m) : "l"(m), "r"(s));  // clamped: 0 from 64 on
  const long long sg = static_cast<int>(hi) >> 31;
  return (static_cast<long long>(m) ^ sg) - sg;
}

// v 2^k as a double, rounded once (kLow <= k <= kHigh, see Block),
// or NaN where `nan` holds its exponent bits.
__device__ __forceinline__ double fx_to_double(long long v, int k, int nan) {
  const double d = __ll2double_rn(v);
  const int hi = __double2hiint(d);
  return __hiloint2double((hi == 0 ? 0 : hi + (k << 20)) | nan, __double2loint(d));
}

// How a codelet's R complex values of type T are computed: float as they are,
// double in block fixed point.
template <typename T, int R> struct Block;

template <int R> struct Block<float, R> {
  float re[R], im[R];
  __device__ __forceinline__ void load(const float (&x)[R], const float (&y)[R]) {
#pragma unroll
    for (int j = 0; j < R; ++j) {
      re[j] = x[j];
      im[j] = y[j];
    }
  }
  template <int S> __device__ __forceinline__ void run() { Codelet<R, S>::run(re, im); }
  // Element j times w (S < 0: its conjugate).
  template <int S> __device__ __forceinline__ void twiddle(int j, float2 w) {
    const float wy = S > 0 ? w.y : -w.y;
    const float x = re[j] * w.x - im[j] * wy;
    im[j] = re[j] * wy + im[j] * w.x;
    re[j] = x;
  }
  __device__ __forceinline__ void scale(const float (&v)[R]) {
#pragma unroll
    for (int j = 0; j < R; ++j) {
      re[j] *= v[j];
      im[j] *= v[j];
    }
  }
  // put(j, value()) for every element; value() is what converts it.
  template <typename F> __device__ __forceinline__ void store(F put) const {
#pragma unroll
    for (int j = 0; j < R; ++j) put(j, [&] { return make_float2(re[j], im[j]); });
  }
};

template <int R> struct Block<double, R> {
  static constexpr int B = fx_bits<R>();
  static constexpr int kLow = -1022, kHigh = 962;  // v 2^k of 1 <= |v| < 2^61 is a normal number
  Fx re[R], im[R];
  int k;     // a value is v 2^k
  bool bad;  // a NaN or an infinity among the inputs, or outputs that could overflow
  __device__ __forceinline__ void load(const double (&x)[R], const double (&y)[R]) {
    const int e = fx_exponent<R>(x, y, B);  // k >= kLow
    k = e - 1023 - (B - 1);
    bad = k > kHigh;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      re[j] = fx_raw(fx_from_double<B>(x[j], e));
      im[j] = fx_raw(fx_from_double<B>(y[j], e));
    }
  }
  template <int S> __device__ __forceinline__ void run() { Codelet<R, S>::run(re, im); }
  template <int S> __device__ __forceinline__ void twiddle(int j, double2 w) {
    fx_twiddle<S>(re[j], im[j], FxConst{__double2loint(w.x), __double2hiint(w.x)},
                  FxConst{__double2loint(w.y), __double2hiint(w.y)});
  }
  // Times real factors, and back below 2^B for another transform: the factors
  // are fixed-point numbers scaled by their largest and by the bits the values
  // have grown.
  __device__ __forceinline__ void scale(const double (&v)[R]) {
    unsigned mv = 64u << 20, mx = 0;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      mv = max(mv, static_cast<unsigned>(__double2hiint(v[j])) & 0x7FFFFFFFu);
      const int a = static_cast<int>(re[j].v >> 32), b = static_cast<int>(im[j].v >> 32);
      mx |= static_cast<unsigned>(a ^ (a >> 31)) | static_cast<unsigned>(b ^ (b >> 31));
    }
    const int e = static_cast<int>(mv >> 20);
    const int grown = max(0, 64 - __clz(static_cast<int>(mx)) - B);  // |value| < 2^(B + grown)
    k += e - 1022 + grown;
    bad |= e == 0x7FF || k > kHigh;
    const int low = max(kLow - k, 0);  // products near the smallest double: as multiples of 2^kLow
    k += low;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const long long f = fx_from_double<62>(v[j], e + grown + low);  // |v| 2^(62 - grown), below 2^62
      const int l = static_cast<int>(f);
      const FxConst c{l, static_cast<int>((f - l) >> 32)};
      re[j] = fx_mul(re[j], c);
      im[j] = fx_mul(im[j], c);
    }
  }
  template <typename F> __device__ __forceinline__ void store(F put) const {
    const int nan = bad ? 0x7FF80000 : 0;
#pragma unroll
    for (int j = 0; j < R; ++j)
      put(j, [&] { return make_double2(fx_to_double(re[j].v, k, nan), fx_to_double(im[j].v, k, nan)); });
  }
};

// Twiddle tables in shared memory: doubles are kept as the fixed-point halves.
__device__ __forceinline__ float2 pack_twiddle(float2 w) { return w; }
__device__ __forceinline__ double2 pack_twiddle(double2 w) {
  const FxConst x = fx_const(w.x), y = fx_const(w.y);
  return make_double2(__hiloint2double(x.h, x.l), __hiloint2double(y.h, y.l));
}

}  // namespace qgb
