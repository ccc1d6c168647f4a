// Two FP32 columns in one register pair, for the packed add, multiply and
// multiply-add of sm_100 and later.
//
// They do two FP32 operations an issue slot (measured 120 to 133 results a clock
// and SM, as FADD and FFMA reach with twice the instructions), so codelets on
// pairs of columns halve the arithmetic's share of the issue slots and the
// addressing around it.  Each half is rounded like the scalar operation.
//
// Lazy<L> is the codelets' type T: a pair (L = pair_t) with a pending sign and a
// pending constant factor, both known at compile time once a codelet is unrolled,
// which fold into the next addition (subtraction, multiply-add) as the compiler
// folds them for float.  Lazy<float> does the same operations on one column: the
// batched x-pass, which takes y-rows, gives the same bits.
#pragma once

#include <cstdint>

#include "block_fixed.cuh"
#include "codelets.cuh"

namespace qgb {

using pair_t = unsigned long long;  // (column c, column c + 32)

__device__ __forceinline__ pair_t pair_of(float lo, float hi) {
  pair_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 pair_split(pair_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ pair_t lane_add(pair_t a, pair_t b) {
  pair_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ pair_t lane_mul(pair_t a, pair_t b) {
  pair_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ pair_t lane_fma(pair_t a, pair_t b, pair_t c) {
  pair_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ pair_t lane_neg(pair_t a) { return a ^ 0x8000000080000000ull; }
__device__ __forceinline__ float lane_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float lane_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float lane_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float lane_neg(float a) { return -a; }
template <typename L> __device__ __forceinline__ L lane_const(float c) {
  if constexpr (sizeof(L) == 8)
    return pair_of(c, c);
  else
    return c;
}

template <typename L> struct Lazy {
  L v = 0;
  float c = 1.0f;        // the value is +-c v; a literal is its c alone
  bool neg = false, scaled = false;
  Lazy() = default;
  __device__ __forceinline__ explicit Lazy(double x) : c(static_cast<float>(x)) {}
  __device__ __forceinline__ static Lazy of(L p) {
    Lazy r;
    r.v = p;
    return r;
  }
  __device__ __forceinline__ L value() const {
    if (scaled) return lane_mul(v, lane_const<L>(neg ? -c : c));
    return neg ? lane_mul(v, lane_const<L>(-1.0f)) : v;
  }
};

template <typename L> __device__ __forceinline__ Lazy<L> operator-(Lazy<L> a) {
  a.neg = !a.neg;
  return a;
}

// Literal times pair: left pending, or a product of its own on a pending one.
template <typename L> __device__ __forceinline__ Lazy<L> operator*(const Lazy<L>& l, const Lazy<L>& a) {
  Lazy<L> r;
  r.v = a.scaled ? lane_mul(a.v, lane_const<L>(a.c)) : a.v;
  r.neg = a.neg;
  r.c = l.c;
  r.scaled = true;
  return r;
}

template <typename L> __device__ __forceinline__ Lazy<L> operator+(const Lazy<L>& a, const Lazy<L>& b) {
  Lazy<L> r;
  if (b.scaled) {
    // b's factor takes the sign relative to a's base.
    L base = a.v;
    bool base_neg = a.neg;
    if (a.scaled) {
      base = lane_mul(a.v, lane_const<L>(a.neg ? -a.c : a.c));
      base_neg = false;
    }
    r.v = lane_fma(b.v, lane_const<L>(b.neg != base_neg ? -b.c : b.c), base);
    r.neg = base_neg;
  } else if (a.scaled) {
    r.v = lane_fma(a.v, lane_const<L>(a.neg != b.neg ? -a.c : a.c), b.v);
    r.neg = b.neg;
  } else if (a.neg == b.neg) {
    r.v = lane_add(a.v, b.v);
    r.neg = a.neg;
  } else if (b.neg) {
    r.v = lane_fma(b.v, lane_const<L>(-1.0f), a.v);
  } else {
    r.v = lane_fma(a.v, lane_const<L>(-1.0f), b.v);
  }
  return r;
}
template <typename L> __device__ __forceinline__ Lazy<L> operator-(const Lazy<L>& a, const Lazy<L>& b) { return a + (-b); }
using F2 = Lazy<pair_t>;

// A complex pair in shared memory: 16 B, (re, im) of both columns.
using cpair_t = ulonglong2;

// The codelet block of either; see Block<float, R>.  The twiddles w.x, w.y are of
// the lanes' type (doubled for pairs).
template <typename L, int R> struct LazyBlock {
  Lazy<L> re[R], im[R];
  template <int S> __device__ __forceinline__ void run() { Codelet<R, S>::run(re, im); }
  // Element j times (wx, wy) (S < 0: its conjugate).
  template <int S> __device__ __forceinline__ void twiddle(int j, L wx, L wy) {
    const L x = re[j].value(), y = im[j].value();
    const L wp = S > 0 ? wy : lane_neg(wy), wn = S > 0 ? lane_neg(wy) : wy;
    re[j] = Lazy<L>::of(lane_fma(y, wn, lane_mul(x, wx)));
    im[j] = Lazy<L>::of(lane_fma(x, wp, lane_mul(y, wx)));
  }
  __device__ __forceinline__ void scale(int j, L f) {
    re[j] = Lazy<L>::of(lane_mul(re[j].value(), f));
    im[j] = Lazy<L>::of(lane_mul(im[j].value(), f));
  }
};
template <int R> using PairBlock = LazyBlock<pair_t, R>;

// The x-pass's block on one column: Block<T, R>, in FP32 with the pairs' operations.
template <typename T, int R> struct XBlock : Block<T, R> {};
template <int R> struct XBlock<float, R> {
  LazyBlock<float, R> x;
  __device__ __forceinline__ void load(const float (&re)[R], const float (&im)[R]) {
#pragma unroll
    for (int j = 0; j < R; ++j) {
      x.re[j] = Lazy<float>::of(re[j]);
      x.im[j] = Lazy<float>::of(im[j]);
    }
  }
  template <int S> __device__ __forceinline__ void run() { x.template run<S>(); }
  template <int S> __device__ __forceinline__ void twiddle(int j, float2 w) { x.template twiddle<S>(j, w.x, w.y); }
  __device__ __forceinline__ void scale(const float (&v)[R]) {
#pragma unroll
    for (int j = 0; j < R; ++j) x.scale(j, v[j]);
  }
  template <typename F> __device__ __forceinline__ void store(F put) const {
#pragma unroll
    for (int j = 0; j < R; ++j) put(j, [&] { return make_float2(x.re[j].value(), x.im[j].value()); });
  }
};

}  // namespace qgb
