// Two FP32 columns in one register pair, for the packed add, multiply and
// multiply-add of sm_100 and later.
//
// They do two FP32 operations an issue slot (measured 120 to 133 results a clock
// and SM, as FADD and FFMA reach with twice the instructions), so codelets on
// pairs of columns halve the arithmetic's share of the issue slots and the
// addressing around it.  Each half is rounded like the scalar operation.
//
// F2 is the codelets' type T: a pair with a pending sign and a pending constant
// factor, both known at compile time once a codelet is unrolled, which fold into
// the next addition (subtraction, multiply-add) as the compiler folds them for
// float.
#pragma once

#include <cstdint>

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
__device__ __forceinline__ pair_t pair_add(pair_t a, pair_t b) {
  pair_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ pair_t pair_mul(pair_t a, pair_t b) {
  pair_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ pair_t pair_fma(pair_t a, pair_t b, pair_t c) {
  pair_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ pair_t pair_const(float c) { return pair_of(c, c); }

struct F2 {
  pair_t v = 0;
  float c = 1.0f;        // the value is +-c v; c alone for a literal
  bool neg = false, scaled = false, literal = false;
  F2() = default;
  __device__ __forceinline__ explicit F2(double x) : c(static_cast<float>(x)), literal(true) {}
  __device__ __forceinline__ static F2 of(pair_t p) {
    F2 r;
    r.v = p;
    return r;
  }
  __device__ __forceinline__ pair_t value() const {
    if (scaled) return pair_mul(v, pair_const(neg ? -c : c));
    return neg ? pair_mul(v, pair_const(-1.0f)) : v;
  }
};

__device__ __forceinline__ F2 operator-(F2 a) {
  a.neg = !a.neg;
  return a;
}

// Literal times pair: left pending, or a product of its own on a pending one.
__device__ __forceinline__ F2 operator*(const F2& l, const F2& a) {
  F2 r;
  r.v = a.scaled ? pair_mul(a.v, pair_const(a.c)) : a.v;
  r.neg = a.neg;
  r.c = l.c;
  r.scaled = true;
  return r;
}

__device__ __forceinline__ F2 operator+(const F2& a, const F2& b) {
  F2 r;
  if (b.scaled) {
    // b's factor takes the sign relative to a's base.
    pair_t base = a.v;
    bool base_neg = a.neg;
    if (a.scaled) {
      base = pair_mul(a.v, pair_const(a.neg ? -a.c : a.c));
      base_neg = false;
    }
    r.v = pair_fma(b.v, pair_const(b.neg != base_neg ? -b.c : b.c), base);
    r.neg = base_neg;
  } else if (a.scaled) {
    r.v = pair_fma(a.v, pair_const(a.neg != b.neg ? -a.c : a.c), b.v);
    r.neg = b.neg;
  } else if (a.neg == b.neg) {
    r.v = pair_add(a.v, b.v);
    r.neg = a.neg;
  } else if (b.neg) {
    r.v = pair_fma(b.v, pair_const(-1.0f), a.v);
  } else {
    r.v = pair_fma(a.v, pair_const(-1.0f), b.v);
  }
  return r;
}
__device__ __forceinline__ F2 operator-(const F2& a, const F2& b) { return a + (-b); }

// A complex pair in shared memory: 16 B, (re, im) of both columns.
using cpair_t = ulonglong2;

// The codelet block of pairs; see Block<float, R>.
template <int R> struct PairBlock {
  F2 re[R], im[R];
  template <int S> __device__ __forceinline__ void run() { Codelet<R, S>::run(re, im); }
  // Element j times (w.x, w.y), both already doubled to pairs (S < 0: its conjugate).
  template <int S> __device__ __forceinline__ void twiddle(int j, cpair_t w) {
    const pair_t x = re[j].value(), y = im[j].value();
    const pair_t wy = S > 0 ? w.y : w.y ^ 0x8000000080000000ull, wn = S > 0 ? w.y ^ 0x8000000080000000ull : w.y;
    re[j] = F2::of(pair_fma(y, wn, pair_mul(x, w.x)));
    im[j] = F2::of(pair_fma(x, wy, pair_mul(y, w.x)));
  }
  __device__ __forceinline__ void scale(int j, pair_t f) {
    re[j] = F2::of(pair_mul(re[j].value(), f));
    im[j] = F2::of(pair_mul(im[j].value(), f));
  }
};

}  // namespace qgb
