// Exact quotients and square roots of pairs of floats (packed FP32 instructions of sm_100).
//
// The float form has to give the bits of IEEE division and square root.  These build them from
// fused multiply-adds after P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor" (IBM J. Res. Dev. 34, 1990): with y the correctly rounded reciprocal of
// b and q within one ulp of a / b, q + (a - b q) y rounds to the correctly rounded quotient.  A
// reciprocal is shared by all the quotients that have it, there is no branch, and both halves of
// the packed instructions work.  Range of quot(a, b, y): 2^-100 <= |b| <= 2^100, |a| >= 2^-100 (below
// about 2^-102 the residual a - b q is not exact any more) or a = 0, and quotients in the normal range;
// a caller sees to it.  Dividends that may be as small as they like take quot(a, Divisor).
#pragma once
#include <cuda_runtime.h>

#include "tgv_pixel_fast.cuh"

namespace vfs {
namespace exact {

namespace x2 = fast::x2;

__device__ __forceinline__ x2::f2 neg(x2::f2 v) { return v ^ 0x8000000080000000ull; }
// 1 / b from an approximation within one ulp
__device__ __forceinline__ x2::f2 recip(x2::f2 b, x2::f2 y0) {
  return x2::fma(x2::fma(neg(b), y0, x2::pk(1.f, 1.f)), y0, y0);
}
__device__ __forceinline__ x2::f2 recip(x2::f2 b) {
  const float2 v = x2::upk(b);
  return recip(b, x2::pk(fast::rcp(v.x), fast::rcp(v.y)));
}
// a / b, y = 1 / b
__device__ __forceinline__ x2::f2 quot(x2::f2 a, x2::f2 b, x2::f2 y) {
  const x2::f2 q = x2::mul(a, y);
  return x2::fma(x2::fma(neg(b), q, a), y, q);
}
// A divisor 2^-64 <= |b| <= 2^64 for dividends of at most 2^64, down to the smallest.  The residual is taken
// 2^60 times as large, where it is exact, and the last step brings it back: the same bits for two products a
// divisor and one a quotient more.  A quotient below the normal range is rounded once, on its own grid, and
// rightly so but for one case: halfway between two subnormals, which takes an integer b other than a power
// of two, it may go either way.  (With S the 24-bit significand of b, a quotient that is not halfway is at
// least 1 / S of half a step away from it, and the error of r y is below S 2^-48 of that.)  A zero divided by a
// positive b keeps its sign; divided by a negative one it may not.
// The float form's norms and Iu divide this way, since its disparities shrink through all magnitudes where they
// spread into a part of the images that does not move: 13 packed instructions more a pair of rows (848 x 800:
// 6.12 -> 6.31 us per iteration, the solve 2.17 -> 2.21 ms).  Looking for small dividends, with the plain division
// behind a branch, took more (2.50 ms): the branches keep the pairs' chains from being scheduled side by side.
struct Divisor {
  x2::f2 y, bs, ys;  // 1 / b, 2^60 b, -2^-60 / b
  Divisor() = default;
  __device__ __forceinline__ Divisor(x2::f2 b, x2::f2 y_)
      : y(y_), bs(x2::mul(b, x2::pk(0x1p60f, 0x1p60f))), ys(x2::mul(y_, x2::pk(-0x1p-60f, -0x1p-60f))) {}
  // both halves divided by b's low / high one
  __device__ __forceinline__ Divisor low() const { return of(x2::upk(y).x, x2::upk(bs).x, x2::upk(ys).x); }
  __device__ __forceinline__ Divisor high() const { return of(x2::upk(y).y, x2::upk(bs).y, x2::upk(ys).y); }
  static __device__ __forceinline__ Divisor of(float y, float bs, float ys) {
    Divisor d;
    d.y = x2::pk(y, y);
    d.bs = x2::pk(bs, bs);
    d.ys = x2::pk(ys, ys);
    return d;
  }
};
__device__ __forceinline__ x2::f2 quot(x2::f2 a, const Divisor& d) {
  const x2::f2 q = x2::mul(a, d.y);
  return x2::fma(x2::fma(d.bs, q, x2::mul(a, x2::pk(-0x1p60f, -0x1p60f))), d.ys, q);
}
// s = sqrt(m) and 1 / s for 1 <= m < infinity (a NaN stays)
__device__ __forceinline__ void root(x2::f2 m, x2::f2& s, x2::f2& y) {
  using namespace x2;
  const float2 v = upk(m);
  const f2 y0 = pk(fast::rsqrt(v.x), fast::rsqrt(v.y));
  const f2 g = mul(m, y0), h = mul(y0, pk(0.5f, 0.5f));
  const f2 r = fma(neg(h), g, pk(0.5f, 0.5f));
  const f2 g1 = fma(g, r, g), h1 = fma(h, r, h);
  s = fma(fma(neg(g1), g1, m), h1, g1);
  y = recip(s);
}

}  // namespace exact
}  // namespace vfs
