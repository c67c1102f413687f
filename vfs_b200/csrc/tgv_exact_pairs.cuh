// Exact quotients and square roots of pairs of floats (packed FP32 instructions of sm_100).
//
// The float form has to give the bits of IEEE division and square root.  These build them from
// fused multiply-adds after P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor" (IBM J. Res. Dev. 34, 1990): with y the correctly rounded reciprocal of
// b and q within one ulp of a / b, q + (a - b q) y rounds to the correctly rounded quotient.  A
// reciprocal is shared by all the quotients that have it, there is no branch, and both halves of
// the packed instructions work.  Range: 2^-100 <= |b| <= 2^100 and quotients in the normal range
// (a = 0 included); a caller sees to it.
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
