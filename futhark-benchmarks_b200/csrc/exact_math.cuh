// Correctly rounded f32 reciprocals, quotients and square roots inside a known
// range, for kernels whose f32 results are the IEEE ones bit for bit and whose time
// is in the divisions.
//
// near_rcp: the hardware's approximate reciprocal and one Newton iteration with
// its residual in a fused multiply-add; near_div: the quotient a * (1/b) and one
// correction by its exactly computed residual; near_sqrt the same from the
// approximate reciprocal square root -- Markstein's iterations ("Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990).  All give the
// correctly rounded value: near_rcp was compared with __frcp_rn at every float of
// exponent -125 .. 124, near_sqrt with __fsqrt_rn at every one of -87 .. 87,
// near_div with __fdiv_rn at every pair of significands (2^46), without a
// difference (tests/test_gpu_exact_math.py repeats the first two and a sample of the
// third); scaling by powers of two changes nothing while no operand, quotient or
// residual leaves the normal range.  The caller sees to that: it gathers the
// operands' range (RangeCheck) and starts over with __frcp_rn, __fdiv_rn and
// __fsqrt_rn where it was left.
//
// A reciprocal is three instructions and 27 cycles of a dependent chain, a
// further quotient by the same divisor three and 14; __frcp_rn takes 69 cycles
// and __fdiv_rn 45 there, with a branch each.
#pragma once

namespace {

// 1 / x for 2^-125 <= |x| < 2^125
__device__ __forceinline__ float near_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return __fmaf_rn(__fmaf_rn(-x, y, 1.0f), y, y);
}
// a / b with rb = 1 / b correctly rounded, for |a| in 2^-80 .. 2^80 or zero (-0 / b
// is then 0 of either sign), |b| and |a / b| in 2^-125 .. 2^120
__device__ __forceinline__ float near_div(float a, float b, float rb) {
  const float q = __fmul_rn(a, rb);
  return __fmaf_rn(__fmaf_rn(-b, q, a), rb, q);
}
// sqrt(x) for x in 2^-80 .. 2^80 or zero
__device__ __forceinline__ float near_sqrt(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  const float g = __fmul_rn(x, y);
  return x == 0.0f ? x : __fmaf_rn(__fmaf_rn(-g, g, x), __fmul_rn(0.5f, y), g);
}

// Whether the divisors seen so far lie inside (2^-40, 2^40) and the dividends are
// zero or inside (2^-80, 2^80): in near_rcp's, near_div's and near_sqrt's range.
// A NaN among them passes, and may: the iterations return NaN for it, as division
// does.  But an infinite dividend makes a NaN where division gives an infinity, and
// as a divisor or dividend further on that NaN would pass too, so every dividend is
// to be seen here: by its quotient, where that is a divisor and bounds it, from
// above at least (large).
struct RangeCheck {
  float lo = 1.0f, hi = 1.0f, nlo = 1.0f, nhi = 1.0f;
  __device__ __forceinline__ void divisor(float x) {
    lo = fminf(lo, fabsf(x));
    hi = fmaxf(hi, fabsf(x));
  }
  __device__ __forceinline__ void large(float x) { nhi = fmaxf(nhi, fabsf(x)); }
  __device__ __forceinline__ void dividend(float x) {
    nlo = fminf(nlo, x == 0.0f ? 1.0f : fabsf(x));
    large(x);
  }
  // where the divisors are near_rcp's alone
  __device__ __forceinline__ bool reciprocals_ok() const { return lo >= 0x1p-125f && hi < 0x1p125f; }
  // the dividends' limits: closer to one where quotients are dividends in turn
  __device__ __forceinline__ bool ok(float least = 0x1p-80f, float most = 0x1p80f) const {
    return lo > 0x1p-40f && hi < 0x1p40f && nlo > least && nhi < most;
  }
};

}  // namespace
