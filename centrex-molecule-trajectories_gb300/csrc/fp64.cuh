// IEEE-rounded FP64 building blocks with few FP64-pipe instructions.
//
// The FP64 pipe of this chip is the bound of every exact-mode kernel: one
// warp instruction takes 64 cycles of a scheduler's pipe (2 lanes per cycle
// and SM, whatever the number of active lanes, and without overlap of
// independent instructions of one warp), while integer and FP32 instructions
// issue every cycle.  So range tests, comparisons and scalings by powers of
// two are done on the integer pipe, the reciprocal of a divisor used twice is
// formed once, and divisions by constants use a precomputed reciprocal.
// Results are those of the IEEE operations bit for bit
// (bench_kernels/fp64_check.cu compares them with __dsqrt_rn and __ddiv_rn):
//   sqrt      seed, one third-order Goldschmidt step on sqrt and 1/(2 sqrt),
//             then the FMA residual correction g + (a - g^2) h (Markstein 1990;
//             Cornea, Harrison and Tang, "Scientific Computing on Itanium")
//   a / b     q = a y, r = a - b q by FMA, q + r y with y near 1 / b
//             (Markstein 1990)
//   a / 6     a z + a z' with z + z' the two-double reciprocal (Brisebarre,
//             Muller and Raina 2004)
// The corrected value of sqrt and a / b is within 2^-49 ulp of the exact one
// before its rounding, so the rounding can only be wrong when it lies that
// close to a tie: near_tie looks for 2^-18 ulp on the FP32 and integer pipes
// (20 instructions, a third of one FP64 instruction) and such a result is
// reported as unsure, as is an operand outside the stated exponent ranges,
// where an intermediate could under- or overflow; the caller takes the IEEE
// operation then.  a / 6 needs no look: a quotient by 6 is never nearer than
// 1/6 ulp to a tie.
// FP64 instructions: sqrt 8, which leaves 1 / sqrt as well (__dsqrt_rn 9.7),
// a / b 3 (__ddiv_rn 8.8), a / 6 2.
#pragma once
#include <cstdint>

namespace ctraj {

// The exact-mode lens passes give a molecule four lanes up to this many
// molecules in the queue: 1250 warps, two or three per scheduler of 152 SMs, take
// 87 x 152 cycles a step of k_lens_chunk64, 313 warps of one lane per molecule
// 222 x 64 (5 100 molecules, quads: 18.7 ms; 10 200, one lane while more than this
// are left: 27 ms; 17 000: 40 ms).
constexpr unsigned kQuad64Max = 10000;

__device__ __forceinline__ int hi_word(double a) { return __double2hiint(a); }

// |a| in [2^(lo), 2^(hi)): biased exponents [1023 + lo, 1023 + hi); false for
// zeros, infinities and NaNs when the bounds are inside the normal range.
template <int kLo, int kHi>
__device__ __forceinline__ bool in_range(double a) {
  return (unsigned(hi_word(a)) & 0x7fffffffu) - (unsigned(1023 + kLo) << 20) < (unsigned(kHi - kLo) << 20);
}
__device__ __forceinline__ bool is_zero(double a) {
  return ((unsigned(hi_word(a)) << 1) | unsigned(__double2loint(a))) == 0u;
}
// a * 2^k for normal a whose scaled value stays normal
__device__ __forceinline__ double scale2(double a, int k) {
  return __hiloint2double(hi_word(a) + (k << 20), __double2loint(a));
}
// a < b and a <= b for non-negative, non-NaN values, on the integer pipe
__device__ __forceinline__ bool less_pos(double a, double b) {
  return __double_as_longlong(a) < __double_as_longlong(b);
}

// float nearest below a >= 0 (0 below the normal floats), on the integer pipe
__device__ __forceinline__ float trunc_float(double a) {
  const int hi = hi_word(a);
  const unsigned lo = unsigned(__double2loint(a));
  return __uint_as_float(hi < (897 << 20) ? 0u : (unsigned(hi - (896 << 20)) << 3) | (lo >> 29));
}

// Whether q + a b, a correction of a few ulp(q) at most, may lie within 2^-18
// ulp(q) of a tie between neighbouring doubles; also true where q is next to a
// power of two, since ulp changes there.
__device__ __forceinline__ bool near_tie(double q, double a, double b) {
  const int hq = hi_word(q), ha = hi_word(a), hb = hi_word(b);
  const int e = ((ha & 0x7ff00000) + (hb & 0x7ff00000) - (hq & 0x7ff00000) >> 20) - 1023 + 52;  // a b / ulp(q) >= 2^e
  const float ma = __uint_as_float((__funnelshift_l(__double2loint(a), ha, 3) & 0x7fffffu) | 0x3f800000u);
  const float mb = __uint_as_float((__funnelshift_l(__double2loint(b), hb, 3) & 0x7fffffu) | 0x3f800000u);
  const float c = __int_as_float(__float_as_int(__fmul_rn(ma, mb)) + (max(e, -60) << 23));
  const float n = __fadd_rn(__fadd_rn(c, 8388608.0f), -8388608.0f);  // c to the nearest integer
  return !(fabsf(__fadd_rn(c, -n)) < 0.5f - 0x1p-18f) || (unsigned(hq) + 1u & 0xfffffu) < 2u;
}

// sqrt(a) rounded, and h within a few ulp of 1 / (2 sqrt(a)); sure: see above, a in [2^-500, 2^500).
__device__ __forceinline__ double sqrt64(double a, double& h, bool& sure) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  const double g0 = __dmul_rn(a, y), h0 = scale2(y, -1);
  const double e = __fma_rn(-g0, h0, 0.5);               // g0 h0 = 1/2 - e
  const double c = __dmul_rn(__fma_rn(1.5, e, 1.0), e);  // (1 - 2 e)^-1/2 - 1 to second order, e < 2^-19
  const double g = __fma_rn(g0, c, g0);
  h = __fma_rn(h0, c, h0);
  const double d = __fma_rn(-g, g, a);
  sure = in_range<-500, 500>(a) && !near_tie(g, d, h);
  return __fma_rn(d, h, g);
}

// a / b with y within a few ulp of 1 / b, b in [2^-400, 2^400); sure: see above, a zero or in [2^-400, 2^400).
__device__ __forceinline__ double div64(double a, double b, double y, bool& sure) {
  const double q = __dmul_rn(a, y);
  const double r = __fma_rn(-b, q, a);
  const double v = __fma_rn(r, y, q);
  const bool zero = is_zero(a);
  sure = zero || (in_range<-400, 400>(a) && !near_tie(q, r, y));
  return zero ? a : v;  // the correction gives +0 for a = -0
}

// a / 6; a zero or in [2^-900, 2^900)
__device__ __forceinline__ double div6(double a) {
  const double z = 0x1.5555555555555p-3, zl = 0x1.5555555555555p-57;  // z and 1/6 - z, rounded
  return __fma_rn(a, z, __dmul_rn(a, zl));
}
__device__ __forceinline__ bool div6_ok(double a) { return in_range<-900, 900>(a) || is_zero(a); }

}  // namespace ctraj
