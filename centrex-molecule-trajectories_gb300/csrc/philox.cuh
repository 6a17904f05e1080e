// Counter-based random numbers for on-device initial conditions.
//
// Philox-4x32-10 as published by Salmon, Moraes, Dror and Shaw, "Parallel
// random numbers: as easy as 1, 2, 3" (SC'11): ten rounds of two 32x32->64
// multiplies with the paper's multipliers and Weyl key increments.  Molecule i
// of a run with (seed, offset) uses key = seed and counter
// (lo32(offset + i), hi32(offset + i), call, 0), so any molecule can be
// regenerated from its index alone (used by the trajectory replay and by
// chunked or multi-replica runs with disjoint offsets).
//
// Uniforms: each 32-bit word w gives U = (w + 1/2) * 2^-32 in (0, 1); the FP32
// path rounds that value to float, so both precisions see the same draws.
// Normals: Box and Muller (1958), sqrt(-2 ln U1) * (cos 2 pi U2, sin 2 pi U2).
// FP64 evaluates them with CUDA's log / log1p, sqrt and sincospi; FP32 with
// the branch-free forms below (log1p from the atanh series, the square root
// as t rsqrt(t), sin and cos of pi a from their Taylor series), within a few
// ulp of the exact values (checked against FP64 on the device by
// bench_kernels/box_muller_check.cu).
#pragma once
#include <cstdint>

namespace ctraj {

struct Philox4 {
  uint32_t v[4];
};

__host__ __device__ inline void philox_round(uint32_t& c0, uint32_t& c1, uint32_t& c2, uint32_t& c3,
                                             uint32_t k0, uint32_t k1) {
  const uint64_t p0 = uint64_t(0xD2511F53u) * c0;
  const uint64_t p1 = uint64_t(0xCD9E8D57u) * c2;
  const uint32_t hi0 = uint32_t(p0 >> 32), lo0 = uint32_t(p0);
  const uint32_t hi1 = uint32_t(p1 >> 32), lo1 = uint32_t(p1);
  const uint32_t n0 = hi1 ^ c1 ^ k0;
  const uint32_t n2 = hi0 ^ c3 ^ k1;
  c0 = n0;
  c1 = lo1;
  c2 = n2;
  c3 = lo0;
}

// The ten round keys of a seed (the key plus r Weyl increments), computed on
// the host once per launch and read from the kernel parameters, so that no
// thread repeats the key schedule.
struct PhiloxKey {
  uint32_t k[20];  // round r: k[2r], k[2r + 1]
};

inline PhiloxKey philox_key(uint64_t seed) {
  PhiloxKey K;
  uint32_t k0 = uint32_t(seed), k1 = uint32_t(seed >> 32);
  for (int r = 0; r < 10; ++r) {
    K.k[2 * r] = k0;
    K.k[2 * r + 1] = k1;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return K;
}

__host__ __device__ inline Philox4 philox4x32_10(uint64_t ctr, uint32_t call, const PhiloxKey& K) {
  uint32_t c0 = uint32_t(ctr), c1 = uint32_t(ctr >> 32), c2 = call, c3 = 0u;
#pragma unroll
  for (int r = 0; r < 10; ++r) philox_round(c0, c1, c2, c3, K.k[2 * r], K.k[2 * r + 1]);
  return Philox4{{c0, c1, c2, c3}};
}

// log(1 + x) for x in [-1/2, 1], branch-free: 2 atanh(s) with s = x / (2 + x)
// in [-1/3, 1/3], from the series 2 s (1 + s^2/3 + s^4/5 + ... + s^14/15),
// whose next term is below 1.4e-9 relative; s by the fast division (2 ulp).
__device__ __forceinline__ float log1p_series(float s) {
  const float s2 = __fmul_rn(s, s);
  float p = 1.0f / 15.0f;
  p = __fmaf_rn(p, s2, 1.0f / 13.0f);
  p = __fmaf_rn(p, s2, 1.0f / 11.0f);
  p = __fmaf_rn(p, s2, 1.0f / 9.0f);
  p = __fmaf_rn(p, s2, 1.0f / 7.0f);
  p = __fmaf_rn(p, s2, 1.0f / 5.0f);
  p = __fmaf_rn(p, s2, 1.0f / 3.0f);
  p = __fmaf_rn(p, s2, 1.0f);
  return __fmul_rn(__fmul_rn(2.0f, s), p);
}
__device__ __forceinline__ float log1p_atanh(float x) { return log1p_series(__fdividef(x, __fadd_rn(2.0f, x))); }

// sin(pi a) and cos(pi a) for a in [0, 2], branch-free: a = j/2 + f with
// j = rint(2a) and |f| <= 1/4 (f exact), x = pi f, the Taylor series of sin
// to x^9 and of cos to x^10 (next terms below 3e-9 and 2e-10 relative for
// |x| <= pi/4), rotated by the quadrant j: sin(j pi/2 + x), cos(j pi/2 + x).
__device__ __forceinline__ void sincospi_taylor(float a, float& sn, float& cs) {
  const float j = rintf(__fmul_rn(2.0f, a));
  const float x = __fmul_rn(__fmaf_rn(-0.5f, j, a), 3.14159265358979323846f);
  const float x2 = __fmul_rn(x, x);
  float ps = 1.0f / 362880.0f;
  ps = __fmaf_rn(ps, x2, -1.0f / 5040.0f);
  ps = __fmaf_rn(ps, x2, 1.0f / 120.0f);
  ps = __fmaf_rn(ps, x2, -1.0f / 6.0f);
  const float s = __fmaf_rn(__fmul_rn(ps, x2), x, x);
  float pc = -1.0f / 3628800.0f;
  pc = __fmaf_rn(pc, x2, 1.0f / 40320.0f);
  pc = __fmaf_rn(pc, x2, -1.0f / 720.0f);
  pc = __fmaf_rn(pc, x2, 1.0f / 24.0f);
  pc = __fmaf_rn(pc, x2, -0.5f);
  const float c = __fmaf_rn(pc, x2, 1.0f);
  const int q = int(j) & 3;
  const float s1 = (q & 1) ? c : s, c1 = (q & 1) ? s : c;
  sn = (q & 2) ? -s1 : s1;
  cs = ((q + 1) & 2) ? -c1 : c1;
}

__device__ __forceinline__ float u01f(uint32_t w) {
  // (w + 1/2) 2^-32 rounded once to float; never 0
  return __fmaf_rn(__uint2float_rn(w), 2.3283064365386963e-10f, 1.1641532182693481e-10f);
}

__device__ __forceinline__ double u01d(uint32_t w) {
  return __fma_rn(double(w), 2.3283064365386963e-10, 1.1641532182693481e-10);
}

// ln U for U = (w + 1/2) 2^-32.  Above one half, U is close to 1 and a float
// holds it only to 2^-25 absolute, which would make the Box-Muller radius
// sqrt(-2 ln U) inaccurate near zero; there ln U = log1p(-V) with
// V = 1 - U = (~w + 1/2) 2^-32 formed exactly from the integer.  Below one
// half, U = 2^e m with m in [1, 2) and ln U = e ln 2 + log1p(m - 1) (m - 1
// exact), so both halves take the same single log1p and no lane diverges.
__device__ __forceinline__ float log_u01f(uint32_t w) {
  const bool low = w < 0x80000000u;
  const float u = u01f(low ? w : ~w);  // U, or V = 1 - U
  const uint32_t bits = __float_as_uint(u);
  const float e = float(int(bits >> 23) - 127);
  const float m1 = __fadd_rn(__uint_as_float((bits & 0x007fffffu) | 0x3f800000u), -1.0f);
  const float l = log1p_atanh(low ? m1 : -u);
  return low ? __fmaf_rn(e, 0.693147180559945309f, l) : l;
}

__device__ __forceinline__ double log_u01d(uint32_t w) {
  return (w < 0x80000000u) ? log(u01d(w)) : log1p(-u01d(~w));
}

__device__ __forceinline__ void box_muller(uint32_t w1, uint32_t w2, float& a, float& b) {
  const float t = __fmul_rn(-2.0f, log_u01f(w1));  // > 0: ln U < 0 for every word
  const float r = __fmul_rn(t, rsqrtf(t));
  float s, c;
  sincospi_taylor(__fmul_rn(2.0f, u01f(w2)), s, c);
  a = __fmul_rn(r, c);
  b = __fmul_rn(r, s);
}

__device__ __forceinline__ void box_muller(uint32_t w1, uint32_t w2, double& a, double& b) {
  const double r = sqrt(__dmul_rn(-2.0, log_u01d(w1)));
  double s, c;
  sincospi(__dmul_rn(2.0, u01d(w2)), &s, &c);
  a = __dmul_rn(r, c);
  b = __dmul_rn(r, s);
}

// Two FP32 box_muller calls, (w1.x, w2.x) and (w1.y, w2.y), by the packed
// FP32 instructions: the fronts are bound by the instructions they issue (73 %
// of the cycles at 1e7 molecules; 118 -> 108 us).  Every value is box_muller's: the division
// by 2 + x in [1.5, 3] and the rsqrt of t in [2^-32, 46] are rcp and rsqrt of
// normal numbers, the rounding to an integer j and its quadrant come from
// adding 1.5 2^23, the exponent from the integer behind 2^23.
__device__ __forceinline__ void box_muller_pair(const uint2 w1, const uint2 w2, float2& a, float2& b) {
  auto two = [](float v) { return make_float2(v, v); };
  auto rcp = [](float v) {
    float h;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(h) : "f"(v));
    return h;
  };
  auto rsqrt = [](float v) {
    float h;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(h) : "f"(v));
    return h;
  };
  auto u01 = [&](uint32_t p, uint32_t q) {
    return __ffma2_rn(make_float2(__uint2float_rn(p), __uint2float_rn(q)), two(2.3283064365386963e-10f),
                      two(1.1641532182693481e-10f));
  };
  // ln U (log_u01f)
  const bool low0 = int32_t(w1.x) >= 0, low1 = int32_t(w1.y) >= 0;
  const float2 u = u01(w1.x ^ uint32_t(int32_t(w1.x) >> 31), w1.y ^ uint32_t(int32_t(w1.y) >> 31));
  const uint32_t b0 = __float_as_uint(u.x), b1 = __float_as_uint(u.y);
  const float2 e = __fadd2_rn(make_float2(__uint_as_float((b0 >> 23) | 0x4B000000u), __uint_as_float((b1 >> 23) | 0x4B000000u)),
                              two(-8388735.0f));
  const float2 m1 = __fadd2_rn(make_float2(__uint_as_float((b0 & 0x007fffffu) | 0x3f800000u),
                                           __uint_as_float((b1 & 0x007fffffu) | 0x3f800000u)), two(-1.0f));
  const float2 x = make_float2(low0 ? m1.x : -u.x, low1 ? m1.y : -u.y);
  const float2 n = __fadd2_rn(two(2.0f), x);
  const float2 s = __fmul2_rn(x, make_float2(rcp(n.x), rcp(n.y))), s2 = __fmul2_rn(s, s);
  float2 p = two(1.0f / 15.0f);
  p = __ffma2_rn(p, s2, two(1.0f / 13.0f));
  p = __ffma2_rn(p, s2, two(1.0f / 11.0f));
  p = __ffma2_rn(p, s2, two(1.0f / 9.0f));
  p = __ffma2_rn(p, s2, two(1.0f / 7.0f));
  p = __ffma2_rn(p, s2, two(1.0f / 5.0f));
  p = __ffma2_rn(p, s2, two(1.0f / 3.0f));
  p = __ffma2_rn(p, s2, two(1.0f));
  const float2 l = __fmul2_rn(__fmul2_rn(two(2.0f), s), p);
  const float2 ln = __ffma2_rn(make_float2(low0 ? e.x : 0.0f, low1 ? e.y : 0.0f), two(0.693147180559945309f), l);
  const float2 t = __fmul2_rn(two(-2.0f), ln);
  const float2 r = __fmul2_rn(t, make_float2(rsqrt(t.x), rsqrt(t.y)));
  // sin and cos of 2 pi U2 (sincospi_taylor)
  const float2 ang = __fmul2_rn(two(2.0f), u01(w2.x, w2.y));
  const float2 m = __ffma2_rn(two(2.0f), ang, two(12582912.0f));
  const float2 j = __fadd2_rn(m, two(-12582912.0f));
  const float2 f = __fmul2_rn(__ffma2_rn(two(-0.5f), j, ang), two(3.14159265358979323846f));
  const float2 f2 = __fmul2_rn(f, f);
  float2 ps = two(1.0f / 362880.0f);
  ps = __ffma2_rn(ps, f2, two(-1.0f / 5040.0f));
  ps = __ffma2_rn(ps, f2, two(1.0f / 120.0f));
  ps = __ffma2_rn(ps, f2, two(-1.0f / 6.0f));
  const float2 sn = __ffma2_rn(__fmul2_rn(ps, f2), f, f);
  float2 pc = two(-1.0f / 3628800.0f);
  pc = __ffma2_rn(pc, f2, two(1.0f / 40320.0f));
  pc = __ffma2_rn(pc, f2, two(-1.0f / 720.0f));
  pc = __ffma2_rn(pc, f2, two(1.0f / 24.0f));
  pc = __ffma2_rn(pc, f2, two(-0.5f));
  const float2 cs = __ffma2_rn(pc, f2, two(1.0f));
  // the quadrant: q = j mod 4 in the low bits of m
  auto turn = [](uint32_t q, float sv, float cv, float& so, float& co) {
    const float s1 = (q & 1u) ? cv : sv, c1 = (q & 1u) ? sv : cv;
    so = __uint_as_float(__float_as_uint(s1) ^ ((q << 30) & 0x80000000u));
    co = __uint_as_float(__float_as_uint(c1) ^ (((q << 30) + 0x40000000u) & 0x80000000u));
  };
  float2 so, co;
  turn(__float_as_uint(m.x), sn.x, cs.x, so.x, co.x);
  turn(__float_as_uint(m.y), sn.y, cs.y, so.y, co.y);
  a = __fmul2_rn(r, co);
  b = __fmul2_rn(r, so);
}
// FP64: one after the other
__device__ __forceinline__ void box_muller_pair(const uint2 w1, const uint2 w2, double2& a, double2& b) {
  box_muller(w1.x, w2.x, a.x, b.x);
  box_muller(w1.y, w2.y, a.y, b.y);
}

// The eight words of two Philox calls and how they are used:
//   (w0, w1) -> normals n0, n1 -> vx, vy
//   (w2, w3) -> normals n2, n3 -> vz, Gaussian x
//   (w4, w5) -> normals n4, _  -> Gaussian y
//   w6, w7   -> disc angle and radius (CeNTREXPositionDistribution)
struct Words8 {
  uint32_t w[8];
};

__device__ __forceinline__ Words8 molecule_words(uint64_t id, const PhiloxKey& K) {
  const Philox4 a = philox4x32_10(id, 0u, K);
  const Philox4 b = philox4x32_10(id, 1u, K);
  return Words8{{a.v[0], a.v[1], a.v[2], a.v[3], b.v[0], b.v[1], b.v[2], b.v[3]}};
}

}  // namespace ctraj
