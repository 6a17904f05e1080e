// Part of libctraj_probes.so (bench_kernels/).  Checks of the square roots and
// quotients the kernels form themselves.  The lens pass's FP32 root (sqrt32)
// against sqrtf for every float of its range; the soft lens pass's edge test
// (soft_test_r2) against the general one; the exact mode's FP64
// forms (fp64.cuh) against the IEEE operations they stand for, over generated
// operands: random significands with exponents of the lens pass and of the
// whole allowed range, significands near all-zeros and all-ones, and operands
// built to lie next to exact results and rounding boundaries (squares, products
// and their neighbours).
#include <cuda_runtime.h>

#include "adjoint.cuh"
#include "fp64.cuh"
#include "molecule.cuh"

namespace {

__device__ __forceinline__ unsigned long long mix(unsigned long long x) {  // splitmix64
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// a double in [2^-e, 2^e) with a random or extreme significand
__device__ __forceinline__ double operand(unsigned long long h, int e, unsigned kind) {
  unsigned long long sig = mix(h) & 0xFFFFFFFFFFFFFull;
  if (kind == 1) sig = mix(h) & 0x1F;
  if (kind == 2) sig = 0xFFFFFFFFFFFFFull - (mix(h) & 0x1F);
  if (kind == 3) sig &= ~((1ull << (mix(h + 7) % 52)) - 1);
  const unsigned long long ex = 1023ull - unsigned(e) + mix(h + 1) % unsigned(2 * e);
  return __longlong_as_double((long long)(ex << 52 | sig));
}
__device__ __forceinline__ double nudge(double a, unsigned long long h) {
  return __longlong_as_double(__double_as_longlong(a) + (long long)(h % 5) - 2);
}
__device__ __forceinline__ bool same(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }

__global__ void k_fp64_check(const long long n, const unsigned long long seed, unsigned long long* bad) {
  unsigned long long b_sqrt = 0, b_div = 0, b_div6 = 0, unsure = 0;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const unsigned long long h = mix(seed * 0x100000001ull + (unsigned long long)k);
    const unsigned kind = unsigned(h & 7);
    const int e = (h >> 3 & 3) ? 60 : 190;
    const double a = operand(h, e, kind), b = operand(h + 100, e, unsigned(h >> 5 & 7));
    // a square root and quotients by it, as the lens force forms them
    double x = a;
    if (kind == 4) x = nudge(__dmul_rn(a, a), h >> 9);
    double hh;
    bool sure;
    const double r = ctraj::sqrt64(x, hh, sure);
    b_sqrt += !sure || same(r, __dsqrt_rn(x)) ? 0 : 1;
    unsure += kind > 0 || sure ? 0 : 1;
    double num = b;
    if (kind == 5) num = nudge(__dmul_rn(b, r), h >> 9);
    if (kind == 6) num = -num;
    if (kind == 7) num = (h >> 12 & 1) ? 0.0 : -0.0;
    if (sure) {  // r is the rounded root
      const double v = ctraj::div64(num, r, ctraj::scale2(hh, 1), sure);
      b_div += !sure || same(v, __ddiv_rn(num, r)) ? 0 : 1;
      unsure += kind > 0 || sure ? 0 : 1;
    }
    // by a divisor whose rounded reciprocal is given
    if (kind == 5) num = nudge(__dmul_rn(b, a), h >> 9);
    const double v = ctraj::div64(num, a, __ddiv_rn(1.0, a), sure);
    b_div += !sure || same(v, __ddiv_rn(num, a)) ? 0 : 1;
    unsure += kind > 0 || sure ? 0 : 1;
    num = kind == 5 ? nudge(__dmul_rn(6.0, b), h >> 9) : kind == 7 ? -0.0 : num;
    if (ctraj::div6_ok(num)) b_div6 += same(ctraj::div6(num), __ddiv_rn(num, 6.0)) ? 0 : 1;
  }
  if (b_sqrt) atomicAdd(bad, b_sqrt);
  if (b_div) atomicAdd(bad + 1, b_div);
  if (b_div6) atomicAdd(bad + 2, b_div6);
  if (unsure) atomicAdd(bad + 3, unsure);
}

// every float of [2^-100, 2^100), and 0
__global__ void k_sqrt32_check(unsigned long long* bad) {
  unsigned long long b = 0;
  const unsigned lo = unsigned(127 - 100) << 23, hi = unsigned(127 + 100) << 23;
  for (unsigned k = lo + blockIdx.x * blockDim.x + threadIdx.x; k < hi; k += gridDim.x * blockDim.x) {
    const float a = __uint_as_float(k);
    b += __float_as_uint(ctraj::sqrt32(a)) == __float_as_uint(sqrtf(a)) && ctraj::sqrt32_ok(a) ? 0 : 1;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) b += __float_as_uint(ctraj::sqrt32(0.0f)) != 0u || !ctraj::sqrt32_ok(0.0f);
  if (b) atomicAdd(bad, b);
}

// At an edge of radius R and width 1 / inv_w: every y >= 0, infinity and a NaN
// with x = 0, then every squared radius t = x^2 + y^2: y is the root of t
// rounded down and x the root of what is left, exact there, so that
// fma(y, y, x x) rounds to t (from 2^-90 up, where what is left is a normal
// number; one that is not t there is counted as well).
__global__ void k_soft_test_check(float R, float inv_w, unsigned long long* bad) {
  unsigned long long b = 0;
  auto same = [](float p, float q) { return p == q || (isnan(p) && isnan(q)); };
  auto differ = [&](float x, float y, float r2) {
    float ls, d, ls2, d2;
    ctraj::soft_test(x, y, R, inv_w, ls, d);
    ctraj::soft_test_r2(r2, R, inv_w, ls2, d2);
    return same(ls, ls2) && same(d, d2) ? 0 : 1;
  };
  for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k <= 0x7f800001u; k += gridDim.x * blockDim.x) {
    const float v = __uint_as_float(k);
    b += differ(0.0f, v, __fmaf_rn(v, v, 0.0f));
    if (v < INFINITY) {
      const float y = __fsqrt_rd(v), x = __fsqrt_rn(fmaxf(__fmaf_rn(-y, y, v), 0.0f));
      const float t = __fmaf_rn(y, y, __fmul_rn(x, x));
      b += differ(x, y, t) + (v >= 0x1p-90f && t != v ? 1 : 0);
    }
  }
  if (b) atomicAdd(bad, b);
}

}  // namespace

extern "C" int ctraj_peak_soft_test_check(float R, float inv_w, unsigned long long* mismatches) {
  if (!mismatches) return -1;
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, sizeof *d) != cudaSuccess) return -3;
  cudaMemset(d, 0, sizeof *d);
  k_soft_test_check<<<1216, 256>>>(R, inv_w, d);
  cudaError_t e = cudaMemcpy(mismatches, d, sizeof *d, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? 0 : -2;
}

extern "C" int ctraj_peak_sqrt32_check(unsigned long long* mismatches) {
  if (!mismatches) return -1;
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, sizeof *d) != cudaSuccess) return -3;
  cudaMemset(d, 0, sizeof *d);
  k_sqrt32_check<<<1216, 256>>>(d);
  cudaError_t e = cudaMemcpy(mismatches, d, sizeof *d, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? 0 : -2;
}

// Returns 0 and, of n generated operand sets, the number of square roots,
// quotients and quotients by 6 that differ from the IEEE operation without
// saying so, and how many of the random ones (an eighth of the sets, three
// operations each) were unsure.
extern "C" int ctraj_peak_fp64_check(long long n, unsigned long long seed, unsigned long long* mismatches) {
  if (n < 1 || !mismatches) return -1;
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, 4 * sizeof *d) != cudaSuccess) return -3;
  cudaMemset(d, 0, 4 * sizeof *d);
  k_fp64_check<<<1216, 256>>>(n, seed, d);
  cudaError_t e = cudaMemcpy(mismatches, d, 4 * sizeof *d, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? 0 : -2;
}
