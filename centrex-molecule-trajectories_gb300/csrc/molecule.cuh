// Per-molecule state and element physics, in two precisions.
//
// Mol64 follows the reference's float64 operation order step for step, using
// __dadd_rn/__dmul_rn (never contracted into FMA) and IEEE division and square
// root, so on ballistic paths it reproduces the reference bit for bit:
//   update_trajectory    molecule.py:26-68
//   aperture hit tests   apertures.py:101-115, 174-189
//   field plates         apertures.py:227-270
//   lens force           electrostatic_lens.py:215-227 with scipy's PPoly
//                        (nu = 1) or numpy.interp evaluation order
//   lens RK4 step        electrostatic_lens.py:91-118
//
// Mol32 restates the same physics for speed.  The molecule always sits on the
// last plane it reached, so a flight is (plane gap) * (1/vz) with the gap
// precomputed in double on the host; z itself is never accumulated in float.
// Inside the lens only the transverse state (x, y, vx, vy) evolves (a_z = 0)
// and the force is a_perp = w(|r|) * (x, y) - g y^, w read from a per-interval
// polynomial table.  The RK4 combination is rewritten exactly:
//   x' = x + dt v + dt^2/6 (l1 + l2 + l3),  v' = v + dt/6 (l1 + 2 l2 + 2 l3 + l4)
// (the reference's k1..k4 substituted); each increment is formed in full
// precision and added with a carried rounding error (compensated summation),
// and the step count, step size and exit-snap time are computed once per
// molecule in double.
#pragma once
#include <cfloat>
#include <cmath>
#include <cstdint>

#include "fp64.cuh"
#include "philox.cuh"
#include "plan.cuh"

namespace ctraj {

__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }

// ---------------------------------------------------------------------------
// FP64 force table lookups (reference evaluation order)
// ---------------------------------------------------------------------------

// scipy PPoly.__call__(E, nu=1): interval knots[i] <= E < knots[i+1], end
// pieces extrapolated; res = 0 + c2*1*1; res += (c1*s)*2; res += (c0*(s*s))*3.
__device__ inline double spline_deriv64(const TableD& T, double E, int& range) {
  const int n = T.n;
  int i;
  if (isnan(E)) return E;
  if (E < T.x0) {
    i = 0;
    range = 1;
  } else if (E >= __ldg(T.knots + n - 1)) {
    i = n - 2;
    if (E > __ldg(T.knots + n - 1)) range = 1;
  } else {
    i = int(floor((E - T.x0) / T.h));
    i = max(0, min(i, n - 2));
    while (i > 0 && E < __ldg(T.knots + i)) --i;
    while (i < n - 2 && E >= __ldg(T.knots + i + 1)) ++i;
  }
  const double* c = T.coef + 4 * size_t(i);
  const double s = dadd(E, -__ldg(T.knots + i));
  double res = 0.0;
  res = dadd(res, dmul(dmul(__ldg(c + 2), 1.0), 1.0));
  res = dadd(res, dmul(dmul(__ldg(c + 1), s), 2.0));
  res = dadd(res, dmul(dmul(__ldg(c + 0), dmul(s, s)), 3.0));
  return res;
}

// numpy.interp(r, knots, values) (what scipy's float64 linear interp1d calls),
// with interp1d's bounds error above the last knot reported through err.
__device__ inline double radial64(const TableD& T, double r, int& err) {
  const int n = T.n;
  const double last = __ldg(T.knots + n - 1);
  if (r < T.x0 || r > last) {
    err = 1;
    return nan("");
  }
  if (isnan(r)) return r;
  int j = int(floor((r - T.x0) / T.h));
  j = max(0, min(j, n - 1));
  while (j > 0 && __ldg(T.knots + j) > r) --j;
  while (j < n - 1 && __ldg(T.knots + j + 1) <= r) ++j;
  const double xj = __ldg(T.knots + j), yj = __ldg(T.values + j);
  if (j == n - 1 || xj == r) return yj;
  const double slope = (__ldg(T.values + j + 1) - yj) / (__ldg(T.knots + j + 1) - xj);
  return dadd(dmul(slope, dadd(r, -xj)), yj);
}

// ElectrostaticLens.lens_acceleration (electrostatic_lens.py:215-227).
__device__ inline void lens_force64(const Plan& P, const ctraj_element& e, double x0, double x1,
                                    double& a0, double& a1, int& range, int& err) {
  const TableD& T = P.td[e.table];
  const double r = __dsqrt_rn(dadd(dmul(x0, x0), dmul(x1, x1)));
  double a_r;
  if (T.kind == CTRAJ_TABLE_RADIAL_LINEAR) {
    a_r = radial64(T, r, err);
  } else {
    const double alpha = e.p[6], mass = e.p[5];
    if (e.field_order == 1) {
      const double E = dmul(alpha, r);
      a_r = -dmul(spline_deriv64(T, E, range), alpha) / mass;
    } else {
      const double E = dmul(alpha, dmul(r, r));
      a_r = -dmul(spline_deriv64(T, E, range), dmul(dmul(2.0, alpha), r)) / mass;
    }
  }
  a0 = 0.0;
  a1 = 0.0;
  if (r != 0.0) {
    a0 = dmul(a_r, x0) / r;
    a1 = dmul(a_r, x1) / r;
  }
  a1 = dadd(a1, -P.g);
}

// ---------------------------------------------------------------------------
// Honeycomb nearest cell (meshes.py:104-108)
// ---------------------------------------------------------------------------
// The reference takes numpy's argmin over ALL centres of
// sqrt((px - xc)**2 + (py - yc)**2): the first of equal minima, 0 when no
// distance is finite.  The centres form hexalattice rows of nx cells (odd rows
// shifted by half a pitch), so the nearest centre of an interior point is at
// most one row and one cell from the rounded estimate, and the second-nearest
// at most two.  Outside the grid the estimate is clamped; the nearest and
// second-nearest centres of a point beyond the first or last row are among
// the outermost four rows (the nearest of each row is its cell closest in x,
// and rows alternate their half-pitch shift), so the window takes rows
// j0-2..j0+2, widened to four rows at either end, and cells i0-2..i0+2 of each.
// Scanning the window rows and cells in ascending order visits cells in
// ascending index, so strict < keeps the first minimum as argmin does.

// rows of the search window around the (clamped) estimate j0 of ny rows
__device__ __forceinline__ void window_rows(int j0, int ny, int& lo, int& hi) {
  lo = j0 == ny - 1 ? max(ny - 4, 0) : max(j0 - 2, 0);
  hi = j0 == 0 ? min(3, ny - 1) : min(j0 + 2, ny - 1);
}

// round(u) clamped to [0, hi]; NaN -> 0
__device__ __forceinline__ int window_index(double u, int hi) {
  const double r = floor(u + 0.5);
  if (!(r >= 0.0)) return 0;
  return r >= double(hi) ? hi : int(r);
}

// FP64, the reference's operations; best / second: the two smallest distances.
__device__ inline int mesh_nearest64(const TableD& T, const double* p, double px, double py, double& best,
                                     double& second) {
  const int nx = int(p[1]), ny = T.n / nx;
  const int j0 = window_index((py - __ldg(T.values)) * p[2], ny - 1);
  int lo, hi;
  window_rows(j0, ny, lo, hi);
  int idx = -1;
  best = INFINITY;
  second = INFINITY;
  for (int j = lo; j <= hi; ++j) {
    const int row = j * nx;
    const int i0 = window_index((px - __ldg(T.knots + row)) * p[3], nx - 1);
    for (int k = row + max(i0 - 2, 0); k <= row + min(i0 + 2, nx - 1); ++k) {
      const double dx = dadd(px, -__ldg(T.knots + k)), dy = dadd(py, -__ldg(T.values + k));
      const double d = __dsqrt_rn(dadd(dmul(dx, dx), dmul(dy, dy)));
      if (d < best) {
        second = best;
        best = d;
        idx = k;
      } else if (d < second) {
        second = d;
      }
    }
  }
  return idx < 0 ? 0 : idx;
}

// FP32 on the float4 (x, y, 0, 0) centre table; squared distances.
__device__ __forceinline__ int window_index32(float u, int hi) {
  const float r = floorf(u + 0.5f);
  if (!(r >= 0.0f)) return 0;
  return r >= float(hi) ? hi : int(r);
}

__device__ inline int mesh_nearest32(const LensF& L, const ElemF& f, float px, float py, float& best2,
                                     float& second2) {
  const int nx = L.cols, ny = L.n_int / nx;
  const int j0 = window_index32((py - __ldg(&L.q[0].y)) * f.c[2], ny - 1);
  int lo, hi;
  window_rows(j0, ny, lo, hi);
  int idx = -1;
  best2 = INFINITY;
  second2 = INFINITY;
  for (int j = lo; j <= hi; ++j) {
    const int row = j * nx;
    const int i0 = window_index32((px - __ldg(&L.q[row].x)) * f.c[3], nx - 1);
    for (int k = row + max(i0 - 2, 0); k <= row + min(i0 + 2, nx - 1); ++k) {
      const float4 c = __ldg(L.q + k);
      const float dx = px - c.x, dy = py - c.y;
      const float d2 = __fmaf_rn(dy, dy, __fmul_rn(dx, dx));
      if (d2 < best2) {
        second2 = best2;
        best2 = d2;
        idx = k;
      } else if (d2 < second2) {
        second2 = d2;
      }
    }
  }
  return idx < 0 ? 0 : idx;
}

// ---------------------------------------------------------------------------
// FP32 table interval: i = min(trunc_to_unsigned(s), last) and u = s - i, as
// the truncating float-to-unsigned conversion and its inverse give them
// (negative and NaN s -> interval 0; u keeps s's own offset), without the
// conversion unit: 2^23 + max(s, 0) rounded toward -inf is 2^23 + floor(s)
// for s < 2^23 (the spacing of floats in [2^23, 2^24) is 1), so floor(s)
// sits in the low mantissa bits and 2^23 subtracts back exactly; larger s
// and infinity land on the clamp.  Bit-identical to the conversions, on
// FP32 / integer pipes instead of the conversion pipe.  The soft-transmission
// kernels (4 % faster) and the linear-table lens lookups (one warp's step
// 323 -> 231 cycles) use it, the lens lookups in packed form (force_pair).
// kNonNeg: s is known to be >= 0 or NaN (a linear Stark table starts at
// |E| = 0 and its coordinate scale is not negative), so max(s, 0) is left
// out; only a NaN s then takes the last interval instead of the first, and
// u, hence the force, is NaN either way.
// ---------------------------------------------------------------------------
template <bool kNonNeg = false>
__device__ __forceinline__ void table_interval(const float s, const unsigned last, const float last_f,
                                               unsigned& i, float& u) {
  const float t = __fadd_rd(kNonNeg ? s : fmaxf(s, 0.0f), 8388608.0f);
  i = min(__float_as_uint(t) - 0x4B000000u, last);
  u = __fadd_rn(s, -fminf(__fadd_rn(t, -8388608.0f), last_f));
}

// ---------------------------------------------------------------------------
// FP32 force: w such that a_perp = w * (x, y), at two points at once
// ---------------------------------------------------------------------------
// A step's force evaluations come in two pairs: the stage-2 point does not
// depend on the stage-1 force, nor the stage-4 point on the stage-3 force.
// Each pair's table coordinates, intervals and offsets go through the packed
// FP32 instructions (two components per instruction, each rounded as the
// scalar one).
// kStaged: the whole table is in shared memory (tab); otherwise tab is read
// from global memory through the read-only cache.  Lookups past the last
// interval extrapolate it (as scipy CubicSpline does); s < 0 uses interval 0.
// `beta` is the table-coordinate scale (L.beta, or a molecule's own in a
// batched sweep where each configuration has its lens voltage).
// The interval is table_interval's; the linear form leaves its max(s, 0) out:
// the table starts at |E| = 0 and no coordinate scale is negative, so s >= 0
// or NaN (last piece; u and the force are NaN).
struct PairTable {
  const float4* tab;
  unsigned last;  // last interval (linear form: last of the 2 n_int pieces)
  float last_f;
  __device__ __forceinline__ const float2* pieces() const { return reinterpret_cast<const float2*>(tab); }
};
template <int F>
__device__ __forceinline__ PairTable pair_table(const LensArgs& L, const float4* tab) {
  const int n = F == kForceStark2Lin ? 2 * L.n_int : L.n_int;
  return PairTable{tab, unsigned(n - 1), float(n - 1)};
}

__device__ __forceinline__ float2 pack2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }

// interval of t = 2^23 + s rounded toward -inf
__device__ __forceinline__ unsigned interval_of(float t, unsigned last) {
  return __viaddmin_u32(__float_as_uint(t), 0u - 0x4B000000u, last);
}

// The rounded square root for a in [2^-100, 2^100) or 0, without the slow-path
// call of sqrtf that keeps a pair's evaluations from overlapping: g + (a - g^2)
// h from an approximate root g and h = 1 / (2 g) (Markstein 1990), equal to
// sqrtf for every such a (bench_kernels/fp64_check.cu runs through them all).
__device__ __forceinline__ float sqrt32(float a) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(fmaxf(a, 0x1p-100f)));
  const float g = __fmul_rn(a, y);
  return __fmaf_rn(__fmaf_rn(-g, g, a), __fmul_rn(0.5f, y), g);
}
__device__ __forceinline__ bool sqrt32_ok(float a) { return (a >= 0x1p-100f && a < 0x1p100f) || a == 0.0f; }

// Bits of a step's flags: a lookup above a radial table; kFast: a root outside
// sqrt32's range.
enum : unsigned { kFlagAbove = 2u, kFlagRoot = 4u };

// w at squared radii r2.  kFast: roots by sqrt32, the step's flags telling
// when one was out of its range and the step is to be taken again without.
template <int F, bool kStaged, bool kFast>
__device__ __forceinline__ float2 force_pair(const LensArgs& L, const PairTable& T, const float2 r2, const float beta,
                                             unsigned& flags) {
  const float2 c23 = pack2(8388608.0f, 8388608.0f);
  float2 r = r2;
  if constexpr (F == kForceStark1 || F == kForceRadial) {
    if constexpr (kFast) {
      r = pack2(sqrt32(r2.x), sqrt32(r2.y));
      flags |= sqrt32_ok(r2.x) && sqrt32_ok(r2.y) ? 0u : kFlagRoot;
    } else {
      r = pack2(sqrtf(r2.x), sqrtf(r2.y));
    }
    if (F == kForceRadial) flags |= (r.x > L.r_max || r.y > L.r_max) ? kFlagAbove : 0u;
  }
  const float2 s = __ffma2_rn(pack2(beta, beta), r, pack2(-L.s0, -L.s0));
  const float2 t = __fadd2_rd(F == kForceStark2Lin ? s : pack2(fmaxf(s.x, 0.0f), fmaxf(s.y, 0.0f)), c23);
  const unsigned i = interval_of(t.x, T.last), j = interval_of(t.y, T.last);
  const float2 f = __fadd2_rn(t, neg2(c23));
  const float2 u = __fadd2_rn(s, pack2(-fminf(f.x, T.last_f), -fminf(f.y, T.last_f)));
  if constexpr (F == kForceStark2Lin) {
    const float2 a = kStaged ? T.pieces()[i] : __ldg(T.pieces() + i);
    const float2 b = kStaged ? T.pieces()[j] : __ldg(T.pieces() + j);
    return pack2(__fmaf_rn(u.x, a.y, a.x), __fmaf_rn(u.y, b.y, b.x));
  } else {
    const float4 a = kStaged ? T.tab[i] : __ldg(T.tab + i), b = kStaged ? T.tab[j] : __ldg(T.tab + j);
    if constexpr (F == kForceRadial) {
      const float2 w = pack2(__fmaf_rn(u.x, a.y, a.x), __fmaf_rn(u.y, b.y, b.x));
      return pack2(r.x > 0.0f ? __fdividef(w.x, r.x) : 0.0f, r.y > 0.0f ? __fdividef(w.y, r.y) : 0.0f);
    }
    const float2 w = pack2(__fmaf_rn(u.x, __fmaf_rn(u.x, a.z, a.y), a.x), __fmaf_rn(u.y, __fmaf_rn(u.y, b.z, b.y), b.x));
    if constexpr (F == kForceStark1)
      return pack2(r.x > 0.0f ? __fdividef(w.x, r.x) : 0.0f, r.y > 0.0f ? __fdividef(w.y, r.y) : 0.0f);
    return w;
  }
}

// Pieces loaded a step ahead of their use (lens_step_ahead; linear form): the
// table coordinates s of the last step's stages (1, 2) and (4, 3) and their
// differences d to the step before, and the pieces at the coordinates
// extrapolated from them, with the pieces' starts k.
struct LinAhead {
  float2 s12, d12, s43, d43;
  float2 k12, k43;
  float2 e1, e2, e4, e3;
  __device__ __forceinline__ void clear() {
    s12 = d12 = s43 = d43 = e1 = e2 = e4 = e3 = pack2(0.0f, 0.0f);
    k12 = k43 = pack2(-1.0f, -1.0f);  // s - k >= 1: not a piece's offset
  }
  // the next coordinates after s, from the last three: 3 s - 3 s' + s'' = s + 2 d - d'
  static __device__ __forceinline__ float2 next(const float2 s, float2& last, float2& diff) {
    const float2 d = __fadd2_rn(s, neg2(last)), p = __fadd2_rn(__ffma2_rn(pack2(2.0f, 2.0f), d, s), neg2(diff));
    last = s;
    diff = d;
    return p;
  }
  // the pieces at expected coordinates p12, p43 (any value: the index is clamped)
  __device__ __forceinline__ void load(const PairTable& T, const float2 p12, const float2 p43) {
    const float2 c = pack2(8388608.0f, 8388608.0f);
    const float2 t = __fadd2_rd(p12, c), u = __fadd2_rd(p43, c);
    e1 = T.pieces()[interval_of(t.x, T.last)];
    e2 = T.pieces()[interval_of(t.y, T.last)];
    e4 = T.pieces()[interval_of(u.x, T.last)];
    e3 = T.pieces()[interval_of(u.y, T.last)];
    const float2 f = __fadd2_rn(t, neg2(c)), g = __fadd2_rn(u, neg2(c));
    // as unsigned words a negative start is above the last one and is clamped with it
    auto clamp = [&](float b) { return __uint_as_float(min(__float_as_uint(b), __float_as_uint(T.last_f))); };
    k12 = pack2(clamp(f.x), clamp(f.y));
    k43 = pack2(clamp(g.x), clamp(g.y));
  }
};

// Per-molecule lens integration parameters (both precisions).
struct LensStep {
  int n_total;  // rint(L/dz), at most CTRAJ_MAX_LENS_STEPS; -1 while the setup is pending
  int n_done;
  int bound;    // upper bound on n_total while the setup is pending
  double dt;        // dz / vz
  double snap;      // FP32: exit-snap time (z1 - z0 - N dz) / vz
  double dz;
};

// Step count and step size exactly as electrostatic_lens.py:87-88, in double.
__device__ __forceinline__ bool lens_setup(const ctraj_element& e, double vz, LensStep& s) {
  const double dz = e.step_mode == CTRAJ_STEP_DT ? dmul(vz, e.p[2]) : e.p[1];
  const double nf = rint(e.p[7] / dz);
  s.dz = dz;
  s.n_done = 0;
  if (!(fabs(nf) <= double(CTRAJ_MAX_LENS_STEPS))) {  // also catches NaN / inf
    s.n_total = 0;
    s.dt = 0.0;
    s.snap = 0.0;
    return false;
  }
  s.n_total = nf < 0.0 ? 0 : int(nf);
  s.dt = dz / vz;
  s.snap = ((e.z1 - e.z0) - double(s.n_total) * dz) / vz;
  return true;
}

// Trajectory row sink used by the replay kernel.
struct RowSink {
  double* out;   // (max_rows, 10)
  int max_rows;
  int stride;
  int64_t row;   // index of the last stored row (0 = initial)
  int written;
  bool last_written;
  // Plane mode (stride 1, out unused): follow the rows to the crossing of the
  // plane z = zp the way post_processing.py:37-76 reads a trajectory: the first
  // row anywhere with z == zp (pexact; the lens's last steps can overshoot z1
  // and the exit snap come back to it), else the row before the first one with
  // z >= zp (pcross = 2; 3 when that is the first row: Python's index -1, the
  // last row); rows with a non-finite value are skipped, as drop_nans
  // (molecule.py:160-167) removes them.
  bool plane;
  bool pexact;
  int pcross;
  double zp;
  double prev[10], hit[10], last[10], exact[10];
  __device__ void put(double x, double y, double z, double vx, double vy, double vz, double ax,
                      double ay, double az, double t) {
    ++row;
    last_written = false;
    if (row % stride == 0) write(x, y, z, vx, vy, vz, ax, ay, az, t);
  }
  __device__ void write(double x, double y, double z, double vx, double vy, double vz, double ax,
                        double ay, double az, double t) {
    if (plane) {
      const double r[10] = {x, y, z, vx, vy, vz, ax, ay, az, t};
      bool finite = true;
      for (int k = 0; k < 10; ++k) finite = finite && isfinite(r[k]);
      if (finite) {
        if (!pexact && z == zp) {
          for (int k = 0; k < 10; ++k) exact[k] = r[k];
          pexact = true;
        }
        if (pcross == 0 && !(z < zp)) {
          if (written == 0) {
            pcross = 3;
          } else {
            for (int k = 0; k < 10; ++k) hit[k] = prev[k];
            pcross = 2;
          }
        }
        for (int k = 0; k < 10; ++k) prev[k] = last[k] = r[k];
        ++written;
      }
      last_written = true;
      return;
    }
    if (written < max_rows) {
      double* o = out + size_t(written) * 10;
      o[0] = x; o[1] = y; o[2] = z; o[3] = vx; o[4] = vy; o[5] = vz;
      o[6] = ax; o[7] = ay; o[8] = az; o[9] = t;
    }
    ++written;
    last_written = true;
  }
};

// ===========================================================================
// FP64: the reference's arithmetic
// ===========================================================================
template <bool kRec>
struct Mol64 {
  static constexpr bool kScreenable = false;  // the front's screening is FP32's (Mol32)
  double x[3], v[3], a[3], t;
  double margin;
  int rows;
  int32_t id;
  RowSink* sink;

  __device__ void row_out() {
    if (kRec) sink->put(x[0], x[1], x[2], v[0], v[1], v[2], a[0], a[1], a[2], t);
  }

  __device__ void init(const Plan& P, const RunDev& R, int64_t i) {
    id = int32_t(i);
    margin = INFINITY;
    rows = 0;
    if (R.ic_mode == CTRAJ_IC_DEVICE_DRAW) {
      const Words8 w = molecule_words(R.offset + uint64_t(i), R.key);
      double n0, n1, n2, n3, n4, n5;
      box_muller(w.w[0], w.w[1], n0, n1);
      box_muller(w.w[2], w.w[3], n2, n3);
      box_muller(w.w[4], w.w[5], n4, n5);
      const double* vp = R.vd.p;
      v[0] = __fma_rn(vp[1], n0, vp[0]);
      v[1] = __fma_rn(vp[3], n1, vp[2]);
      v[2] = __fma_rn(vp[5], n2, vp[4]);
      const double* xp = R.xd.p;
      if (R.xd.kind == CTRAJ_DIST_DISC_POSITION) {
        double s, c;
        sincospi(2.0 * u01d(w.w[6]), &s, &c);
        const double rr = dmul(sqrt(u01d(w.w[7])), dmul(xp[0], 0.5));
        x[0] = dmul(rr, c);
        x[1] = dmul(rr, s);
        x[2] = xp[1];
      } else {
        x[0] = dmul(xp[0], n3);
        x[1] = dmul(xp[1], n4);
        x[2] = xp[2];
      }
    } else {
      const size_t n = size_t(R.n);
      for (int k = 0; k < 3; ++k) {
        x[k] = R.ics[k * n + size_t(i)];
        v[k] = R.ics[(3 + k) * n + size_t(i)];
      }
    }
    a[0] = 0.0;
    a[1] = -P.g;
    a[2] = 0.0;
    t = 0.0;
    if (kRec) sink->write(x[0], x[1], x[2], v[0], v[1], v[2], a[0], a[1], a[2], t);
  }

  // Molecule.update_trajectory(delta_t, a=(0,-g,0)).  In a flight with a_x and
  // a_z zero their terms are +0 or -0, which change a sum only where it is -0
  // itself: 22 FP64 instructions instead of 35 (with the tests on the integer
  // pipe; front of 1e5 ballistic molecules 35.7 -> 29.5 us), all of them for
  // other accelerations and for numbers whose products could leave the normal
  // range.
  __device__ void update(double dt, const Plan& P) {
    if (!is_zero(dt)) {  // `if not delta_t` keeps x and v (molecule.py:31,41)
      const double dt2 = dmul(dt, dt);
      if (__double_as_longlong(a[0]) == 0 && __double_as_longlong(a[2]) == 0 && in_range<-200, 200>(dt) &&
          in_range<-200, 200>(a[1]) && !is_zero(v[0]) && !is_zero(v[2])) {
        const double sx = dadd(x[0], dmul(v[0], dt)), sz = dadd(x[2], dmul(v[2], dt));
        x[0] = is_zero(sx) ? 0.0 : sx;
        x[2] = is_zero(sz) ? 0.0 : sz;
        x[1] = dadd(dadd(x[1], dmul(v[1], dt)), dmul(scale2(a[1], -1), dt2));
        v[1] = dadd(v[1], dmul(a[1], dt));
      } else {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          x[k] = dadd(dadd(x[k], dmul(v[k], dt)), dmul(dmul(a[k], dt2), 0.5));
          v[k] = dadd(v[k], dmul(a[k], dt));
        }
      }
    }
    t = dadd(t, dt);
    a[0] = 0.0;
    a[1] = -P.g;
    a[2] = 0.0;
    rows += (hi_word(t) & 0x7ff00000) != 0x7ff00000 ? 1 : 0;  // finite
    row_out();
  }

  __device__ void fly(const Plan& P, int i, int which) {
    const double z = which ? P.el[i].z1 : P.el[i].z0;
    update((z - x[2]) / v[2], P);
  }

  __device__ double rho() const { return __dsqrt_rn(dadd(dmul(x[0], x[0]), dmul(x[1], x[1]))); }

  __device__ void note(double d) { margin = fmin(margin, fabs(d)); }

  __device__ bool circle_out(const Plan& P, int i) {
    const double r = rho(), h = dmul(P.el[i].p[0], 0.5);
    note(dadd(r, -h));
    return r > h;
  }
  __device__ bool rect_out(const Plan& P, int i) {
    const double* p = P.el[i].p;
    note(dadd(x[0], -p[0])); note(dadd(x[0], -p[1])); note(dadd(x[1], -p[2])); note(dadd(x[1], -p[3]));
    return !((p[0] < x[0] && x[0] < p[1]) && (p[2] < x[1] && x[1] < p[3]));
  }
  // FieldPlates after the z0 flight: returns true when lost (apertures.py:238-270)
  __device__ bool plates(const Plan& P, int i) {
    const double x1 = P.el[i].p[0], x2 = P.el[i].p[1];
    note(dadd(x[0], -x1)); note(dadd(x[0], -x2));
    if (!(x1 < x[0] && x[0] < x2)) return true;
    double dt = (P.el[i].z1 - x[2]) / v[2];
    const double xe = dt != 0.0 ? dadd(dadd(x[0], dmul(v[0], dt)), dmul(dmul(a[0], dmul(dt, dt)), 0.5)) : x[0];
    note(dadd(xe, -x1)); note(dadd(xe, -x2));
    if (!(x1 < xe && xe < x2)) {
      if (v[0] < 0) dt = (x1 - x[0]) / v[0];
      else if (v[0] > 0) dt = (x2 - x[0]) / v[0];
      update(dt, P);
      return true;
    }
    update(dt, P);
    return false;
  }
  // Honeycomb test at the plane just reached (meshes.py:98-116): cell = the
  // nearest centre, looked up while it is None or 0 (`if not idx`); lost when
  // outside that cell's hexagon, |dx| < R sqrt(3)/2 and |dy| < R - |dx|/sqrt(3).
  // Margins: half the gap between nearest and second-nearest centre, and the
  // nearer hexagon side.
  __device__ bool honeycomb_out(const Plan& P, int i, int& cell) {
    const ctraj_element& e = P.el[i];
    const TableD& T = P.td[e.table];
    if (cell <= 0) {
      double best, second;
      cell = mesh_nearest64(T, e.p, x[0], x[1], best, second);
      note(dadd(second, -best) / 2.0);
    }
    const double s3 = __dsqrt_rn(3.0), R = e.p[0];
    const double dx = fabs(dadd(x[0], -__ldg(T.knots + cell))), dy = fabs(dadd(x[1], -__ldg(T.values + cell)));
    const double hw = dmul(R, s3) / 2.0, q = __ddiv_rn(dx, s3);
    const double side = dadd(hw, -dx), slant = dmul(dadd(dadd(R, -q), -dy), s3 / 2.0);
    note(side < slant ? side : slant);
    return !(dx < hw && dy < dadd(R, -q));
  }

  __device__ bool lens_entrance_out(const Plan& P, int i) { return circle_out(P, i); }

  __device__ double vel_z() const { return v[2]; }

  // One reference RK4 step (electrostatic_lens.py:91-118); returns true when lost.
  __device__ bool lens_step(const Plan& P, int i, const LensStep& s, int& range, int& err) {
    const ctraj_element& e = P.el[i];
    const double dt = s.dt;
    const bool classic = e.scheme == CTRAJ_RK4_CLASSIC;
    double k1[3], l1[3], k2[3], l2[3], k3[3], l3[3], k4[3], l4[3], p[3];
    for (int k = 0; k < 3; ++k) k1[k] = v[k];
    lens_force64(P, e, x[0], x[1], l1[0], l1[1], range, err);
    l1[2] = 0.0;
    for (int k = 0; k < 3; ++k) {
      k2[k] = dadd(k1[k], dmul(dmul(dt, l1[k]), 0.5));
      p[k] = classic ? dadd(x[k], dmul(dmul(dt, k1[k]), 0.5)) : dadd(x[k], dmul(dt, k1[k]));
    }
    lens_force64(P, e, p[0], p[1], l2[0], l2[1], range, err);
    l2[2] = 0.0;
    for (int k = 0; k < 3; ++k) {
      k3[k] = dadd(k1[k], dmul(dmul(dt, l2[k]), 0.5));
      p[k] = dadd(x[k], dmul(dmul(dt, k2[k]), 0.5));
    }
    lens_force64(P, e, p[0], p[1], l3[0], l3[1], range, err);
    l3[2] = 0.0;
    for (int k = 0; k < 3; ++k) {
      k4[k] = dadd(k1[k], dmul(dt, l3[k]));
      p[k] = dadd(x[k], dmul(dt, k3[k]));
    }
    lens_force64(P, e, p[0], p[1], l4[0], l4[1], range, err);
    l4[2] = 0.0;
    for (int k = 0; k < 3; ++k) {
      const double sk = dadd(dadd(dadd(k1[k], dmul(2.0, k2[k])), dmul(2.0, k3[k])), k4[k]);
      const double sl = dadd(dadd(dadd(l1[k], dmul(2.0, l2[k])), dmul(2.0, l3[k])), l4[k]);
      x[k] = dadd(x[k], dmul(dt, sk) / 6.0);
      v[k] = dadd(k1[k], dmul(dt, sl) / 6.0);
      a[k] = l1[k];
    }
    t = dadd(t, dt);
    rows += isfinite(t) ? 1 : 0;
    row_out();
    if (err) return true;
    const double r = rho(), h = dmul(e.p[0], 0.5);
    note(dadd(r, -h));
    return r > h;
  }

  __device__ void lens_begin(const Plan&, int, const LensStep&) {}
  __device__ void lens_row(const Plan&, int, const LensStep&) {}
  // After the last step: the exit snap with the stored acceleration l1
  // (electrostatic_lens.py:74-77) unless the molecule was lost inside.
  __device__ void lens_end(const Plan& P, int i, const LensStep&, bool lost) {
    if (!lost) fly(P, i, 1);
  }

  __device__ void final_row(double* f, int64_t i, int64_t n) const {
    const double vals[10] = {x[0], x[1], x[2], v[0], v[1], v[2], a[0], a[1], a[2], t};
    for (int k = 0; k < 10; ++k) f[size_t(k) * size_t(n) + size_t(i)] = vals[k];
  }
  __device__ void flush_last() {
    if (kRec && !sink->last_written) sink->write(x[0], x[1], x[2], v[0], v[1], v[2], a[0], a[1], a[2], t);
  }

  __device__ void store(const Queue& Q, unsigned s, const LensStep& st) const {
    Q.dx[s] = x[0]; Q.dy[s] = x[1]; Q.dz[s] = x[2];
    Q.dvx[s] = v[0]; Q.dvy[s] = v[1]; Q.dvz[s] = v[2];
    Q.dt[s] = t; Q.margin[s] = margin; Q.rows[s] = rows; Q.id[s] = id;
    Q.lens_dt[s] = st.dt; Q.n_done[s] = int32_t(st.n_done); Q.n_total[s] = int32_t(st.n_total);
  }
  // The stored acceleration is not carried: the next RK4 step recomputes it.
  __device__ void load_state(const Queue& Q, unsigned s, const Plan& P, LensStep& st) {
    x[0] = Q.dx[s]; x[1] = Q.dy[s]; x[2] = Q.dz[s];
    v[0] = Q.dvx[s]; v[1] = Q.dvy[s]; v[2] = Q.dvz[s];
    t = Q.dt[s]; margin = Q.margin[s]; rows = Q.rows[s]; id = Q.id[s];
    a[0] = 0.0; a[1] = -P.g; a[2] = 0.0;
    st.dt = Q.lens_dt[s]; st.n_done = Q.n_done[s]; st.n_total = Q.n_total[s];
  }
  __device__ void load_vz(const Queue&, unsigned) {}
  __device__ void load_rest(const Queue&, unsigned, LensStep&, bool) {}
  static constexpr bool kDeferLensSetup = false;
};

// ===========================================================================
// FP32 fast path
// ===========================================================================
template <bool kOut, bool kRec>
struct Mol32 {
  float x, y, vx, vy, vz, inv_vz, t;
  float gap0;     // first flight length (from the initial z)
  float margin;
  int rows;
  int32_t id;
  double zc;      // current z, kept only for outputs / recording
  float ax, ay;   // stored acceleration (recording)
  float cx, cy, cvx, cvy;  // rounding errors carried by the lens integration
  RowSink* sink;

  __device__ void row_out() {
    if (kRec) sink->put(x, y, zc, vx, vy, vz, ax, ay, 0.0, t);
  }

  __device__ void init(const Plan& P, const RunDev& R, int64_t i) {
    id = int32_t(i);
    margin = INFINITY;
    rows = 0;
    double z_ic;
    if (R.ic_mode == CTRAJ_IC_DEVICE_DRAW) {
      const Words8 w = molecule_words(R.offset + uint64_t(i), R.key);
      float2 n02, n13;
      float n4, n5;
      box_muller_pair(make_uint2(w.w[0], w.w[2]), make_uint2(w.w[1], w.w[3]), n02, n13);
      box_muller(w.w[4], w.w[5], n4, n5);
      vx = __fmaf_rn(R.vf[1], n02.x, R.vf[0]);
      vy = __fmaf_rn(R.vf[3], n13.x, R.vf[2]);
      vz = __fmaf_rn(R.vf[5], n02.y, R.vf[4]);
      if (R.xd.kind == CTRAJ_DIST_DISC_POSITION) {
        float s, c;
        sincospif(2.0f * u01f(w.w[6]), &s, &c);
        const float rr = __fmul_rn(sqrtf(u01f(w.w[7])), R.xf[0]);
        x = __fmul_rn(rr, c);
        y = __fmul_rn(rr, s);
        z_ic = R.xd.p[1];
      } else {
        x = __fmul_rn(R.xf[0], n13.y);
        y = __fmul_rn(R.xf[1], n4);
        z_ic = R.xd.p[2];
      }
      gap0 = R.gap0f;
    } else {
      const size_t n = size_t(R.n);
      x = float(R.ics[size_t(i)]);
      y = float(R.ics[n + size_t(i)]);
      z_ic = R.ics[2 * n + size_t(i)];
      vx = float(R.ics[3 * n + size_t(i)]);
      vy = float(R.ics[4 * n + size_t(i)]);
      vz = float(R.ics[5 * n + size_t(i)]);
      gap0 = P.n_el > 0 ? float(P.el[0].z0 - z_ic) : 0.0f;
    }
    inv_vz = __frcp_rn(vz);
    t = 0.0f;
    ax = 0.0f;
    ay = -P.gf;
    if (kOut || kRec) zc = z_ic;
    if (kRec) sink->write(x, y, zc, vx, vy, vz, ax, ay, 0.0, t);
  }

  // The device draw of init in two parts, for the front's screening of
  // element 0 (FP32 runs without per-molecule outputs, Gaussian positions):
  // screen_draw: the first Philox call's words, vx, vy, vz and x exactly as
  // init draws them; screen_rest: the second call (y) and the rest of init.
  static constexpr bool kScreenable = !kOut && !kRec;
  __device__ void screen_draw(const RunDev& R, int64_t i) {
    const Philox4 a = philox4x32_10(R.offset + uint64_t(i), 0u, R.key);
    float2 n02, n13;
    box_muller_pair(make_uint2(a.v[0], a.v[2]), make_uint2(a.v[1], a.v[3]), n02, n13);
    vx = __fmaf_rn(R.vf[1], n02.x, R.vf[0]);
    vy = __fmaf_rn(R.vf[3], n13.x, R.vf[2]);
    vz = __fmaf_rn(R.vf[5], n02.y, R.vf[4]);
    x = __fmul_rn(R.xf[0], n13.y);
  }
  __device__ void screen_rest(const Plan& P, const RunDev& R, int64_t i) {
    const Philox4 b = philox4x32_10(R.offset + uint64_t(i), 1u, R.key);
    float n4, n5;
    box_muller(b.v[0], b.v[1], n4, n5);
    y = __fmul_rn(R.xf[1], n4);
    id = int32_t(i);
    margin = INFINITY;
    rows = 0;
    gap0 = R.gap0f;
    inv_vz = __frcp_rn(vz);
    t = 0.0f;
    ax = 0.0f;
    ay = -P.gf;
  }
  // True when the walk would stop this molecule (vx, vy, vz, x from
  // screen_draw) at the entrance plane of element 0, a circular or rectangular
  // aperture, whatever its y, which is at most 7 sigma (a normal is at most
  // sqrt(66 ln 2) = 6.764): x' = fma(vx, dt, x) is the walk's, and its |y'| is
  // at least w = |vy dt| - g dt^2 / 2 - 7 sigma, taken low by more than the
  // roundings.  So fma(w, w, x'^2) > R^2 (w no less than 0) makes the walk's
  // fma(y', y', x'^2) > R^2 (the rounding is monotone), and x' outside (x1, x2)
  // or w above |y1| and |y2| fails the rectangle.  |dt| < dt_max keeps all of
  // it finite; otherwise the molecule is not screened.  The molecule then has
  // the walk's one trajectory row.  By x' alone 15 % of the lens beamline's molecules were
  // left to walk, with w 5 %: the front of 1e7 molecules 108 -> 96 us.
  struct Screen {
    bool circle;
    float limit;          // R^2 or max(|y1|, |y2|)
    float y_max, half_g;  // 7 sigma, |g| / 2 (1 + 1e-5)
    float dt_max;
  };
  static __device__ Screen screen(const Plan& P, const RunDev& R) {
    const float g = fabsf(P.gf), v = fabsf(R.vf[2]) + 7.0f * fabsf(R.vf[3]);  // |vy| <= v
    const float* c = P.ef[0].c;
    Screen s;
    s.circle = P.el[0].type == CTRAJ_CIRCULAR_APERTURE;
    s.limit = s.circle ? c[0] : fmaxf(fabsf(c[2]), fabsf(c[3]));
    s.y_max = 7.0f * fabsf(R.xf[1]);
    s.half_g = 0.500005f * g;
    s.dt_max = g < 1e30f && v < 1e15f ? sqrtf(1e30f / fmaxf(g, 100.0f)) : 0.0f;
    return s;
  }
  __device__ bool screened_out(const Plan& P, const float gap0f, const Screen& s) const {
    const float dt = __fmul_rn(gap0f, __frcp_rn(vz));  // the walk's first flight (fly, element 0)
    const float xe = __fmaf_rn(vx, dt, x);             // the walk adds 0 h
    const float w = fmaxf(
        __fmaf_rn(fabsf(__fmul_rn(vy, dt)), 0.99999f, -__fmaf_rn(__fmul_rn(dt, dt), s.half_g, s.y_max)), 0.0f);
    const float* c = P.ef[0].c;
    const bool out = s.circle ? __fmaf_rn(w, w, __fmul_rn(xe, xe)) > s.limit
                              : !(c[0] < xe && xe < c[1]) || w > s.limit;
    return out && fabsf(dt) < s.dt_max;
  }

  // ballistic flight of dt with stored acceleration (ax, ay); afterwards a = (0, -g)
  __device__ void flight(float dt, const Plan& P) {
    const float h = __fmul_rn(__fmul_rn(0.5f, dt), dt);
    x = __fmaf_rn(ax, h, __fmaf_rn(vx, dt, x));
    y = __fmaf_rn(ay, h, __fmaf_rn(vy, dt, y));
    vx = __fmaf_rn(ax, dt, vx);
    vy = __fmaf_rn(ay, dt, vy);
    t = __fadd_rn(t, dt);
    ax = 0.0f;
    ay = -P.gf;
    rows += isfinite(t) ? 1 : 0;
  }

  __device__ void fly(const Plan& P, int i, int which) {
    const float gap = which ? P.ef[i].len : (i == 0 ? gap0 : P.ef[i].gap);
    flight(__fmul_rn(gap, inv_vz), P);
    if (kOut || kRec) zc = which ? P.el[i].z1 : P.el[i].z0;
    row_out();
  }

  __device__ void note(float d) {
    if (kOut) margin = fminf(margin, fabsf(d));
  }

  __device__ bool circle_out(const Plan& P, int i) {
    const float r2 = __fmaf_rn(y, y, __fmul_rn(x, x));
    if (kOut) note(__fadd_rn(sqrtf(r2), -P.ef[i].c[1]));
    return r2 > P.ef[i].c[0];
  }
  __device__ bool rect_out(const Plan& P, int i) {
    const float* c = P.ef[i].c;
    if (kOut) { note(x - c[0]); note(x - c[1]); note(y - c[2]); note(y - c[3]); }
    return !((c[0] < x && x < c[1]) && (c[2] < y && y < c[3]));
  }
  __device__ bool plates(const Plan& P, int i) {
    const float x1 = P.ef[i].c[0], x2 = P.ef[i].c[1];
    if (kOut) { note(x - x1); note(x - x2); }
    if (!(x1 < x && x < x2)) return true;
    float dt = __fmul_rn(P.ef[i].len, inv_vz);
    const float xe = __fmaf_rn(vx, dt, x);  // a_x = 0 after a ballistic flight
    if (kOut) { note(xe - x1); note(xe - x2); }
    if (!(x1 < xe && xe < x2)) {
      if (vx < 0.0f) dt = __fdiv_rn(x1 - x, vx);
      else if (vx > 0.0f) dt = __fdiv_rn(x2 - x, vx);
      flight(dt, P);
      if (kOut || kRec) zc += double(dt) * double(vz);
      row_out();
      return true;
    }
    flight(dt, P);
    if (kOut || kRec) zc = P.el[i].z1;
    row_out();
    return false;
  }
  // Honeycomb (meshes.py:98-116) on the float centre table; ef c[0] = R sqrt(3)/2,
  // c[1] = R.
  __device__ bool honeycomb_out(const Plan& P, int i, int& cell) {
    const LensF& L = P.lf[i];
    const float* c = P.ef[i].c;
    if (cell <= 0) {
      float best2, second2;
      cell = mesh_nearest32(L, P.ef[i], x, y, best2, second2);
      if (kOut) note(0.5f * (sqrtf(second2) - sqrtf(best2)));
    }
    const float4 q = __ldg(L.q + cell);
    const float dx = fabsf(x - q.x), dy = fabsf(y - q.y);
    const float lim = __fmaf_rn(-0.57735026919f, dx, c[1]);
    if (kOut) note(fminf(c[0] - dx, 0.8660254038f * (lim - dy)));
    return !(dx < c[0] && dy < lim);
  }
  __device__ bool lens_entrance_out(const Plan& P, int i) { return circle_out(P, i); }

  __device__ double vel_z() const { return double(vz); }

  // One step, table-coordinate scale beta; kScaled (batched sweeps): the table
  // holds the unscaled polynomial and the molecule brings its configuration's
  // force scale kappa.  r2 is the squared radius of (x, y) on entry and of the
  // new position on return; the molecule is lost when that exceeds bore2.
  // The stage pairs are packed (a stage per component), the position and
  // velocity updates by (x, y); per component each operation is the scalar
  // one.  Increments are formed in full precision, then added once with the
  // carried rounding error (the lens defocuses, so uncompensated rounding of x
  // and v grows to micrometres at the detector).  Stages (4, 3) in this order
  // make l1 + l4 and l2 + l3 one packed addition.
  // Linear form, run in groups without a bore test in between (persist_pass): a
  // warp alone on its scheduler takes 229 cycles (292 with (x, y) packed
  // throughout and the bore tested between steps), 33.6 instead of 35.4 per SM
  // at 16 warps, 30.3 instead of 32.0 at 32.
  struct StagePair {
    float2 X, Y, Lx, Ly;  // stage points and accelerations, one stage per component
  };
  __device__ __forceinline__ void pair_begin(const float c2, StagePair& a) const {
    a.X = pack2(x, __fmaf_rn(c2, vx, x));
    a.Y = pack2(y, __fmaf_rn(c2, vy, y));
  }
  __device__ __forceinline__ void pair_force(const float2 w, const float g, StagePair& a) const {
    a.Lx = __ffma2_rn(w, a.X, pack2(0.0f, 0.0f));
    a.Ly = __ffma2_rn(w, a.Y, pack2(-g, -g));
  }
  // the points of stages 4 and 3 from the accelerations of stages 1 and 2; their squared radii
  __device__ __forceinline__ float2 pair_middle(const float dt, const float hdt, const StagePair& a, StagePair& b) const {
    const float k2x = __fmaf_rn(hdt, a.Lx.x, vx), k2y = __fmaf_rn(hdt, a.Ly.x, vy);
    const float k3x = __fmaf_rn(hdt, a.Lx.y, vx), k3y = __fmaf_rn(hdt, a.Ly.y, vy);
    b.X = pack2(__fmaf_rn(dt, k3x, x), __fmaf_rn(hdt, k2x, x));
    b.Y = pack2(__fmaf_rn(dt, k3y, y), __fmaf_rn(hdt, k2y, y));
    return __ffma2_rn(b.Y, b.Y, __fmul2_rn(b.X, b.X));
  }
  __device__ __forceinline__ void pair_end(const float dt, const float dt6, const float dt26, const StagePair& a,
                                          const StagePair& b, float& r2) {
    const float2 sum = pack2(__fadd_rn(__fadd_rn(a.Lx.x, a.Lx.y), b.Lx.y), __fadd_rn(__fadd_rn(a.Ly.x, a.Ly.y), b.Ly.y));
    const float2 dx = __ffma2_rn(pack2(dt26, dt26), sum, __fmul2_rn(pack2(dt, dt), pack2(vx, vy)));
    const float2 ux = __fadd2_rn(a.Lx, b.Lx), uy = __fadd2_rn(a.Ly, b.Ly);  // (l1 + l4, l2 + l3)
    const float2 dv = __fmul2_rn(pack2(dt6, dt6), pack2(__fmaf_rn(2.0f, ux.y, ux.x), __fmaf_rn(2.0f, uy.y, uy.x)));
    add_carried(dx, dv);
    ax = a.Lx.x;
    ay = a.Ly.x;
    r2 = __fmaf_rn(y, y, __fmul_rn(x, x));
  }
  // s += inc with the rounding error carried in c (Fast2Sum: |s| >= |inc + c|
  // holds because one step changes x and v by far less than their size)
  __device__ __forceinline__ void add_carried(const float2 dx, const float2 dv) {
    const float2 p = pack2(x, y), v = pack2(vx, vy);
    float2 cp = pack2(cx, cy), cv = pack2(cvx, cvy);
    const float2 d1 = __fadd2_rn(dx, cp), t1 = __fadd2_rn(p, d1);
    cp = __fadd2_rn(d1, neg2(__fadd2_rn(t1, neg2(p))));
    const float2 d2 = __fadd2_rn(dv, cv), t2 = __fadd2_rn(v, d2);
    cv = __fadd2_rn(d2, neg2(__fadd2_rn(t2, neg2(v))));
    x = t1.x;
    y = t1.y;
    vx = t2.x;
    vy = t2.y;
    cx = cp.x;
    cy = cp.y;
    cvx = cv.x;
    cvy = cv.y;
  }
  template <int F, bool kStaged, bool kScaled, bool kFast>
  __device__ __forceinline__ void lens_step_pair(const LensArgs& L, const PairTable& T, const float dt, const float hdt,
                                                 const float c2, const float dt6, const float dt26, float& r2,
                                                 unsigned& flags, const float beta, const float kappa) {
    StagePair a, b;
    pair_begin(c2, a);
    const float2 q12 = pack2(r2, __fmaf_rn(a.Y.y, a.Y.y, __fmul_rn(a.X.y, a.X.y)));
    float2 w = force_pair<F, kStaged, kFast>(L, T, q12, beta, flags);
    pair_force(kScaled ? __fmul2_rn(pack2(kappa, kappa), w) : w, L.g, a);
    const float2 q43 = pair_middle(dt, hdt, a, b);
    w = force_pair<F, kStaged, kFast>(L, T, q43, beta, flags);
    pair_force(kScaled ? __fmul2_rn(pack2(kappa, kappa), w) : w, L.g, b);
    pair_end(dt, dt6, dt26, a, b, r2);
  }
  // The linear form's step with the pieces in q, loaded during the step before,
  // so that no lookup waits for its address: 176 cycles for a warp alone.
  // `bad` collects the offsets in their pieces as unsigned words: one not in
  // [0, 1) -- at or above 0x3f800000 -- means a piece was not the lookup's and
  // the state is not the step's (0.02 % of the pieces: the coordinates' rounding
  // makes the extrapolation uncertain by about 2 ulp.  A fading-memory filter
  // instead missed a third of that and took as long, for its own instructions).
  template <bool kScaled>
  __device__ __forceinline__ void lens_step_ahead(const LensArgs& L, const PairTable& T, const float dt, const float hdt,
                                                  const float c2, const float dt6, const float dt26, LinAhead& q,
                                                  float& r2, unsigned& bad, const float beta, const float kappa) {
    StagePair a, b;
    pair_begin(c2, a);
    const float2 B = pack2(beta, beta), S0 = pack2(-L.s0, -L.s0);
    const float2 s = __ffma2_rn(B, pack2(r2, __fmaf_rn(a.Y.y, a.Y.y, __fmul_rn(a.X.y, a.X.y))), S0);
    const float2 u = __fadd2_rn(s, neg2(q.k12));
    float2 w = pack2(__fmaf_rn(u.x, q.e1.y, q.e1.x), __fmaf_rn(u.y, q.e2.y, q.e2.x));
    pair_force(kScaled ? __fmul2_rn(pack2(kappa, kappa), w) : w, L.g, a);
    const float2 s4 = __ffma2_rn(B, pair_middle(dt, hdt, a, b), S0);
    const float2 u4 = __fadd2_rn(s4, neg2(q.k43));
    w = pack2(__fmaf_rn(u4.x, q.e4.y, q.e4.x), __fmaf_rn(u4.y, q.e3.y, q.e3.x));
    bad = max(max(bad, max(__float_as_uint(u.x), __float_as_uint(u.y))),
              max(__float_as_uint(u4.x), __float_as_uint(u4.y)));
    const float2 p12 = LinAhead::next(s, q.s12, q.d12), p43 = LinAhead::next(s4, q.s43, q.d43);
    q.load(T, p12, p43);
    pair_force(kScaled ? __fmul2_rn(pack2(kappa, kappa), w) : w, L.g, b);
    pair_end(dt, dt6, dt26, a, b, r2);
  }

  // The quadratic form's step with one force after the other and (x, y) packed
  // throughout: the same values as lens_step_pair in fewer instructions (the
  // interval by the conversion unit, which runs beside the others), but with its
  // lookups on one chain.  For passes whose SMs are full (persist_pass).
  template <bool kStaged, bool kScaled>
  __device__ __forceinline__ void lens_step_xy(const LensArgs& L, const float4* tab, const float dt, const float hdt,
                                               const float c2, const float dt6, const float dt26, float& r2,
                                               const float beta, const float kappa) {
    auto force = [&](const float2 p, const float q2) {
      const float s = __fmaf_rn(beta, q2, -L.s0);
      const unsigned i = min(__float2uint_rz(s), unsigned(L.n_int - 1));  // negative s and NaN -> 0
      const float u = __fadd_rn(s, -__uint2float_rn(i));
      const float4 q = kStaged ? tab[i] : __ldg(tab + i);
      const float w = __fmaf_rn(u, __fmaf_rn(u, q.z, q.y), q.x), k = kScaled ? __fmul_rn(kappa, w) : w;
      return __ffma2_rn(pack2(k, k), p, pack2(0.0f, -L.g));
    };
    auto radius2 = [](const float2 p) { return __fmaf_rn(p.y, p.y, __fmul_rn(p.x, p.x)); };
    const float2 p = pack2(x, y), v = pack2(vx, vy), Hdt = pack2(hdt, hdt), Dt = pack2(dt, dt);
    const float2 l1 = force(p, r2), k2 = __ffma2_rn(Hdt, l1, v), p2 = __ffma2_rn(pack2(c2, c2), v, p);
    const float2 l2 = force(p2, radius2(p2)), k3 = __ffma2_rn(Hdt, l2, v), p3 = __ffma2_rn(Hdt, k2, p);
    const float2 l3 = force(p3, radius2(p3)), p4 = __ffma2_rn(Dt, k3, p), l4 = force(p4, radius2(p4));
    const float2 sum = __fadd2_rn(__fadd2_rn(l1, l2), l3);
    const float2 dx = __ffma2_rn(pack2(dt26, dt26), sum, __fmul2_rn(Dt, v));
    const float2 dv = __fmul2_rn(pack2(dt6, dt6), __ffma2_rn(pack2(2.0f, 2.0f), __fadd2_rn(l2, l3), __fadd2_rn(l1, l4)));
    add_carried(dx, dv);
    ax = l1.x;
    ay = l1.y;
    r2 = __fmaf_rn(y, y, __fmul_rn(x, x));
  }

  // One step looked at by itself; true when the molecule left the bore.  Without
  // kScaled the coordinate scale comes from L and kappa is folded into the table.
  template <int F, bool kStaged, bool kScaled = false>
  __device__ bool lens_step(const LensArgs& L, const float dt, const float hdt, const float c2,
                            const float dt6, const float dt26, const float4* s_tab, unsigned& flags,
                            const float beta = 0.0f, const float kappa = 1.0f) {
    float r2 = __fmaf_rn(y, y, __fmul_rn(x, x));
    if constexpr (F == kForceStark2)
      lens_step_xy<kStaged, kScaled>(L, kStaged ? s_tab : L.q, dt, hdt, c2, dt6, dt26, r2, kScaled ? beta : L.beta, kappa);
    else
      lens_step_pair<F, kStaged, kScaled, false>(L, pair_table<F>(L, kStaged ? s_tab : L.q), dt, hdt, c2, dt6, dt26, r2,
                                                 flags, kScaled ? beta : L.beta, kappa);
    if (kOut) note(__fadd_rn(sqrtf(r2), -L.bore));
    return r2 > L.bore2;
  }

  // Inside the lens t keeps the entrance time and z is not tracked: both
  // follow from the step count (t + n dt, z0 + n dz) instead of being
  // accumulated in float.
  __device__ void lens_begin(const Plan&, int, const LensStep&) { cx = cy = cvx = cvy = 0.0f; }
  __device__ double lens_dz(const ctraj_element& e) const {
    return e.step_mode == CTRAJ_STEP_DT ? dmul(double(vz), e.p[2]) : e.p[1];
  }
  __device__ void lens_row(const Plan& P, int i, const LensStep& s) {
    if (kRec) {
      zc = P.el[i].z0 + double(s.n_done) * lens_dz(P.el[i]);
      sink->put(x, y, zc, vx, vy, vz, ax, ay, 0.0, double(t) + double(s.n_done) * s.dt);
    }
  }
  // After the last step: t from the step count, then the exit snap of
  // (z1 - z0 - N dz) / vz with the stored acceleration l1 unless lost inside.
  __device__ void lens_end(const Plan& P, int i, const LensStep& s, bool lost) {
    t = float(double(t) + double(s.n_done) * s.dt);
    rows += int(s.n_done);
    x = __fadd_rn(x, cx);
    y = __fadd_rn(y, cy);
    vx = __fadd_rn(vx, cvx);
    vy = __fadd_rn(vy, cvy);
    if (kOut || kRec) zc = P.el[i].z0 + double(s.n_done) * lens_dz(P.el[i]);
    if (lost) return;
    flight(float(s.snap), P);
    if (kOut || kRec) zc = P.el[i].z1;
    row_out();
  }

  __device__ void final_row(double* f, int64_t i, int64_t n) const {
    const double vals[10] = {x, y, zc, vx, vy, vz, ax, ay, 0.0, t};
    for (int k = 0; k < 10; ++k) f[size_t(k) * size_t(n) + size_t(i)] = vals[k];
  }
  __device__ void flush_last() {
    if (kRec && !sink->last_written) sink->write(x, y, zc, vx, vy, vz, ax, ay, 0.0, t);
  }

  __device__ void store(const Queue& Q, unsigned s, const LensStep& st) const {
    Q.x[s] = x; Q.y[s] = y; Q.vx[s] = vx; Q.vy[s] = vy; Q.vz[s] = vz; Q.t[s] = t;
    Q.cx[s] = cx; Q.cy[s] = cy; Q.cvx[s] = cvx; Q.cvy[s] = cvy;
    Q.lens_dt[s] = st.dt; Q.snap[s] = float(st.snap);
    Q.n_done[s] = int32_t(st.n_done); Q.n_total[s] = int32_t(st.n_total);
    Q.rows[s] = rows; Q.id[s] = id;
    if (kOut) Q.margin[s] = margin;
  }
  // What the RK4 loop needs; the stored acceleration is not carried (the next
  // RK4 step recomputes it).
  __device__ void load_state(const Queue& Q, unsigned s, const Plan& P, LensStep& st) {
    x = Q.x[s]; y = Q.y[s]; vx = Q.vx[s]; vy = Q.vy[s];
    cx = Q.cx[s]; cy = Q.cy[s]; cvx = Q.cvx[s]; cvy = Q.cvy[s];
    st.dt = Q.lens_dt[s];
    st.n_done = Q.n_done[s]; st.n_total = Q.n_total[s];
    ax = 0.0f;
    ay = -P.gf;
    margin = INFINITY;  // edges seen during this chunk; merged with the queued value below
  }
  __device__ void load_vz(const Queue& Q, unsigned s) { vz = Q.vz[s]; }
  static constexpr bool kDeferLensSetup = true;
  // The rest, read after the RK4 loop so it does not occupy registers during
  // it (the exit-snap time too, unless the setup was just done in this chunk).
  __device__ void load_rest(const Queue& Q, unsigned s, LensStep& st, bool snap_from_queue) {
    vz = Q.vz[s];
    t = Q.t[s];
    if (snap_from_queue) st.snap = double(Q.snap[s]);
    rows = Q.rows[s];
    id = Q.id[s];
    inv_vz = __frcp_rn(vz);
    if (kOut) margin = fminf(margin, float(Q.margin[s]));
  }
};

// ---------------------------------------------------------------------------
// Element walk shared by both precisions (beamline.py:20-38).  Starts at
// element `from`; returns the counter slot of the element the molecule was
// lost on, kLabelDetected when it leaves the beamline, or kQueued when it
// passed the entrance of the lens at element index *lens_at.
// ---------------------------------------------------------------------------
template <class M>
__device__ int walk(M& m, const Plan& P, int from, int* lens_at) {
  for (int i = from; i < P.n_el; ++i) {
    const ctraj_element& e = P.el[i];
    switch (e.type) {
      case CTRAJ_CIRCULAR_APERTURE:
        m.fly(P, i, 0);
        if (m.circle_out(P, i)) return e.label;
        m.fly(P, i, 1);
        if (m.circle_out(P, i)) return e.label;
        break;
      case CTRAJ_RECTANGULAR_APERTURE:
        m.fly(P, i, 0);
        if (m.rect_out(P, i)) return e.label;
        m.fly(P, i, 1);
        if (m.rect_out(P, i)) return e.label;
        break;
      case CTRAJ_FIELD_PLATES:
        m.fly(P, i, 0);
        if (m.plates(P, i)) return e.label;
        break;
      case CTRAJ_HONEYCOMB: {
        int cell = -1;  // None
        m.fly(P, i, 0);
        if (m.honeycomb_out(P, i, cell)) return e.label;
        m.fly(P, i, 1);
        if (m.honeycomb_out(P, i, cell)) return e.label;
        break;
      }
      case CTRAJ_ELECTROSTATIC_LENS:
        m.fly(P, i, 0);
        *lens_at = i;  // also reported for a loss at the entrance test
        if (m.lens_entrance_out(P, i)) return e.label;
        return kQueued;
      default:
        return e.label;
    }
  }
  return kLabelDetected;
}

}  // namespace ctraj
