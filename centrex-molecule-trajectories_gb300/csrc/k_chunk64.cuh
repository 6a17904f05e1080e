// The exact-mode (FP64) lens pass: k_lens_chunk64, the reference's RK4 step in
// the reference's operation order (Mol64::lens_step, bit for bit) with the
// FP64 instruction count cut to what the rounding of the result needs.
//
// Bound: the FP64 pipe (fp64.cuh: 64 cycles of a scheduler's pipe per warp
// instruction, 19 per SM when all four pipes are busy).  Mol64::lens_step
// issues 421 FP64 instructions per warp and step, the step here 222 (counted by
// ncu; all in the pipe, comparisons and conversions too):
//  * square roots and quotients from fp64.cuh, the square root's reciprocal
//    serving both components;
//  * x + (dt v) / 2 and a + 2 b as one FMA (the scaling is exact, so the FMA
//    rounds the same sum);
//  * a_z = 0: z gains the same increment every step, computed once;
//  * the bore test of a step uses the square root of the next step's first
//    stage (the same r), and the margin keeps the largest r (rounding is
//    monotone, so the smallest |r - R| inside the bore is at the largest r);
//  * comparisons, table intervals and range tests on the integer and FP32
//    pipes (a guessed interval is corrected against the knots, so the interval
//    is the reference's).
// A step in which a form is not sure of its rounding (2e-5 of the quotients and
// roots), r = 0 or a lookup is outside the table (with one lane per molecule: a
// radial table) is redone by Mol64::lens_step.
//
// kQuad: four lanes per molecule, (stages 1 and 3 | stages 2 and 4) x (x | y):
// stage 2 does not depend on stage 1, nor stage 4 on stage 3, so two force
// evaluations follow one another instead of four, and each component has its
// own lane: 87 FP64 instructions per step, at 4 x the warps.  A warp
// instruction costs the same for any number of lanes, so this is the shorter
// way while the warps fit the schedulers (quad_max); beyond, one lane per
// molecule does the least work in total.
//
// Measured (lens beamline, GB300; Mol64::lens_step in 512-thread CTAs before):
// 1e5 molecules 103 -> 15.0 ms (the longest stay's ~4 000 steps at 3.8 us;
// 15.8 with the table's records read through L2 instead of shared memory),
// 1e6 molecules 122 -> 21 ms, 3e6 130 -> 40 ms (1.1e9 steps/s).
#pragma once
#include "engine.h"
#include "fp64.cuh"
#include "kernels.cuh"

namespace ctraj {

constexpr int kLens64Threads = 256;  // one CTA per SM beside its staged table, two warps per scheduler

constexpr size_t kLens64Staged = 200 * 1024;  // bytes of records a CTA stages at most

// Lens constants of k_lens_chunk64 (built by launch_chunk64).
struct Lens64 {
  // per interval: (knot, c0, c1, c2) of the spline, or (knot, value, slope, 0)
  // of a radial table; the record after the last holds the last knot
  const double2* rec;
  int staged;          // the records fit in shared memory
  double first, last;  // the knots' ends
  double alpha, alpha2;  // |E| = alpha r^n; 2 alpha
  double mass, inv_mass;
  float x0, inv_h;     // interval guess
  int n;               // intervals
};

// a_r of lens_force64 at radius r; false when the plain path has to decide.
// kExtend: a spline's end pieces are extrapolated here, as PPoly does, and
// `outside` is set.  With one lane per molecule the SMs are full, and a molecule
// outside its table taking every step twice made the pass slower than
// k_lens_chunk (74 000 molecules through 300 steps of a lens whose table begins
// 2.4 mm off the axis: 14.2 ms there, 17.6 with the steps taken again, 8.8 so).
// With four lanes taking them again still is the faster one (9.9 -> 5.6 ms), and
// the steps inside the table are 1.4 % faster without the code for it.
template <int F, bool kExtend>
__device__ __forceinline__ bool accel64(const Lens64& L, const double2* rec, const double r, double& ar, bool& outside) {
  const double E = F == kForceRadial ? r : F == kForceStark1 ? __dmul_rn(L.alpha, r)
                                                             : __dmul_rn(L.alpha, __dmul_rn(r, r));
  // r is positive here, hence E is not negative; neither are the knots (records64)
  int j = max(0, min(__float2int_rz((trunc_float(E) - L.x0) * L.inv_h), L.n - 1));
  double2 a, b;
  if (less_pos(E, L.first) || !less_pos(E, L.last)) {
    if (F == kForceRadial || !kExtend) return false;
    const bool below = less_pos(E, L.first);
    j = below ? 0 : L.n - 1;
    a = rec[2 * j];
    b = rec[2 * j + 1];
    outside = outside || below || less_pos(L.last, E);
  } else {
    for (;;) {
      a = rec[2 * j];
      b = rec[2 * j + 1];
      const double next = rec[2 * j + 2].x;
      if (less_pos(E, a.x)) --j;              // stops at j = 0: E >= first
      else if (!less_pos(E, next)) ++j;       // and at n - 1: E < last
      else break;
    }
  }
  const double s = dadd(E, -a.x);
  if (F == kForceRadial) {
    ar = __double_as_longlong(r) == __double_as_longlong(a.x) ? a.y : dadd(dmul(b.x, s), a.y);
    return true;
  }
  double w = __fma_rn(dmul(b.x, s), 2.0, b.y);
  w = dadd(w, dmul(dmul(a.y, dmul(s, s)), 3.0));
  const double num = -dmul(w, F == kForceStark1 ? L.alpha : dmul(L.alpha2, r));
  bool sure;
  ar = div64(num, L.mass, L.inv_mass, sure);
  return sure;
}

// Mol64::lens_step on the values of one molecule; s: x y z vx vy vz t, then
// the stored acceleration (ax, ay).  Returns the table flags (1: outside the
// spline, 2: above a radial table).
static __device__ __noinline__ unsigned plain_step64(const Plan& P, const int li, const double dt, double (&s)[9]) {
  Mol64<false> m;
  LensStep st;
  st.dt = dt;
  m.margin = INFINITY;
  m.rows = 0;
  for (int k = 0; k < 3; ++k) {
    m.x[k] = s[k];
    m.v[k] = s[3 + k];
  }
  m.t = s[6];
  int range = 0, err = 0;
  m.lens_step(P, li, st, range, err);
  for (int k = 0; k < 3; ++k) {
    s[k] = m.x[k];
    s[3 + k] = m.v[k];
  }
  s[6] = m.t;
  s[7] = m.a[0];
  s[8] = m.a[1];
  return (range ? 1u : 0u) | (err ? 2u : 0u);
}

// What a batch's lane carries through the RK4 loop: kQuad: its component's
// x[0], v[0], a[0] and, by stage half, z or t in zt; else all of them.
struct Lane64 {
  double x[2], v[2], a[2], z, t, vz, dt, zinc;
  double rmax, rlost;  // largest radius tested inside the bore, radius where lost (< 0: none)
  int n_done, n_total, phase;
  unsigned flags;
};

// Result of the bore test at radius r (NaN: passes, as r > R is false)
__device__ __forceinline__ void bore_test(Lane64& m, const double r, const bool finite, const double bore) {
  if (m.phase != kRun) return;
  if (finite) {
    if (less_pos(bore, r)) {
      m.rlost = r;
      m.phase = kLost;
    } else if (less_pos(m.rmax, r)) {  // rmax starts below every r
      m.rmax = r;
    }
  }
  if (m.phase == kRun && m.n_done == m.n_total) m.phase = kExit;
}

// Up to `chunk` steps of the warp's molecules, one lane each.
template <int F>
__device__ __forceinline__ void advance_one64(Lane64& m, const Plan& P, const int li, const Lens64& L,
                                              const double2* rec, const double bore, const bool classic, const int chunk) {
  const double c2 = classic ? 0.5 : 1.0;
  for (int k = 0;; ++k) {
    double h, r2 = dadd(dmul(m.x[0], m.x[0]), dmul(m.x[1], m.x[1]));
    bool ok, sure;
    double r = sqrt64(r2, h, ok);
    if (!ok) r = __dsqrt_rn(r2);
    bore_test(m, r, !isnan(r2), bore);
    if (k == chunk || !__any_sync(kFull, m.phase == kRun)) return;
    if (m.phase != kRun) continue;
    bool outside = false;
    // l = the force at p, whose radius is r
    auto force = [&](const double (&p)[2], double (&l)[2]) {
      double ar = 0.0;
      ok = ok && accel64<F, true>(L, rec, r, ar, outside);
      l[0] = div64(dmul(ar, p[0]), r, scale2(h, 1), sure);
      ok = ok && sure;
      l[1] = dadd(div64(dmul(ar, p[1]), r, scale2(h, 1), sure), -P.g);
      ok = ok && sure;
    };
    auto radius = [&](const double (&p)[2]) {
      r = sqrt64(dadd(dmul(p[0], p[0]), dmul(p[1], p[1])), h, sure);
      ok = ok && sure;
    };
    double l1[2], l2[2], l3[2], l4[2], k2[2], k3[2], p[2], x[2], v[2];
    force(m.x, l1);
#pragma unroll
    for (int c = 0; c < 2; ++c) p[c] = __fma_rn(dmul(m.dt, m.v[c]), c2, m.x[c]);
    radius(p);
    force(p, l2);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      k2[c] = __fma_rn(dmul(m.dt, l1[c]), 0.5, m.v[c]);
      p[c] = __fma_rn(dmul(m.dt, k2[c]), 0.5, m.x[c]);
    }
    radius(p);
    force(p, l3);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      k3[c] = __fma_rn(dmul(m.dt, l2[c]), 0.5, m.v[c]);
      p[c] = dadd(m.x[c], dmul(m.dt, k3[c]));
    }
    radius(p);
    force(p, l4);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const double k4 = dadd(m.v[c], dmul(m.dt, l3[c]));
      const double ik = dmul(m.dt, dadd(__fma_rn(2.0, k3[c], __fma_rn(2.0, k2[c], m.v[c])), k4));
      const double il = dmul(m.dt, dadd(__fma_rn(2.0, l3[c], __fma_rn(2.0, l2[c], l1[c])), l4[c]));
      ok = ok && div6_ok(ik) && div6_ok(il);
      x[c] = dadd(m.x[c], div6(ik));
      v[c] = dadd(m.v[c], div6(il));
    }
    if (!ok) {
      double s[9] = {m.x[0], m.x[1], m.z, m.v[0], m.v[1], m.vz, m.t, 0.0, 0.0};
      const unsigned f = plain_step64(P, li, m.dt, s);
      m.x[0] = s[0];
      m.x[1] = s[1];
      m.z = s[2];
      m.v[0] = s[3];
      m.v[1] = s[4];
      m.t = s[6];
      m.a[0] = s[7];
      m.a[1] = s[8];
      m.flags |= f;
      if (f & 2u) m.phase = kLost;
    } else {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        m.x[c] = x[c];
        m.v[c] = v[c];
        m.a[c] = l1[c];
      }
      m.z = dadd(m.z, m.zinc);
      m.t = dadd(m.t, m.dt);
      m.flags |= outside ? 1u : 0u;
    }
    ++m.n_done;
  }
}

// The same with four lanes per molecule: bit 0 of the lane its component,
// bit 1 its half (0: stages 1 and 3, and z; 1: stages 2 and 4, and t).  Every
// lane of the warp runs every step; lanes whose molecule is done keep their
// state.
template <int F>
__device__ __forceinline__ void advance_quad64(Lane64& m, const Plan& P, const int li, const Lens64& L,
                                               const double2* rec, const double bore, const bool classic, const int chunk) {
  const int lane = threadIdx.x & 31, home = lane & ~3;
  const bool half = lane & 2;
  const double c2 = classic ? 0.5 : 1.0, c34 = half ? 1.0 : 0.5;
  const double g = (lane & 1) ? -P.g : -0.0;  // a + (-0.0) is a
  double X = m.x[0], V = m.v[0], zt = half ? m.t : m.z;
  const double zt_inc = half ? m.dt : m.zinc;
  for (int k = 0;; ++k) {
    bool ok = true, sure, outside = false;
    double h, r;
    auto radius = [&](const double p) {
      const double q = dmul(p, p), r2 = dadd(q, __shfl_xor_sync(kFull, q, 1));
      r = sqrt64(r2, h, sure);
      ok = ok && sure;
      return r2;
    };
    auto force = [&](const double p) {
      double ar = 0.0;
      ok = ok && accel64<F, false>(L, rec, r, ar, outside);
      const double l = dadd(div64(dmul(ar, p), r, scale2(h, 1), sure), g);
      ok = ok && sure;
      return l;
    };
    double p = __fma_rn(dmul(m.dt, V), c2, X);
    p = half ? p : X;
    const double r2 = radius(p);
    double rt = r;
    if (!ok) rt = __dsqrt_rn(r2);
    rt = __shfl_sync(kFull, rt, home);  // the radius of the state: the stage-1 lanes'
    bore_test(m, rt, !isnan(rt), bore);
    if (k == chunk || !__any_sync(kFull, m.phase == kRun)) break;
    const double l12 = force(p);
    const double k23 = __fma_rn(dmul(m.dt, l12), 0.5, V);
    p = __fma_rn(dmul(m.dt, k23), c34, X);
    radius(p);
    const double l34 = force(p);
    const double k4 = dadd(V, dmul(m.dt, l34));
    const double k3 = __shfl_xor_sync(kFull, k23, 2), l1 = __shfl_xor_sync(kFull, l12, 2),
                 l3 = __shfl_xor_sync(kFull, l34, 2);
    // stage-1 lanes sum k1 + 2 k2 + 2 k3 + k4, stage-2 lanes l1 + 2 l2 + 2 l3 + l4
    double u = __fma_rn(2.0, half ? l12 : k23, half ? l1 : V);
    u = __fma_rn(2.0, half ? l3 : k3, u);
    const double i6 = dmul(m.dt, dadd(u, half ? l34 : k4));
    ok = ok && div6_ok(i6);
    const double mine = dadd(half ? V : X, div6(i6)), other = __shfl_xor_sync(kFull, mine, 2);
    const bool run = m.phase == kRun;
    const unsigned bad = __ballot_sync(kFull, run && !ok);
    const bool redo = (bad >> home) & 0xfu;
    if (bad) {
      double s[9];
      s[0] = __shfl_sync(kFull, X, home);
      s[1] = __shfl_sync(kFull, X, home + 1);
      s[2] = __shfl_sync(kFull, zt, home);
      s[3] = __shfl_sync(kFull, V, home);
      s[4] = __shfl_sync(kFull, V, home + 1);
      s[5] = m.vz;
      s[6] = __shfl_sync(kFull, zt, home + 2);
      if (redo) {  // every lane of the molecule computes the same step
        const unsigned f = plain_step64(P, li, m.dt, s);
        X = (lane & 1) ? s[1] : s[0];
        V = (lane & 1) ? s[4] : s[3];
        zt = half ? s[6] : s[2];
        m.a[0] = (lane & 1) ? s[8] : s[7];
        m.flags |= f;
        if (f & 2u) m.phase = kLost;
      }
    }
    if (run && !redo) {
      X = half ? other : mine;
      V = half ? mine : other;
      zt = dadd(zt, zt_inc);
      m.a[0] = half ? l1 : l12;
    }
    if (run) ++m.n_done;
  }
  // back to whole molecules, in each lane of the quad
  const double x0 = __shfl_sync(kFull, X, home), x1 = __shfl_sync(kFull, X, home + 1);
  const double v0 = __shfl_sync(kFull, V, home), v1 = __shfl_sync(kFull, V, home + 1);
  const double a0 = __shfl_sync(kFull, m.a[0], home), a1 = __shfl_sync(kFull, m.a[0], home + 1);
  m.z = __shfl_sync(kFull, zt, home);
  m.t = __shfl_sync(kFull, zt, home + 2);
  m.x[0] = x0;
  m.x[1] = x1;
  m.v[0] = v0;
  m.v[1] = v1;
  m.a[0] = a0;
  m.a[1] = a1;
}

// k_lens_chunk for FP64: at most `chunk` steps of every molecule of Qin, those
// still inside appended to Qcont, the others ended here (exit snap, the
// elements behind the lens, tally, or the next lens's queue).  Batches of a
// warp: the first interleaved across CTAs, later ones from a counter.
template <bool kOut, int F>
__global__ void __launch_bounds__(kLens64Threads) k_lens_chunk64(const __grid_constant__ Plan P, const RunDev R,
                                                                 const int li, const Queue Qin, const Queue Qcont,
                                                                 const Queue Qnext, const int chunk, const Lens64 L,
                                                                 const unsigned quad_max) {
  extern __shared__ __align__(16) unsigned char s_rec64[];
  __shared__ BlockTally S;
  const unsigned n_in = *(volatile unsigned*)Qin.count;
  if (n_in == 0) return;
  const int lane = threadIdx.x & 31;
  const bool quad = n_in <= quad_max;
  const unsigned per = quad ? 8u : 32u;  // molecules per warp
  const unsigned static_entries = gridDim.x * (blockDim.x / 32) * per;
  unsigned base = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * per;
  tally_init(S);
  if (!__syncthreads_or(base < n_in)) return;
  const double2* rec = L.rec;
  if (L.staged) {
    double2* s_rec = reinterpret_cast<double2*>(s_rec64);
    for (int k = threadIdx.x; k < 2 * (L.n + 1); k += blockDim.x) s_rec[k] = __ldg(L.rec + k);
    rec = s_rec;
    __syncthreads();
  }
  const ctraj_element& e = P.el[li];
  const bool classic = e.scheme == CTRAJ_RK4_CLASSIC;
  const double bore = dmul(e.p[0], 0.5);
  unsigned long long steps = 0, lsteps = 0, band = 0, bad = 0, range = 0, rerr = 0;
  while (base < n_in) {
    const unsigned idx = base + (quad ? unsigned(lane >> 2) : unsigned(lane));
    const bool have = idx < n_in;
    Mol64<false> m;
    LensStep st, nst;
    Lane64 w;
    w.phase = kIdle;
    w.x[0] = w.x[1] = w.v[0] = w.v[1] = w.z = w.t = w.dt = w.zinc = w.vz = w.a[0] = w.a[1] = 0.0;
    w.rmax = w.rlost = -1.0;
    w.flags = 0;
    w.n_done = w.n_total = 0;
    int n0 = 0;
    if (have) {
      m.load_state(Qin, idx, P, st);
      n0 = st.n_done;
      const int c = quad ? lane & 1 : 0;
      w.x[0] = m.x[c];
      w.v[0] = m.v[c];
      w.a[0] = m.a[c];
      w.x[1] = m.x[1];
      w.v[1] = m.v[1];
      w.a[1] = m.a[1];
      w.z = m.x[2];
      w.vz = m.v[2];
      w.t = m.t;
      w.dt = st.dt;
      // k1 = .. = k4 = vz: the z increment of every step
      const double vz = m.v[2];
      w.zinc = dmul(st.dt, dadd(dadd(dadd(vz, dmul(2.0, vz)), dmul(2.0, vz)), vz)) / 6.0;
      w.n_done = st.n_done;
      w.n_total = st.n_total;
      w.phase = kRun;
    }
    if (quad) advance_quad64<F>(w, P, li, L, rec, bore, classic, chunk);
    else advance_one64<F>(w, P, li, L, rec, bore, classic, chunk);
    int phase = w.phase;
    if (quad && (lane & 3)) phase = kIdle;  // the quad's first lane ends or requeues the molecule
    if (phase != kIdle) {
      m.x[0] = w.x[0];
      m.x[1] = w.x[1];
      m.x[2] = w.z;
      m.v[0] = w.v[0];
      m.v[1] = w.v[1];
      m.a[0] = w.a[0];
      m.a[1] = w.a[1];
      m.a[2] = 0.0;
      m.t = w.t;
      st.n_done = w.n_done;
      m.rows += isfinite(m.t) ? st.n_done - n0 : 0;
      if (w.rmax >= 0.0) m.note(dadd(w.rmax, -bore));
      if (w.rlost >= 0.0) m.note(dadd(w.rlost, -bore));
      lsteps += unsigned(st.n_done - n0);
    }
    int label = kNone;
    bool enter = false;
    if (phase == kLost || phase == kExit) {
      range += (w.flags & 1u) ? 1 : 0;
      rerr += (w.flags & 2u) ? 1 : 0;
      m.lens_end(P, li, st, phase == kLost);
      if (phase == kLost) {
        label = e.label_inside;
      } else {
        int lens_at = -1;
        label = walk(m, P, li + 1, &lens_at);
        if (label == kQueued) {
          enter = enter_lens(m, P, lens_at, nst);
          if (!enter) {
            label = P.el[lens_at].label_inside;
            ++bad;
          }
        }
      }
      if (label != kQueued) {
        steps += unsigned(m.rows);
        band += (m.margin < double(kEdgeBand)) ? 1 : 0;
        write_outputs<Mol64<false>, kOut>(R, m, label);
      }
    }
    push_lens(Qcont, phase == kRun, m, st);
    push_lens(Qnext, enter, m, nst);
    tally_warp(S, label, P.n_labels);
    unsigned b = 0;
    if (lane == 0) b = atomicAdd(Qin.head, per);
    base = static_entries + __shfl_sync(kFull, b, 0);
  }
  stat_add(S, kStatSteps, steps);
  stat_add(S, kStatLensSteps, lsteps);
  stat_add(S, kStatEdgeBand, band);
  stat_add(S, kStatBadSteps, bad);
  stat_add(S, kStatTableRange, range);
  stat_add(S, kStatRangeError, rerr);
  tally_flush(S, R, P.n_labels);
}

}  // namespace ctraj
