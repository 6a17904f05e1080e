// libctraj.so: the exact-mode lens kernel (k_lens_chunk64, k_chunk64.cuh), its
// table records and its launcher.
#include "k_chunk64.cuh"

namespace ctraj {
namespace {

using Kernel64 = void (*)(const Plan, const RunDev, const int, const Queue, const Queue, const Queue, const int,
                          const Lens64, const unsigned);
template <bool kOut>
Kernel64 kernel64(int kind, int field_order) {
  if (kind == CTRAJ_TABLE_RADIAL_LINEAR) return k_lens_chunk64<kOut, kForceRadial>;
  return field_order == 1 ? k_lens_chunk64<kOut, kForceStark1> : k_lens_chunk64<kOut, kForceStark2>;
}

// The records of a force table: per interval (knot, c0, c1, c2) of a spline or
// (knot, value, slope, 0) of a radial table, then the last knot.  False when
// the table does not fit k_lens_chunk64 (a negative or non-finite entry where
// it compares or divides): such a lens takes k_lens_chunk.
bool records64(const HostTable& t, std::vector<double>& rec) {
  if (!(t.knots[0] >= 0.0) || !std::isfinite(t.knots[t.n - 1])) return false;
  rec.assign(size_t(t.n) * 4, 0.0);
  for (int j = 0; j < t.n; ++j) {
    double* r = &rec[size_t(j) * 4];
    r[0] = t.knots[j] + 0.0;  // no -0.0
    if (j == t.n - 1) break;
    if (!(t.knots[j] < t.knots[j + 1])) return false;
    if (t.kind == CTRAJ_TABLE_RADIAL_LINEAR) {
      r[1] = t.values[j];
      r[2] = (t.values[j + 1] - t.values[j]) / (t.knots[j + 1] - t.knots[j]);  // numpy.interp's slope
    } else {
      const double* c = &t.coef[size_t(j) * 4];
      r[1] = c[0];
      r[2] = c[1];
      r[3] = 0.0 + c[2];  // PPoly's sum starts at 0.0
    }
    if (!std::isfinite(r[1]) || !std::isfinite(r[2]) || !std::isfinite(r[3])) return false;
  }
  return true;
}

}  // namespace

int launch_chunk64(ctraj_context* c, bool out, const Plan& P, const RunDev& R, int li, const Queue& Qin,
                   const Queue& Qcont, const Queue& Qnext, unsigned count, int chunk, bool* launched) {
  *launched = false;
  const ctraj_element& e = P.el[li];
  HostTable& t = c->tables[e.table];
  if (!t.rec64_built) {
    std::vector<double> rec;
    t.rec64_ok = records64(t, rec);
    if (t.rec64_ok) {
      const int st = t.rec64.ensure(rec.size() * 8);
      if (st) return st;
      CT_CUDA(cudaMemcpyAsync(t.rec64.p, rec.data(), rec.size() * 8, cudaMemcpyHostToDevice, c->stream));
    }
    t.rec64_built = true;
  }
  if (!t.rec64_ok) return CTRAJ_OK;
  const double alpha = e.p[6], mass = e.p[5];
  if (t.kind == CTRAJ_TABLE_STARK_SPLINE &&
      (!std::isfinite(alpha) || std::signbit(alpha) || !(mass >= 0x1p-300 && mass < 0x1p300)))
    return CTRAJ_OK;
  Lens64 L{};
  L.rec = t.rec64.as<double2>();
  L.first = t.knots[0] + 0.0;
  L.last = t.knots[t.n - 1];
  L.alpha = alpha;
  L.alpha2 = 2.0 * alpha;
  L.mass = mass;
  L.inv_mass = 1.0 / mass;
  L.x0 = float(L.first);
  L.inv_h = float(double(t.n - 1) / (L.last - L.first));
  L.n = t.n - 1;
  const Kernel64 k = out ? kernel64<true>(t.kind, e.field_order) : kernel64<false>(t.kind, e.field_order);
  const size_t bytes = size_t(t.n) * 4 * sizeof(double);
  L.staged = bytes <= kLens64Staged;
  const size_t smem = L.staged ? bytes : 0;
  CT_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  // one batch per CTA while they last: warps spread over the SMs' schedulers
  const unsigned per = count <= kQuad64Max ? 8u : 32u;
  const unsigned most = unsigned(blocks_per_sm(k, kLens64Threads, smem) * c->sm_count);
  const unsigned grid = std::max(1u, std::min(most, (count + per - 1) / per));
  k<<<grid, kLens64Threads, smem, c->stream>>>(P, R, li, Qin, Qcont, Qnext, chunk, L, kQuad64Max);
  CT_CUDA(cudaGetLastError());
  *launched = true;
  return CTRAJ_OK;
}

}  // namespace ctraj
