// Per-task kernels: one GPU kernel set per reference task, same signature and
// semantics, operating on the caller's fields in the reference's numbering.
//
// Each kernel evaluates every output element with the same sequence of IEEE
// operations as the reference loop it cites (this file is compiled with
// -fmad=false, so no multiply-add is fused), and scatter loops of the
// reference become gathers over the reverse connectivity in the order the
// scatter visited them.  Results therefore agree value for value with the
// reference tasks (bit for bit, signs of zero in the ocean tasks aside), infinities
// and NaN included.  One thread per (entity, level); tracers loop inside.
#include <type_traits>

#include "softmul.cuh"
#include "task_io.cuh"

namespace mpaso {
namespace {

constexpr int TPB = 256;

// ---------------------------------------------------------------- sw tasks
// apps/sw/tasks/solve.cc:31-39 (h_edge), :41-60 (circulation, vorticity),
// :62-77 (ke), :81-92 (h_vertex, pv_vertex).
__global__ void k_sw_diag_a(DMesh m, Lev L, const double *__restrict__ h, const double *__restrict__ u,
                            double *h_edge, double *h_vertex, double *circulation, double *vorticity,
                            double *ke, double *pv_vertex) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t nEL = (int64_t)m.nE * L, nVL = (int64_t)m.nV * L, nCL = (int64_t)m.nC * L;
  if (i < nEL) {
    int e, k;
    L.split(i, e, k);
    const int2 c = m.coe[e];
    h_edge[i] = 0.5 * (h[(int64_t)c.x * L + k] + h[(int64_t)c.y * L + k]);
    return;
  }
  i -= nEL;
  if (i < nVL) {
    int v, k;
    L.split(i, v, k);
    double circ = 0.0;
    for (int j = 0; j < kVertexDegree; ++j) {  // edges in ascending reference order
      const int e = m.eov[(int64_t)j * m.nV + v];
      const double t = m.dcEdge[e] * u[(int64_t)e * L + k];
      circ = (m.eovSign[(int64_t)j * m.nV + v] < 0.0) ? circ - t : circ + t;
    }
    circulation[i] = circ;
    const double vort = circ / m.areaTriangle[v];
    vorticity[i] = vort;
    double hv = 0.0;
    for (int j = 0; j < kVertexDegree; ++j)
      hv += h[(int64_t)m.cov[(int64_t)j * m.nV + v] * L + k] * m.kite[(int64_t)j * m.nV + v];
    hv /= m.areaTriangle[v];
    h_vertex[i] = hv;
    pv_vertex[i] = (m.fVertex[v] + vort) / hv;
    return;
  }
  i -= nVL;
  if (i < nCL) {
    int c, k;
    L.split(i, c, k);
    double s = 0.0;
    const int n = m.nEoC[c];
    for (int j = 0; j < n; ++j) {
      const int e = m.eoc[(int64_t)j * m.nC + c];
      const double ue = u[(int64_t)e * L + k];
      s += 0.25 * m.dcEdge[e] * m.dvEdge[e] * (ue * ue);
    }
    ke[i] = s / m.areaCell[c];
  }
}

// apps/sw/tasks/solve.cc:95-106: pv_edge(e) = 0 + 0.5 pv(v) over the edge's two vertices.
__global__ void k_sw_diag_b(DMesh m, Lev L, const double *__restrict__ pv_vertex, double *pv_edge) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= (int64_t)m.nE * L) return;
  int e, k;
  L.split(i, e, k);
  const int2 v = m.voe[e];
  const double a = 0.5 * pv_vertex[(int64_t)v.x * L + k], b = 0.5 * pv_vertex[(int64_t)v.y * L + k];
  pv_edge[i] = (0.0 + a) + b;  // two terms: order-free
}

// apps/sw/tasks/solve.cc:169-234
__global__ void k_sw_tend(DMesh m, Lev L, double g, const double *__restrict__ h_edge,
                          const double *__restrict__ h, const double *__restrict__ u,
                          const double *__restrict__ ke, const double *__restrict__ pv_edge,
                          double *tend_h, double *tend_u) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t nEL = (int64_t)m.nE * L, nCL = (int64_t)m.nC * L;
  if (i < nEL) {
    int e, k;
    L.split(i, e, k);
    const int2 c = m.coe[e];
    const int n = m.nEoE[e];
    const double pve = pv_edge[i];
    double q = 0;
    for (int j = 0; j < n; ++j) {
      const int eo = m.eoe[(int64_t)j * m.nE + e];
      const double workpv = 0.5 * (pve + pv_edge[(int64_t)eo * L + k]);
      q = q + m.woe[(int64_t)j * m.nE + e] * u[(int64_t)eo * L + k] * workpv * h_edge[(int64_t)eo * L + k];
    }
    const int64_t i1 = (int64_t)c.x * L + k, i2 = (int64_t)c.y * L + k;
    tend_u[i] = q - (ke[i2] - ke[i1] + g * (h[i2] + m.bottomDepth[c.y] - h[i1] - m.bottomDepth[c.x])) /
                        m.dcEdge[e];
    return;
  }
  i -= nEL;
  if (i < nCL) {
    int c, k;
    L.split(i, c, k);
    double t = 0;
    const int n = m.nEoC[c];
    for (int j = 0; j < n; ++j) {  // scatter order: ascending reference edge id
      const int e = m.eocAsc[(int64_t)j * m.nC + c];
      const double flux = u[(int64_t)e * L + k] * m.dvEdge[e] * h_edge[(int64_t)e * L + k];
      t = (m.eocAscSign[(int64_t)j * m.nC + c] < 0.0) ? t - flux : t + flux;
    }
    tend_h[i] = t / m.areaCell[c];
  }
}

// apps/sw/tasks/solve.cc:237-270
__global__ void k_sw_scalar_tend(DMesh m, Lev L, int T, const double *__restrict__ h_edge,
                                 const double *__restrict__ u, const double *__restrict__ tr,
                                 double *tend) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= (int64_t)m.nC * L) return;
  int c, k;
  L.split(i, c, k);
  const int n = m.nEoC[c];
  for (int t = 0; t < T; ++t) {
    double acc = 0.0;
    for (int j = 0; j < n; ++j) {
      const int e = m.eocAsc[(int64_t)j * m.nC + c];
      const int2 cc = m.coe[e];
      const double tr_edge = 0.5 * (tr[((int64_t)cc.x * L + k) * T + t] + tr[((int64_t)cc.y * L + k) * T + t]);
      const double flux = u[(int64_t)e * L + k] * m.dvEdge[e] * h_edge[(int64_t)e * L + k] * tr_edge;
      acc = (m.eocAscSign[(int64_t)j * m.nC + c] < 0.0) ? acc - flux / m.areaCell[c]
                                                         : acc + flux / m.areaCell[c];
    }
    tend[i * T + t] = acc;
  }
}

// Elementwise sw tasks (no connectivity): apps/sw/tasks/solve.cc:273-367.
__global__ void k_sw_substep(int64_t nEL, int64_t nCL, int T, double *u_p, const double *u_o,
                             const double *u_t, double *h_p, const double *h_o, const double *h_t,
                             double *tr_p, const double *tr_o, const double *tr_t, double w, int pin_u) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < nEL) u_p[i] = pin_u ? u_o[i] : u_o[i] + w * u_t[i];
  if (i < nCL) {
    const double hp = h_o[i] + w * h_t[i];
    h_p[i] = hp;
    for (int t = 0; t < T; ++t) tr_p[i * T + t] = (h_o[i] * tr_o[i * T + t] + w * tr_t[i * T + t]) / hp;
  }
}

__global__ void k_sw_accumulate(int64_t nEL, int64_t nCL, int T, double *u_n, const double *u_t,
                                double *h_n, const double *h_t, double *tr_n, const double *tr_t,
                                double w) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < nEL) u_n[i] += w * u_t[i];
  if (i < nCL) {
    h_n[i] += w * h_t[i];
    for (int t = 0; t < T; ++t) tr_n[i * T + t] += w * tr_t[i * T + t];
  }
}

__global__ void k_sw_finalize(int64_t nEL, int64_t nCL, int T, const double *u_o, double *u_n,
                              const double *h_n, double *tr_n, int pin_u) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < nCL)
    for (int t = 0; t < T; ++t) tr_n[i * T + t] /= h_n[i];
  if (pin_u && i < nEL) u_n[i] = u_o[i];
}

// ---------------------------------------------------------------- ocean tasks
__global__ void k_oc_ntf(int64_t n, const double *hE, const double *u, double *ntf) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) ntf[i] = u[i] * hE[i];  // apps/ocean/tasks/solve.cc:49-54
}

// The products of the kernels below run on the integer pipe (softmul.cuh, the
// hardware's rounding bit for bit) and comparisons on the bit patterns, which
// leaves the FP64 pipe the sums; tracers are unrolled at compile time, and what
// levels share (1 / area, the mixing coefficient) is not divided out in each.
// Level 5, 20 levels x 3 tracers, us: high order 130 -> 63, fct_a + fct_b + fct_c
// 187 -> 87, hmix 128 -> 34, accumulate 35 -> 21, low order 20 -> 11, provisional
// 20 -> 16; a tracer stage task by task 456 -> 186.

// IEEE a < b on the integer pipe (false with a NaN; zeros are equal).
__device__ __forceinline__ bool ieee_lt(double a, double b) {
  constexpr long long kInf = 0x7ff0000000000000LL;
  const long long x = dbits(a), y = dbits(b);
  const long long ka = x < 0 ? kSignBit - x : x, kb = y < 0 ? kSignBit - y : y;
  return ka < kb && kb <= kInf && ka >= -kInf;
}

static __device__ __noinline__ double rare_product(double a, double b) { return a * b; }

// s * x for an edge sign s: a sign flip for the +-1 it is, else the product.
struct EdgeSign {
  double s;
  long long flip;
  bool unit;
  __device__ explicit EdgeSign(double v)
      : s(v), flip(dbits(v) & kSignBit), unit((dbits(v) & ~kSignBit) == 0x3ff0000000000000LL) {}
  __device__ double times(double x) const { return unit ? dflip(x, flip) : rare_product(s, x); }
};

// apps/ocean/tasks/solve.cc:60-97
__global__ void __launch_bounds__(TPB) k_oc_provisional(DMesh m, Lev L, const double *__restrict__ h,
                                                        const double *__restrict__ ntf, double *hProv,
                                                        double *hProvInv, double *hNewInv, double dt) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= (int64_t)m.nC * L) return;
  int c, k;
  L.split(i, c, k);
  if (k >= m.maxLevelCell[c]) return;
  const double dtInvAreaCell = dt / m.areaCell[c];
  double hp = h[i];
  const int n = m.nEoC[c];
  for (int j = 0; j < n; ++j) {
    const int64_t s = (int64_t)j * m.nC + c;
    const int e = m.eoc[s];
    const double sf = EdgeSign(m.eocSign[s]).times(mul_int(m.dvEdge[e], dtInvAreaCell));
    hp += mul_int(ntf[(int64_t)e * L + k], sf);
  }
  hProv[i] = hp;
  const double inv = 1.0 / hp;
  hProvInv[i] = inv;
  hNewInv[i] = inv;
}

// max(0, f) tr1 + min(0, f) tr2 where a factor is not finite or outside the products' window
static __device__ __noinline__ double rare_upwind(double f, double tr1, double tr2) {
  const double ntf1 = (0.0 < f) ? f : 0.0;  // std::max(0.0, f)
  const double ntf2 = (f < 0.0) ? f : 0.0;  // std::min(0.0, f)
  return ntf1 * tr1 + ntf2 * tr2;
}

// apps/ocean/tasks/solve.cc:99-118: dv (max(0, f) tr1 + min(0, f) tr2), one of
// whose two products is a zero
template <int T>
__global__ void __launch_bounds__(TPB) k_oc_low_order(DMesh m, Lev L, const double *__restrict__ ntf,
                                                      const double *__restrict__ tr, double *lo) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= (int64_t)m.nE * L) return;
  int e, k;
  L.split(i, e, k);
  const int2 c = m.coe[e];
  const double f = ntf[i], dv = m.dvEdge[e];
  const int64_t i1 = ((int64_t)c.x * L + k) * T, i2 = ((int64_t)c.y * L + k) * T;
  uint32_t badf = 0, badv = 0;
  const SoftFactor ff = soft_factor(f, badf), fv = soft_factor(dv, badv);
  constexpr long long kInf = 0x7ff0000000000000LL;
  const bool up1 = dgt0(f);
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const double t1 = tr[i1 + t], t2 = tr[i2 + t];
    uint32_t bad = badf;
    double x = soft_mul(up1 ? t1 : t2, ff, bad);
    if (bad || (dbits(up1 ? t2 : t1) & kInf) == kInf) x = rare_upwind(f, t1, t2);
    bad = badv;
    double r = soft_mul(x, fv, bad);
    if (bad) r = rare_product(dv, x);
    lo[i * T + t] = r;
  }
}

// apps/ocean/tasks/solve.cc:120-167 (coef3rdOrder = 0.25, :11).  The factor
// coef1 + coef3 sgn is advCp / advCm by the sign of the flux (a zero flux
// weighs every term with zero).
template <int T>
__global__ void __launch_bounds__(TPB) k_oc_high_order(DMesh m, Lev L, const double *__restrict__ ntf,
                                                       const double *__restrict__ tr, double *ho) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= (int64_t)m.nE * L) return;
  int e, k;
  L.split(i, e, k);
  const double f = ntf[i];
  const int mask = m.hoMask[(int64_t)e * m.fctLev + k];
  const double wgt = mask == 1 ? f : mask == 0 ? bitsd(dbits(f) & kSignBit) : masked_weight(f, mask);
  const double *coef = dlt0(f) ? m.advCm : m.advCp;
  uint32_t badw = 0;
  const SoftFactor fw = soft_factor(wgt, badw);
  double flx[T];
#pragma unroll
  for (int t = 0; t < T; ++t) flx[t] = 0.0;
  const int n = m.nAdv[e];
#pragma unroll 2
  for (int a = 0; a < n; ++a) {
    const int64_t sa = (int64_t)a * m.nE + e;
    const int cell = m.advCells[sa];
    if (k >= m.maxLevelCell[cell]) continue;
    const double cf = coef[sa];
    const double *x = tr + ((int64_t)cell * L + k) * T;
    uint32_t bad = badw;
    const SoftFactor wf = soft_factor(soft_mul(cf, fw, bad), bad);
    double p[T];
#pragma unroll
    for (int t = 0; t < T; ++t) p[t] = soft_mul(x[t], wf, bad);
    if (bad) {
      const double wx = rare_product(wgt, cf);
#pragma unroll
      for (int t = 0; t < T; ++t) p[t] = rare_product(x[t], wx);
    }
#pragma unroll
    for (int t = 0; t < T; ++t) flx[t] += p[t];
  }
#pragma unroll
  for (int t = 0; t < T; ++t) ho[i * T + t] = flx[t];
}

// x + tw (t1 + t2) with a weight tw of zero: x unless f or the sum is not finite.
static __device__ __noinline__ double add_weightless_flux(double x, double f, double sum) { return x + (0.0 * f) * sum; }

// apps/ocean/tasks/solve.cc:216-229: anti-diffusive flux of the edges.  The
// centred flux has the weight ((mask + 1) & 1), which is 0 on almost all of them.
template <int T>
__global__ void __launch_bounds__(TPB) k_oc_fct_a(DMesh m, Lev L, const double *__restrict__ ntf,
                                                  const double *__restrict__ lo, const double *__restrict__ tr,
                                                  double *ho) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= (int64_t)m.nE * L) return;
  int e, k;
  L.split(i, e, k);
  if (k >= m.maxLevelEdgeTop[e]) return;
  const bool centred = (m.hoMask[(int64_t)e * m.fctLev + k] + 1) & 1;
  const double f = ntf[i];
  const int2 c = m.coe[e];
  const int64_t i1 = ((int64_t)c.x * L + k) * T, i2 = ((int64_t)c.y * L + k) * T;
#pragma unroll
  for (int t = 0; t < T; ++t) {
    double x = ho[i * T + t];
    const double t1 = tr[i1 + t], t2 = tr[i2 + t], sum = t1 + t2;
    if (centred)
      x = add_centred_flux(x, m.dvEdge[e], f, t1, t2);
    else if (nonfinite(f) || nonfinite(sum))
      x = add_weightless_flux(x, f, sum);
    ho[i * T + t] = x - lo[i * T + t];
  }
}

// std::min(1, std::max(0, num / den)) (solve.cc:258-265), divided only where the
// quotient may lie inside (0, 1) or be no number.
static __device__ __noinline__ double rare_limit(double num, double den) {
  const double q = num / den, p = (0.0 < q) ? q : 0.0;
  return (p < 1.0) ? p : 1.0;
}
__device__ __forceinline__ double limiter_factor(double num, double den) {
  const bool pos = dgt0(num);
  double r = pos ? 1.0 : 0.0;
  if (!dgt0(den) || nonfinite(num) || nonfinite(den) || (pos && dkey(num) < dkey(den))) r = rare_limit(num, den);
  return r;
}

// apps/ocean/tasks/solve.cc:194-214, 232-267: bounds over the cell and its
// neighbours, per-cell sums and limiter factors.
template <int T>
__global__ void __launch_bounds__(TPB) k_oc_fct_b(DMesh m, Lev L, const double *__restrict__ hProvInv,
                                                  const double *__restrict__ h, const double *__restrict__ lo,
                                                  const double *__restrict__ tr, const double *__restrict__ ho,
                                                  double *flxIn, double *flxOut, double *tend, double *trMax,
                                                  double *trMin, double dt) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= (int64_t)m.nC * L) return;
  int c, k;
  L.split(i, c, k);
  const double eps = 1.e-10;
  const double invAreaCell1 = m.invAreaCell[c];  // 1 / areaCell
  const int n = m.nEoC[c], mlc = m.maxLevelCell[c];
  const bool live = k < mlc;
  double trc[T], mx[T], mn[T], td[T], fin[T], fout[T];
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const int64_t it = i * T + t;
    trc[t] = mx[t] = mn[t] = tr[it];
    td[t] = tend[it];
    fin[t] = live ? 0.0 : flxIn[it], fout[t] = live ? 0.0 : flxOut[it];
  }
  for (int j = 0; j < n; ++j) {
    const int64_t s = (int64_t)j * m.nC + c;
    const int e = m.eoc[s], c2 = m.coc[s];
    if (live && k < m.maxLevelCell[c2]) {
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const double x = tr[((int64_t)c2 * L + k) * T + t];
        mx[t] = ieee_lt(mx[t], x) ? x : mx[t];  // std::max
        mn[t] = ieee_lt(x, mn[t]) ? x : mn[t];  // std::min
      }
    }
    if (k >= m.maxLevelEdgeTop[e]) continue;
    const double sf = EdgeSign(m.eocSign[s]).times(invAreaCell1);
    uint32_t bads = 0;
    const SoftFactor fs = soft_factor(sf, bads);
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const double xl = lo[((int64_t)e * L + k) * T + t], xh = ho[((int64_t)e * L + k) * T + t];
      uint32_t bad = bads;
      double pl = soft_mul(xl, fs, bad), x = soft_mul(xh, fs, bad);
      if (bad) pl = rare_product(sf, xl), x = rare_product(sf, xh);
      td[t] += pl;
      // flxIn += max(0, x), flxOut += min(0, x): one add into the sum the sign selects
      const bool in = ieee_lt(0.0, x), out = ieee_lt(x, 0.0);
      const double acc = opaque(in ? fin[t] : fout[t]) + x;
      fin[t] = in ? acc : fin[t];
      fout[t] = out ? acc : fout[t];
    }
  }
  const double hc = h[i], hpi = live ? hProvInv[i] : 0.0;
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const int64_t it = i * T + t;
    tend[it] = td[t];
    if (live) {
      const double up = mul_int(mul_int(trc[t], hc) + mul_int(td[t], dt), hpi);
      const double mxn = up + mul_int(mul_int(fin[t], dt), hpi);
      const double mnn = up + mul_int(mul_int(fout[t], dt), hpi);
      trMax[it] = mx[t];
      trMin[it] = mn[t];
      fin[t] = limiter_factor(mx[t] - up, (mxn - up) + eps);
      fout[t] = limiter_factor(up - mn[t], (up - mnn) + eps);
    }
    flxIn[it] = fin[t];
    flxOut[it] = fout[t];
  }
}

// max(0, x) min(in2, out1) + min(0, x) min(out2, in1), both products formed.
static __device__ __noinline__ double rare_rescale(double x, double in1, double out1, double in2, double out2) {
  const double a = in2 < out1 ? in2 : out1, b = out2 < in1 ? out2 : in1;
  return ((0.0 < x) ? x : 0.0) * a + ((x < 0.0) ? x : 0.0) * b;
}

// apps/ocean/tasks/solve.cc:270-282: rescale anti-diffusive fluxes,
// max(0, x) min(R-(c1), R+(c2)) + min(0, x) min(R+(c1), R-(c2)), whose factor the
// sign of x selects: the other, times zero, counts for nothing where both cells
// have the level, whose factors k_oc_fct_b put into [0, 1].  In a level below a
// cell's column (an edge goes down to the deeper of its two cells) flxIn and
// flxOut are the caller's plus sums, which may be infinite or NaN.
template <int T>
__global__ void __launch_bounds__(TPB) k_oc_fct_c(DMesh m, Lev L, const double *__restrict__ flxIn,
                                                  const double *__restrict__ flxOut, double *ho) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= (int64_t)m.nE * L) return;
  int e, k;
  L.split(i, e, k);
  if (k >= m.maxLevelEdgeTop[e]) return;
  const int2 c = m.coe[e];
  const int64_t i1 = ((int64_t)c.x * L + k) * T, i2 = ((int64_t)c.y * L + k) * T;
  if (k >= m.maxLevelCell[c.x] || k >= m.maxLevelCell[c.y]) {
    for (int t = 0; t < T; ++t)
      ho[i * T + t] = rare_rescale(ho[i * T + t], flxIn[i1 + t], flxOut[i1 + t], flxIn[i2 + t], flxOut[i2 + t]);
    return;
  }
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const double x = ho[i * T + t];
    const bool pos = ieee_lt(0.0, x), neg = ieee_lt(x, 0.0);
    const double r1 = pos ? flxOut[i1 + t] : flxIn[i1 + t], r2 = pos ? flxIn[i2 + t] : flxOut[i2 + t];
    const double r = ieee_lt(r2, r1) ? r2 : r1;
    // (r as the first operand: it is often zero)
    ho[i * T + t] = pos || neg ? mul_int(r, x) : 0.0;
  }
}

// apps/ocean/tasks/solve.cc:287-326
template <int T>
__global__ void __launch_bounds__(TPB) k_oc_accumulate_fct(DMesh m, Lev L, const double *__restrict__ hProvInv,
                                                           const double *__restrict__ h,
                                                           const double *__restrict__ ho,
                                                           const double *__restrict__ tr, double *trProv,
                                                           double *tend, double dt) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= (int64_t)m.nC * L) return;
  int c, k;
  L.split(i, c, k);
  const double invAreaCell1 = m.invAreaCell[c];
  const int n = m.nEoC[c];
  double td[T];
#pragma unroll
  for (int t = 0; t < T; ++t) td[t] = tend[i * T + t];
  for (int j = 0; j < n; ++j) {
    const int64_t s = (int64_t)j * m.nC + c;
    const int e = m.eoc[s];
    if (k >= m.maxLevelEdgeTop[e]) continue;
    const double sf = EdgeSign(m.eocSign[s]).times(invAreaCell1);
    uint32_t bads = 0;
    const SoftFactor fs = soft_factor(sf, bads);
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const double x = ho[((int64_t)e * L + k) * T + t];
      uint32_t bad = bads;
      double p = soft_mul(x, fs, bad);
      if (bad) p = rare_product(sf, x);
      td[t] += p;
    }
  }
  const bool live = k < m.maxLevelCell[c];
  const double hc = h[i], hpi = live ? hProvInv[i] : 0.0;
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const int64_t it = i * T + t;
    tend[it] = td[t];
    if (live) trProv[it] = mul_int(mul_int(tr[it], hc) + mul_int(td[t], dt), hpi);
  }
}

// apps/ocean/tasks/solve.cc:328-366.  rho (:352) is formed once per cell and slot of
// the block's cells, in shared memory, instead of in every level.  (An array of
// the call's own for it, once per edge in a launch ahead, would have to outlive
// graphs that recorded the call and be private to each stream.)
constexpr int hmix_cells(int L) { return (L + TPB - 2) / L + 1; }  // most cells that TPB cell-levels touch

template <int T>
__global__ void __launch_bounds__(TPB) k_oc_hmix(DMesh m, Lev L, const double *__restrict__ hE,
                                                 const double *__restrict__ tr, double coef, double *tend) {
  extern __shared__ double rho[];  // [maxEoC][cells of the block]
  const int64_t i0 = blockIdx.x * (int64_t)blockDim.x, i = i0 + threadIdx.x, n_all = (int64_t)m.nC * L;
  int c0, c1, unused;
  L.split(i0, c0, unused);
  L.split(min(i0 + blockDim.x, n_all) - 1, c1, unused);
  const int nc = c1 - c0 + 1;
  for (int s = threadIdx.x; s < nc * m.maxEoC; s += blockDim.x) {
    const int j = s / nc, e = m.eoc[(int64_t)j * m.nC + c0 + (s - j * nc)];
    rho[s] = m.meshScalingDel2[e] * coef * m.dvEdge[e] / m.dcEdge[e];
  }
  __syncthreads();
  if (i >= n_all) return;
  int c, k;
  L.split(i, c, k);
  const double invArea = m.invAreaCell[c];
  const int n = m.nEoC[c];
  uint32_t bada = 0;
  const SoftFactor fa = soft_factor(invArea, bada);
  double td[T];
#pragma unroll
  for (int t = 0; t < T; ++t) td[t] = tend[i * T + t];
  for (int j = 0; j < n; ++j) {
    const int64_t s = (int64_t)j * m.nC + c;
    const int e = m.eoc[s];
    if (k >= m.maxLevelEdgeTop[e]) continue;
    const int2 cc = m.coe[e];
    const double he = hE[(int64_t)e * L + k], re = rho[j * nc + c - c0];
    const EdgeSign sg(m.eocSign[s]);
    uint32_t badm = bada;
    const SoftFactor fh = soft_factor(he, badm), fr = soft_factor(re, badm);
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const double ttf = tr[((int64_t)cc.y * L + k) * T + t] - tr[((int64_t)cc.x * L + k) * T + t];
      uint32_t bad = badm;
      const double flux = soft_mul(soft_mul(ttf, fh, bad), fr, bad);
      double x = soft_mul(sg.times(flux), fa, bad);
      if (bad) x = rare_product(rare_product(sg.s, rare_product(rare_product(he, ttf), re)), invArea);
      td[t] -= x;
    }
  }
#pragma unroll
  for (int t = 0; t < T; ++t) tend[i * T + t] = td[t];
}

// apps/ocean/tasks/solve.cc:368-399
__global__ void k_oc_step_forward(int64_t n, const double *tend, const double *tr, double *trNew,
                                  double *trPrev, double w, double wsub) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  trNew[i] += w * tend[i];
  trPrev[i] = tr[i] + wsub * tend[i];
}

// Calls f with the tracer count as a compile-time constant.
template <class F> void with_tracers(int T, F &&f) {
  switch (T) {
    case 1: f(std::integral_constant<int, 1>{}); break;
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 5: f(std::integral_constant<int, 5>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    case 7: f(std::integral_constant<int, 7>{}); break;
    case 8: f(std::integral_constant<int, 8>{}); break;
    default: fail(MPASO_ERR_ARG, "ntr out of range (max 8)");
  }
}

void check_levels(int L, int T) {
  require(L >= 1 && L <= 4096, MPASO_ERR_ARG, "nlev out of range");
  require(T >= 0 && T <= kMaxTracers, MPASO_ERR_ARG, "ntr out of range (max 8)");
}

void require_fct(TaskIO &io, int L) {
  require(io.ctx().has_fct, MPASO_ERR_ARG, "mesh context was created without FCT statics");
  // (the context's own mesh: io.dm() is there only from stage() on)
  require(io.ctx().d.fctLev == L, MPASO_ERR_ARG, "nlev differs from the FCT statics' level count");
}

cudaStream_t plain_stream(mpaso_mesh m, void *stream) {
  require(m != nullptr, MPASO_ERR_ARG, "null mesh context");
  MPASO_CUDA(cudaSetDevice(m->ctx.device));
  return stream ? (cudaStream_t)stream : m->ctx.stream;
}

// Elementwise tasks need no renumbering: they run on the caller's arrays
// directly when all are device memory, else on staged copies.
struct Flat {
  std::vector<std::pair<double *, size_t>> args;  // user ptr, doubles
  std::vector<bool> out;
  std::vector<double *> dev;
  bool host = false;
  cudaStream_t s;
  mpaso_mesh m;
  void add(const double *p, size_t n, bool o) {
    require(p != nullptr, MPASO_ERR_ARG, "null field pointer");
    args.push_back({const_cast<double *>(p), n});
    out.push_back(o);
    host |= !is_device_pointer(p);
  }
  void stage() {
    dev.resize(args.size());
    if (!host) {
      for (size_t a = 0; a < args.size(); ++a) dev[a] = args[a].first;
      return;
    }
    size_t total = 0;
    for (auto &a : args) total += (a.second * sizeof(double) + 255) & ~size_t(255);
    char *base = (char *)m->ctx.ensure_scratch(total);
    for (size_t a = 0; a < args.size(); ++a) {
      dev[a] = (double *)base;
      base += (args[a].second * sizeof(double) + 255) & ~size_t(255);
      const cudaMemcpyKind kind = is_device_pointer(args[a].first) ? cudaMemcpyDeviceToDevice
                                                                    : cudaMemcpyHostToDevice;
      MPASO_CUDA(cudaMemcpyAsync(dev[a], args[a].first, args[a].second * sizeof(double), kind, s));
    }
  }
  void finish() {
    MPASO_CUDA(cudaGetLastError());
    if (!host) return;
    for (size_t a = 0; a < args.size(); ++a)
      if (out[a]) {
        const cudaMemcpyKind kind = is_device_pointer(args[a].first) ? cudaMemcpyDeviceToDevice
                                                                      : cudaMemcpyDeviceToHost;
        MPASO_CUDA(cudaMemcpyAsync(args[a].first, dev[a], args[a].second * sizeof(double), kind, s));
      }
    MPASO_CUDA(cudaStreamSynchronize(s));
  }
};

}  // namespace

// Launches the compute_tend kernel on arrays already in the context's
// numbering (used by the allocation-free entry point in noalloc.cu).
void launch_task_sw_tend(const DMesh &d, int L, double g, const double *h_edge, const double *h,
                         const double *u, const double *ke, const double *pv_edge, double *tend_h,
                         double *tend_u, cudaStream_t s) {
  const int64_t n = ((int64_t)d.nE + d.nC) * L;
  k_sw_tend<<<blocks_for(n, TPB), TPB, 0, s>>>(d, L, g, h_edge, h, u, ke, pv_edge, tend_h, tend_u);
}

}  // namespace mpaso

using namespace mpaso;

extern "C" {

int mpaso_sw_compute_solve_diagnostics(mpaso_mesh m, int32_t nlev, const double *h,
                                       const double *u, double *h_edge, double *h_vertex,
                                       double *circulation, double *vorticity, double *ke,
                                       double *pv_edge, double *pv_vertex, void *stream) {
  return guarded("mpaso_sw_compute_solve_diagnostics", [&] {
    check_levels(nlev, 0);
    TaskIO io(m, stream);
    const int L = nlev;
    const int ih = io.in(h, MPASO_CELLS, L), iu = io.in(u, MPASO_EDGES, L);
    const int ohe = io.out(h_edge, MPASO_EDGES, L), ohv = io.out(h_vertex, MPASO_VERTICES, L);
    const int oci = io.out(circulation, MPASO_VERTICES, L), ovo = io.out(vorticity, MPASO_VERTICES, L);
    const int oke = io.out(ke, MPASO_CELLS, L), ope = io.out(pv_edge, MPASO_EDGES, L);
    const int opv = io.out(pv_vertex, MPASO_VERTICES, L);
    io.stage();
    const DMesh &d = io.dm();
    const int64_t n = ((int64_t)d.nE + d.nV + d.nC) * L;
    k_sw_diag_a<<<blocks_for(n, TPB), TPB, 0, io.stream()>>>(d, L, io.ptr(ih), io.ptr(iu), io.ptr(ohe),
                                                             io.ptr(ohv), io.ptr(oci), io.ptr(ovo),
                                                             io.ptr(oke), io.ptr(opv));
    k_sw_diag_b<<<blocks_for((int64_t)d.nE * L, TPB), TPB, 0, io.stream()>>>(d, L, io.ptr(opv), io.ptr(ope));
    io.finish();
  });
}

int mpaso_sw_compute_tend(mpaso_mesh m, int32_t nlev, const double *h_edge, const double *h,
                          const double *u, const double *ke, const double *pv_edge,
                          double *tend_h, double *tend_u, void *stream) {
  return guarded("mpaso_sw_compute_tend", [&] {
    check_levels(nlev, 0);
    TaskIO io(m, stream);
    const int L = nlev;
    const int ihe = io.in(h_edge, MPASO_EDGES, L), ih = io.in(h, MPASO_CELLS, L);
    const int iu = io.in(u, MPASO_EDGES, L), ike = io.in(ke, MPASO_CELLS, L);
    const int ipe = io.in(pv_edge, MPASO_EDGES, L);
    const int oth = io.out(tend_h, MPASO_CELLS, L), otu = io.out(tend_u, MPASO_EDGES, L);
    io.stage();
    const DMesh &d = io.dm();
    const int64_t n = ((int64_t)d.nE + d.nC) * L;
    k_sw_tend<<<blocks_for(n, TPB), TPB, 0, io.stream()>>>(d, L, io.ctx().gravity, io.ptr(ihe), io.ptr(ih),
                                                           io.ptr(iu), io.ptr(ike), io.ptr(ipe),
                                                           io.ptr(oth), io.ptr(otu));
    io.finish();
  });
}

int mpaso_sw_compute_scalar_tend(mpaso_mesh m, int32_t nlev, int32_t ntr, const double *h_edge,
                                 const double *u, const double *tracers, double *tracer_tend,
                                 void *stream) {
  return guarded("mpaso_sw_compute_scalar_tend", [&] {
    check_levels(nlev, ntr);
    TaskIO io(m, stream);
    const int L = nlev, T = ntr;
    const int ihe = io.in(h_edge, MPASO_EDGES, L), iu = io.in(u, MPASO_EDGES, L);
    const int itr = io.in(tracers, MPASO_CELLS, L * T);
    const int ot = io.out(tracer_tend, MPASO_CELLS, L * T);
    io.stage();
    const DMesh &d = io.dm();
    k_sw_scalar_tend<<<blocks_for((int64_t)d.nC * L, TPB), TPB, 0, io.stream()>>>(
        d, L, T, io.ptr(ihe), io.ptr(iu), io.ptr(itr), io.ptr(ot));
    io.finish();
  });
}

int mpaso_sw_compute_substep(mpaso_mesh m, int32_t nlev, int32_t ntr, double *u_provis,
                             const double *u_old, const double *u_tend, double *h_provis,
                             const double *h_old, const double *h_tend, double *tracers_provis,
                             const double *tracers_old, const double *tracers_tend,
                             double rkweight, int32_t pin_u, void *stream) {
  return guarded("mpaso_sw_compute_substep", [&] {
    check_levels(nlev, ntr);
    Flat f;
    f.s = plain_stream(m, stream), f.m = m;
    const size_t nEL = (size_t)m->ctx.d.nE * nlev, nCL = (size_t)m->ctx.d.nC * nlev;
    f.add(u_provis, nEL, true), f.add(u_old, nEL, false), f.add(u_tend, nEL, false);
    f.add(h_provis, nCL, true), f.add(h_old, nCL, false), f.add(h_tend, nCL, false);
    f.add(tracers_provis, nCL * ntr, true), f.add(tracers_old, nCL * ntr, false);
    f.add(tracers_tend, nCL * ntr, false);
    f.stage();
    k_sw_substep<<<blocks_for((int64_t)std::max(nEL, nCL), TPB), TPB, 0, f.s>>>(
        nEL, nCL, ntr, f.dev[0], f.dev[1], f.dev[2], f.dev[3], f.dev[4], f.dev[5], f.dev[6],
        f.dev[7], f.dev[8], rkweight, pin_u);
    f.finish();
  });
}

int mpaso_sw_accumulate_update(mpaso_mesh m, int32_t nlev, int32_t ntr, double *u_new,
                               const double *u_tend, double *h_new, const double *h_tend,
                               double *tracers_new, const double *tracers_tend, double rkweight,
                               void *stream) {
  return guarded("mpaso_sw_accumulate_update", [&] {
    check_levels(nlev, ntr);
    Flat f;
    f.s = plain_stream(m, stream), f.m = m;
    const size_t nEL = (size_t)m->ctx.d.nE * nlev, nCL = (size_t)m->ctx.d.nC * nlev;
    f.add(u_new, nEL, true), f.add(u_tend, nEL, false), f.add(h_new, nCL, true);
    f.add(h_tend, nCL, false), f.add(tracers_new, nCL * ntr, true), f.add(tracers_tend, nCL * ntr, false);
    f.stage();
    k_sw_accumulate<<<blocks_for((int64_t)std::max(nEL, nCL), TPB), TPB, 0, f.s>>>(
        nEL, nCL, ntr, f.dev[0], f.dev[1], f.dev[2], f.dev[3], f.dev[4], f.dev[5], rkweight);
    f.finish();
  });
}

int mpaso_sw_finalize_timestep(mpaso_mesh m, int32_t nlev, int32_t ntr, const double *u_old,
                               double *u_new, const double *h_new, double *tracers_new,
                               int32_t pin_u, void *stream) {
  return guarded("mpaso_sw_finalize_timestep", [&] {
    check_levels(nlev, ntr);
    Flat f;
    f.s = plain_stream(m, stream), f.m = m;
    const size_t nEL = (size_t)m->ctx.d.nE * nlev, nCL = (size_t)m->ctx.d.nC * nlev;
    f.add(u_old, nEL, false), f.add(u_new, nEL, true), f.add(h_new, nCL, false);
    f.add(tracers_new, nCL * ntr, true);
    f.stage();
    k_sw_finalize<<<blocks_for((int64_t)std::max(nEL, nCL), TPB), TPB, 0, f.s>>>(
        nEL, nCL, ntr, f.dev[0], f.dev[1], f.dev[2], f.dev[3], pin_u);
    f.finish();
  });
}

int mpaso_oc_calc_normal_thickness_flux(mpaso_mesh m, int32_t nlev,
                                        const double *layerThicknessEdge,
                                        const double *normalVelocity,
                                        double *normalThicknessFlux, void *stream) {
  return guarded("mpaso_oc_calc_normal_thickness_flux", [&] {
    check_levels(nlev, 0);
    Flat f;
    f.s = plain_stream(m, stream), f.m = m;
    const size_t nEL = (size_t)m->ctx.d.nE * nlev;
    f.add(layerThicknessEdge, nEL, false), f.add(normalVelocity, nEL, false);
    f.add(normalThicknessFlux, nEL, true);
    f.stage();
    k_oc_ntf<<<blocks_for((int64_t)nEL, TPB), TPB, 0, f.s>>>(nEL, f.dev[0], f.dev[1], f.dev[2]);
    f.finish();
  });
}

int mpaso_oc_calc_provisional_layer_thicknesses(mpaso_mesh m, int32_t nlev,
                                                const double *layerThickness,
                                                const double *normalThicknessFlux,
                                                double *hProv, double *hProvInv, double *hNewInv,
                                                double dt, void *stream) {
  return guarded("mpaso_oc_calc_provisional_layer_thicknesses", [&] {
    check_levels(nlev, 0);
    TaskIO io(m, stream);
    const int L = nlev;
    const int ih = io.in(layerThickness, MPASO_CELLS, L), intf = io.in(normalThicknessFlux, MPASO_EDGES, L);
    const int op = io.out(hProv, MPASO_CELLS, L), opi = io.out(hProvInv, MPASO_CELLS, L);
    const int oni = io.out(hNewInv, MPASO_CELLS, L);
    io.stage();
    const DMesh &d = io.dm();
    k_oc_provisional<<<blocks_for((int64_t)d.nC * L, TPB), TPB, 0, io.stream()>>>(
        d, L, io.ptr(ih), io.ptr(intf), io.ptr(op), io.ptr(opi), io.ptr(oni), dt);
    io.finish();
  });
}

int mpaso_oc_calc_horiz_tracer_advection_flux_mono_low_order(
    mpaso_mesh m, int32_t nlev, int32_t ntr, const double *normalThicknessFlux,
    const double *tracers, double *lowOrderFlux, void *stream) {
  return guarded("mpaso_oc_calc_horiz_tracer_advection_flux_mono_low_order", [&] {
    check_levels(nlev, ntr);
    TaskIO io(m, stream);
    const int L = nlev, T = ntr;
    const int intf = io.in(normalThicknessFlux, MPASO_EDGES, L), itr = io.in(tracers, MPASO_CELLS, L * T);
    const int olo = io.out(lowOrderFlux, MPASO_EDGES, L * T);
    io.stage();
    const DMesh &d = io.dm();
    with_tracers(T, [&](auto t) {
      k_oc_low_order<t.value><<<blocks_for((int64_t)d.nE * L, TPB), TPB, 0, io.stream()>>>(
          d, L, io.ptr(intf), io.ptr(itr), io.ptr(olo));
    });
    io.finish();
  });
}

int mpaso_oc_calc_horiz_tracer_advection_flux_mono_high_order(
    mpaso_mesh m, int32_t nlev, int32_t ntr, const double *normalThicknessFlux,
    const double *tracers, double *highOrderFlux, void *stream) {
  return guarded("mpaso_oc_calc_horiz_tracer_advection_flux_mono_high_order", [&] {
    check_levels(nlev, ntr);
    TaskIO io(m, stream);
    require_fct(io, nlev);
    const int L = nlev, T = ntr;
    const int intf = io.in(normalThicknessFlux, MPASO_EDGES, L), itr = io.in(tracers, MPASO_CELLS, L * T);
    const int oho = io.out(highOrderFlux, MPASO_EDGES, L * T);
    io.stage();
    const DMesh &d = io.dm();
    with_tracers(T, [&](auto t) {
      k_oc_high_order<t.value><<<blocks_for((int64_t)d.nE * L, TPB), TPB, 0, io.stream()>>>(
          d, L, io.ptr(intf), io.ptr(itr), io.ptr(oho));
    });
    io.finish();
  });
}

int mpaso_oc_correct_and_rescale_high_order_mono_horiz_flux(
    mpaso_mesh m, int32_t nlev, int32_t ntr, const double *hProvInv, const double *layerThickness,
    const double *normalThicknessFlux, const double *lowOrderFlux, const double *tracers,
    double *highOrderFlux, double *flxIn, double *flxOut, double *tend, double *tracerMax,
    double *tracerMin, double dt, void *stream) {
  return guarded("mpaso_oc_correct_and_rescale_high_order_mono_horiz_flux", [&] {
    check_levels(nlev, ntr);
    TaskIO io(m, stream);
    require_fct(io, nlev);
    const int L = nlev, T = ntr;
    const int ihpi = io.in(hProvInv, MPASO_CELLS, L), ih = io.in(layerThickness, MPASO_CELLS, L);
    const int intf = io.in(normalThicknessFlux, MPASO_EDGES, L);
    const int ilo = io.in(lowOrderFlux, MPASO_EDGES, L * T), itr = io.in(tracers, MPASO_CELLS, L * T);
    const int oho = io.out(highOrderFlux, MPASO_EDGES, L * T);
    const int ofi = io.out(flxIn, MPASO_CELLS, L * T), ofo = io.out(flxOut, MPASO_CELLS, L * T);
    const int ote = io.out(tend, MPASO_CELLS, L * T);
    const int omx = io.out(tracerMax, MPASO_CELLS, L * T), omn = io.out(tracerMin, MPASO_CELLS, L * T);
    io.stage();
    const DMesh &d = io.dm();
    const cudaStream_t s = io.stream();
    with_tracers(T, [&](auto t) {
      k_oc_fct_a<t.value><<<blocks_for((int64_t)d.nE * L, TPB), TPB, 0, s>>>(d, L, io.ptr(intf), io.ptr(ilo),
                                                                            io.ptr(itr), io.ptr(oho));
      k_oc_fct_b<t.value><<<blocks_for((int64_t)d.nC * L, TPB), TPB, 0, s>>>(
          d, L, io.ptr(ihpi), io.ptr(ih), io.ptr(ilo), io.ptr(itr), io.ptr(oho), io.ptr(ofi), io.ptr(ofo),
          io.ptr(ote), io.ptr(omx), io.ptr(omn), dt);
      k_oc_fct_c<t.value><<<blocks_for((int64_t)d.nE * L, TPB), TPB, 0, s>>>(d, L, io.ptr(ofi), io.ptr(ofo),
                                                                            io.ptr(oho));
    });
    io.finish();
  });
}

int mpaso_oc_accumulate_horiz_tracer_advection_tend_mono_FCT(
    mpaso_mesh m, int32_t nlev, int32_t ntr, const double *hProvInv, const double *layerThickness,
    const double *highOrderFlux, const double *tracers, double *tracersProv, double *tend,
    double dt, void *stream) {
  return guarded("mpaso_oc_accumulate_horiz_tracer_advection_tend_mono_FCT", [&] {
    check_levels(nlev, ntr);
    TaskIO io(m, stream);
    require_fct(io, nlev);
    const int L = nlev, T = ntr;
    const int ihpi = io.in(hProvInv, MPASO_CELLS, L), ih = io.in(layerThickness, MPASO_CELLS, L);
    const int iho = io.in(highOrderFlux, MPASO_EDGES, L * T), itr = io.in(tracers, MPASO_CELLS, L * T);
    const int otp = io.out(tracersProv, MPASO_CELLS, L * T), ote = io.out(tend, MPASO_CELLS, L * T);
    io.stage();
    const DMesh &d = io.dm();
    with_tracers(T, [&](auto t) {
      k_oc_accumulate_fct<t.value><<<blocks_for((int64_t)d.nC * L, TPB), TPB, 0, io.stream()>>>(
          d, L, io.ptr(ihpi), io.ptr(ih), io.ptr(iho), io.ptr(itr), io.ptr(otp), io.ptr(ote), dt);
    });
    io.finish();
  });
}

int mpaso_oc_tracer_hmix_del2_tend(mpaso_mesh m, int32_t nlev, int32_t ntr,
                                   const double *layerThicknessEdge, const double *tracers,
                                   double *tend, double coef, void *stream) {
  return guarded("mpaso_oc_tracer_hmix_del2_tend", [&] {
    check_levels(nlev, ntr);
    TaskIO io(m, stream);
    const int L = nlev, T = ntr;
    const int ihe = io.in(layerThicknessEdge, MPASO_EDGES, L), itr = io.in(tracers, MPASO_CELLS, L * T);
    const int ote = io.out(tend, MPASO_CELLS, L * T);
    io.stage();
    const DMesh &d = io.dm();
    const size_t shared = (size_t)hmix_cells(L) * d.maxEoC * sizeof(double);  // at most 16 KB
    with_tracers(T, [&](auto t) {
      k_oc_hmix<t.value><<<blocks_for((int64_t)d.nC * L, TPB), TPB, shared, io.stream()>>>(
          d, L, io.ptr(ihe), io.ptr(itr), coef, io.ptr(ote));
    });
    io.finish();
  });
}

int mpaso_oc_step_tracers_forward(mpaso_mesh m, int32_t nlev, int32_t ntr, const double *tend,
                                  const double *tracers, double *tracersNew, double *tracersPrev,
                                  double rk_weight, double rk_subweight, void *stream) {
  return guarded("mpaso_oc_step_tracers_forward", [&] {
    check_levels(nlev, ntr);
    Flat f;
    f.s = plain_stream(m, stream), f.m = m;
    const size_t n = (size_t)m->ctx.d.nC * nlev * ntr;
    f.add(tend, n, false), f.add(tracers, n, false), f.add(tracersNew, n, true), f.add(tracersPrev, n, true);
    f.stage();
    k_oc_step_forward<<<blocks_for((int64_t)n, TPB), TPB, 0, f.s>>>(n, f.dev[0], f.dev[1], f.dev[2],
                                                                    f.dev[3], rk_weight, rk_subweight);
    f.finish();
  });
}

}  // extern "C"
