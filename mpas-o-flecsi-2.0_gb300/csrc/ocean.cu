// Fused RK4 tracer step of the ocean app (apps/ocean/run.cc:10-50): FCT
// horizontal advection with a prescribed velocity and layer thickness, plus
// del2 tracer mixing, on the renumbered HBM layout.
//
// The velocity and thickness never change, so the normal thickness flux
// (apps/ocean/tasks/solve.cc:40-57) and 1/hProv (solve.cc:60-97) are computed
// once per dt.  Each RK stage is then three launches:
//   K1 edges : low-order flux, anti-diffusive flux, del2 flux (solve.cc:99-167, 216-229, 328-366)
//   K2 cells : bounds, upwind tendency, limiter factors (solve.cc:194-267)
//   K3 cells : limited tendency, del2 tendency and step_tracers_forward
//              (solve.cc:269-326, 328-366, 368-399)
//
// Reference rounding.  These kernels evaluate every product, sum and quotient
// of the reference tasks in the reference's order, each rounded on its own
// (this file is compiled with -fmad=false and writes no fma), and divide where
// the reference divides.  Fusion only moves where a value is computed: an
// edge's fluxes are formed once and gathered by both cells, and a cell's
// sums run over its edges in the reference's edge order.  The only liberties
// are ones that cannot change a value: a product with a factor that is exactly
// zero is left out of a sum (x + 0 = x), a flux is added only to the one of
// flxIn / flxOut its sign selects (the other gains +0), and a clamped
// quotient whose numerator is <= 0 or >= its (positive) denominator is not
// divided out.  The result equals the reference task sequence value for value
// (signs of zero aside).  That is what the limiter needs: on tracer plateaus
// its quotient (max - upwind) / (dt flxIn / hProv + 1e-10) divides
// rounding-level differences by the regulariser, so any other rounding of the
// chain moves the step by far more than its own rounding.
//
// The FP64 pipe bounds these kernels (82-84% busy with every product and sum on
// it, the issue slots 10-24%), so the products run on the integer pipe
// (softmul.cuh, the same rounding; the sign of a zero aside) and only the sums on
// the FP64 pipe.  Level-6 sphere, 60 levels x 3 tracers, us per launch: oc_edges 1384 ->
// 630 (FP64, ALU and issue each 62-66% busy), oc_cells 659 -> 399, oc_final 484 ->
// 356 (451 and 363 with a branch to the hardware product after each slot; their
// registers are capped at 80 and 64, uncapped 448 and 371).
#include "rk4.cuh"
#include "softmul.cuh"

namespace mpaso {
namespace {

constexpr int TPB = 256;

// Statics of the ocean kernels in the reference's rounding (written over the
// state's cpm1 / kd after build_stat):
//   cpm1[a][e] = {advCoef + 0.25 advCoef_3rd, advCoef - 0.25 advCoef_3rd}, the
//     factor coef1 + coef3 sgn of solve.cc:150-153 for sgn = +1 / -1;
//   kd[e] = meshScalingDel2 kappa dvEdge / dcEdge (solve.cc:352), divided.
__global__ void k_oc_stat(DMesh m, double kappa, double2 *cpm, double *rho) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < (int64_t)m.maxAdv * m.nE) {
    const double coef1 = m.advCoef[i], coef3 = m.advCoef3[i] * 0.25;
    cpm[i] = make_double2(coef1 + coef3, coef1 - coef3);
  }
  if (i < m.nE) rho[i] = m.meshScalingDel2[i] * kappa * m.dvEdge[i] / m.dcEdge[i];
}

// F = u hE (solve.cc:49-54); hProv = h + sum_e (dt / area) dv edgeSign F in the
// cell's edge order, 1/hProv (solve.cc:73-95).  One launch, for small meshes.
__global__ void k_oc_prep(DMesh m, int L, const double *u, const double *h, const double *hE, double *F,
                          double *hpi, double dt) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t nEL = (int64_t)m.nE * L;
  if (i < nEL) {
    F[i] = u[i] * hE[i];
    return;
  }
  i -= nEL;
  if (i >= (int64_t)m.nC * L) return;
  const int c = (int)(i / L), k = (int)(i - (int64_t)c * L);
  const int n = m.nEoC[c];
  const double dtInvAreaCell = dt / m.areaCell[c];
  double hp = h[i];
  for (int j = 0; j < n; ++j) {
    const int64_t s = (int64_t)j * m.nC + c;
    const int e = m.eoc[s];
    const double sf = dtInvAreaCell * m.dvEdge[e] * m.eocSign[s];
    const int64_t ie = (int64_t)e * L + k;
    hp += sf * (u[ie] * hE[ie]);
  }
  hpi[i] = 1.0 / hp;
}

// The same in two launches, for meshes whose cell-levels fill every SM: F, and the
// factors (dt / area) dv edgeSign once per cell and slot instead of in each of
// its levels ...
__global__ void k_oc_prep_edges(DMesh m, int L, const double *u, const double *hE, double *F, double *sf, double dt) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t nEL = (int64_t)m.nE * L;
  if (i < nEL) {
    F[i] = mul_int(u[i], hE[i]);
    return;
  }
  i -= nEL;
  if (i >= (int64_t)m.maxEoC * m.nC) return;
  const int c = (int)(i % m.nC);
  sf[i] = (dt / m.areaCell[c]) * m.dvEdge[m.eoc[i]] * m.eocSign[i];  // pads: sign 0
}

// ... then hProv = h + sum_e sf F and 1/hProv.  Level 6, 60 levels: 37 + 62 us, and
// a step with its field exchange 5870 -> 5720 us against the one launch; on a 77 x
// 54 plane of 7 levels the second launch costs 4 us more than it saves.
__global__ void k_oc_prep_cells(DMesh m, int L, const double *h, const double *F, const double *sf, double *hpi) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= (int64_t)m.nC * L) return;
  const int c = (int)(i / L), k = (int)(i - (int64_t)c * L);
  const int n = m.nEoC[c];
  double hp = h[i];
  for (int j = 0; j < n; ++j) {
    const int64_t s = (int64_t)j * m.nC + c;
    hp += mul_int(F[(int64_t)m.eoc[s] * L + k], sf[s]);
  }
  hpi[i] = 1.0 / hp;
}

// K1: per edge-level, for every tracer, the low-order flux LO
// (solve.cc:106-116), the high-order flux corrected for FCT, A = HO - LO
// (solve.cc:143-165, 216-229), and the del2 flux DF = hE (tr2 - tr1) rho
// (solve.cc:350-356).  NA > 0: advection stencils of exactly NA slots (pads
// carry zero coefficients), unrolled; 0: the mesh's padded width at run time.
template <int T, int NA>
__global__ void __launch_bounds__(TPB) k_oc_edges(DMesh m, DStat st, Stage S, int L) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= (int64_t)m.nE * L) return;
  const int e = (int)(i / L), k = (int)(i - (int64_t)e * L);
  const int2 c = m.coe[e];
  const int64_t i1 = ((int64_t)c.x * L + k) * T, i2 = ((int64_t)c.y * L + k) * T;
  double t1[T], t2[T];
#pragma unroll
  for (int t = 0; t < T; ++t) t1[t] = S.tr_in[i1 + t], t2[t] = S.tr_in[i2 + t];
  if (S.fct) {
    const double f = S.F[i];
    const int mask = m.hoMask[(int64_t)e * m.fctLev + k];
    // wgtTmp = f mask (solve.cc:145): for a mask of 1 f itself, for 0 the zero
    // with f's sign, on the integer pipe (other masks: the product)
    const double wgt = mask == 1 ? f : mask == 0 ? bitsd(dbits(f) & kSignBit) : masked_weight(f, mask);
    // sgnTmp = sign(f) picks the factor coef1 + coef3 sgn; where f = 0 the
    // weight wgt is a zero and so is every weightFactor, whichever is picked
    const bool neg = dlt0(f);
    uint32_t badw = 0;
    const SoftFactor fw = soft_factor(wgt, badw);
    double flx[T];
    const int na = NA > 0 ? NA : m.maxAdv;
#pragma unroll
    for (int a = 0; a < na; ++a) {
      const int64_t sa = (int64_t)a * m.nE + e;
      const int cell = m.advCells[sa];
      const double2 cf2 = st.cpm1[sa];
      const double cf = neg ? cf2.y : cf2.x;
      const double *tr = S.tr_in + ((int64_t)cell * L + k) * T;
      // weightFactor wf = wgt cf (solve.cc:155), then tr wf for every tracer
      uint32_t bad = badw;
      const SoftFactor wf = soft_factor(soft_mul(cf, fw, bad), bad);
      double p[T];
#pragma unroll
      for (int t = 0; t < T; ++t) p[t] = soft_mul(tr[t], wf, bad);
      if (bad) {
        const double wx = product_outside(wgt, cf);
#pragma unroll
        for (int t = 0; t < T; ++t) p[t] = product_outside(tr[t], wx);
      }
      // the first term is the sum's start (0 + x = x)
#pragma unroll
      for (int t = 0; t < T; ++t) flx[t] = a ? flx[t] + p[t] : p[t];
    }
    const double dv = m.dvEdge[e];
    // LO = dv (max(0, f) tr1 + min(0, f) tr2): one of the two products is a zero
    const bool up1 = dgt0(f);
    // tracerWeight of solve.cc:222-223 is a zero on edges whose high-order mask
    // is set (their high-order flux gains nothing); on the others the centred
    // flux, with ((mask + 1) & 1) = 1
    if (!mask) {
#pragma unroll
      for (int t = 0; t < T; ++t) flx[t] = add_centred_flux(flx[t], dv, f, t1[t], t2[t]);
    }
    uint32_t badl = 0;
    const SoftFactor ff = soft_factor(f, badl), fdv = soft_factor(dv, badl);
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const double x = up1 ? t1[t] : t2[t];
      uint32_t bad = badl;
      double lo = soft_mul(soft_mul(x, ff, bad), fdv, bad);
      if (bad) lo = product_outside(dv, product_outside(f, x));
      S.LO[i * T + t] = lo;
      S.A[i * T + t] = flx[t] - lo;
    }
  }
  if (S.hmix) {
    const double hr = S.hE[i];
    const double rho = st.kd[e];
    uint32_t badm = 0;
    const SoftFactor fh = soft_factor(hr, badm), fr = soft_factor(rho, badm);
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const double d = t2[t] - t1[t];
      uint32_t bad = badm;
      double x = soft_mul(soft_mul(d, fh, bad), fr, bad);
      if (bad) x = product_outside(product_outside(hr, d), rho);
      S.DF[i * T + t] = x;
    }
  }
}

// The cell kernels form the products of a whole item without a branch between
// them, so that its loads and sums overlap; where one lay outside the integer
// products' window (softmul.cuh) the item's sums are formed again by these calls.
// (In K1, whose integer work already equals its FP64 work, zero factors would
// have to be handled in line for that: 627 -> 666 us.)
__device__ __noinline__ double product3_outside(double a, double b, double c) { return a * b * c; }

// K2's sums over a cell's edges in hardware products.
struct CellSums {
  double td, fi, fo;
};
__device__ __noinline__ CellSums cell_sums_outside(const int *eoc, const double *sign, const double *LO,
                                                   const double *A, int nC, int c, int n, int64_t off, int64_t row,
                                                   double inva) {
  CellSums r{0.0, 0.0, 0.0};
  for (int j = 0; j < n; ++j) {
    const int64_t s = (int64_t)j * nC + c, ie = eoc[s] * row + off;
    const long long sm = sign_mask(sign[s]);
    r.td += dflip(inva * LO[ie], sm);
    const double ax = dflip(inva * A[ie], sm);
    if (dgt0(ax))
      r.fi += ax;
    else
      r.fo += ax;
  }
  return r;
}

// K2: per cell-level, for every tracer, the bounds over the cell and its
// neighbours (solve.cc:194-214), the upwind tendency and flxIn / flxOut over
// the cell's edges (solve.cc:232-249) and the limiter factors R+ / R-
// (solve.cc:251-265).  Writes R2 = {R+, R-} and tLO = the upwind tendency
// (divided by the area, as the reference's tend holds it).
template <int T, int NC>
__global__ void __launch_bounds__(TPB, 3) k_oc_cells(DMesh m, Stage S, int L) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= (int64_t)m.nC * L || !S.fct) return;
  const int c = (int)(i / L), k = (int)(i - (int64_t)c * L);
  const int n = m.nEoC[c];
  const double invAreaCell1 = m.invAreaCell[c];  // 1 / areaCell
  uint32_t bad = 0;
  const SoftFactor fa = soft_factor(invAreaCell1, bad);
  double trc[T], mx[T], mn[T], td[T], fi[T], fo[T];
#pragma unroll
  for (int t = 0; t < T; ++t) {
    trc[t] = S.tr_in[i * T + t];
    mx[t] = trc[t], mn[t] = trc[t], td[t] = 0.0, fi[t] = 0.0, fo[t] = 0.0;
  }
  for_slots<NC>(n, [&](int j, bool ok) {
    const int64_t s = (int64_t)j * m.nC + c;
    const int64_t in0 = ((int64_t)m.coc[s] * L + k) * T;  // pads: the cell itself
    const int64_t ie0 = ((int64_t)m.eoc[s] * L + k) * T;  // pads: slot 0, masked
    const long long sm = sign_mask(m.eocSign[s]);  // signedFactor = +-invAreaCell1
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const double x = S.tr_in[in0 + t];
      mx[t] = dmax(mx[t], x);
      mn[t] = dmin(mn[t], x);
      const double pl = dflip(soft_mul(dmask(S.LO[ie0 + t], ok), fa, bad), sm);
      const double ax = dflip(soft_mul(dmask(S.A[ie0 + t], ok), fa, bad), sm);
      // flxIn += max(0, ax), flxOut += min(0, ax): one add into the sum the
      // sign selects (integer-pipe selects; a zero ax changes neither sum,
      // so none is kept), instead of an add in each of two divergent branches
      // (the first terms are the sums' starts)
      const bool in = dgt0(ax), out = dlt0(ax);
      if (j == 0) {
        td[t] = pl;
        fi[t] = in ? ax : 0.0;
        fo[t] = out ? ax : 0.0;
      } else {
        td[t] += pl;
        const double acc = opaque(in ? fi[t] : fo[t]) + ax;
        fi[t] = in ? acc : fi[t];
        fo[t] = out ? acc : fo[t];
      }
    }
  });
  if (bad) {
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const CellSums r = cell_sums_outside(m.eoc, m.eocSign, S.LO, S.A, m.nC, c, n, (int64_t)k * T + t, (int64_t)L * T,
                                           invAreaCell1);
      td[t] = r.td, fi[t] = r.fi, fo[t] = r.fo;
    }
  }
  const double h = S.h_in[i], hpi = S.hpi[i], dt = S.dt;
  const double eps = 1.e-10;
  uint32_t badh = 0;
  const SoftFactor fh = soft_factor(h, badh), fp = soft_factor(hpi, badh), fdt = soft_factor(dt, badh);
#pragma unroll
  for (int t = 0; t < T; ++t) {
    // tracerUpwindNew, and what tracerMaxNew / tracerMinNew add to it
    uint32_t out = badh;
    double up = soft_mul(soft_mul(trc[t], fh, out) + soft_mul(td[t], fdt, out), fp, out);
    double di = soft_mul(soft_mul(fi[t], fdt, out), fp, out), dn = soft_mul(soft_mul(fo[t], fdt, out), fp, out);
    if (out) {
      up = product_outside(product_outside(trc[t], h) + product_outside(dt, td[t]), hpi);
      di = product3_outside(dt, fi[t], hpi), dn = product3_outside(dt, fo[t], hpi);
    }
    const double mxn = up + di, mnn = up + dn;
    const double rp = clamp_quotient(mx[t] - up, (mxn - up) + eps);
    const double rm = clamp_quotient(up - mn[t], (up - mnn) + eps);
    S.R2[i * T + t] = make_double2(rp, rm);
    S.tLO[i * T + t] = td[t];
  }
}

// K3's tendency in hardware products: the upwind part td plus the limited fluxes
// (A null: none) minus the del2 fluxes (DF null: none) of a cell's edges.
__device__ __noinline__ double cell_tend_outside(const int *eoc, const int *nbr, const double *sign, const double *A,
                                                 const double2 *R2, const double *DF, int nC, int c, int n,
                                                 int64_t off, int64_t row, double2 own, double inva, double td) {
  for (int j = 0; A && j < n; ++j) {
    const int64_t s = (int64_t)j * nC + c;
    const int nb = nbr[s];
    const double a = A[eoc[s] * row + off];
    const double2 o = R2[(nb >> 1) * row + off];
    const double2 r1 = nb & 1 ? own : o, r2 = nb & 1 ? o : own;
    const double r = dgt0(a) ? dmin(r1.y, r2.x) : dmin(r1.x, r2.y);
    td += dflip(inva * ((dgt0(a) || dlt0(a) ? a : 0.0) * r), sign_mask(sign[s]));
  }
  for (int j = 0; DF && j < n; ++j) {
    const int64_t s = (int64_t)j * nC + c;
    td -= dflip(DF[eoc[s] * row + off] * inva, sign_mask(sign[s]));
  }
  return td;
}

// K3: per cell-level, for every tracer, the tendency: the upwind part, the
// limited anti-diffusive fluxes (solve.cc:270-282, 296-309) and the del2
// mixing (solve.cc:340-364), each summed over the cell's edges in order, then
// step_tracers_forward (solve.cc:368-399).  The limited flux of an edge,
// max(0, A) min(R-(c1), R+(c2)) + min(0, A) min(R+(c1), R-(c2)) with
// (c1, c2) = cells(e), is A times the one minimum its sign selects.
template <int T, int NC>
__global__ void __launch_bounds__(TPB, 4) k_oc_final(DMesh m, Stage S, int L) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= (int64_t)m.nC * L) return;
  const int c = (int)(i / L), k = (int)(i - (int64_t)c * L);
  const int n = m.nEoC[c];
  const double invAreaCell1 = m.invAreaCell[c];
  double td[T];
  double2 own[T];
#pragma unroll
  for (int t = 0; t < T; ++t) {
    td[t] = S.fct ? S.tLO[i * T + t] : 0.0;
    if (S.fct) own[t] = S.R2[i * T + t];
  }
  uint32_t bad = 0;
  const SoftFactor fa = soft_factor(invAreaCell1, bad);
  if (S.fct) {
    for_slots<NC>(n, [&](int j, bool ok) {
      const int64_t s = (int64_t)j * m.nC + c;
      const long long sm = sign_mask(m.eocSign[s]);
      const int nb = m.nbr[s];
      const bool first = nb & 1;  // c is cells(e)[0]
      const int64_t ie0 = ((int64_t)m.eoc[s] * L + k) * T, jn = ((int64_t)(nb >> 1) * L + k) * T;
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const double a = dmask(S.A[ie0 + t], ok);
        const double2 o = S.R2[jn + t];
        const double2 r1 = first ? own[t] : o, r2 = first ? o : own[t];  // {R+, R-} of c1, c2
        // one product with the minimum the sign selects (integer-pipe selects);
        // a zero flux enters as +0, whose products are the +0 the reference's
        // max(0, A) / min(0, A) terms give
        // (a zero factor -- local extrema -- makes the flux the zero, the other 1,
        // unless the flux is infinite or NaN, which zero does not make a zero)
        const bool pos = dgt0(a);
        const double rmin = pos ? dmin(r1.y, r2.x) : dmin(r1.x, r2.y);
        const bool some = dgt0(rmin) || nonfinite(a);
        const double a0 = some && (pos || dlt0(a)) ? a : 0.0, r0 = some ? rmin : 1.0;
        td[t] += dflip(soft_mul(soft_mul(a0, soft_factor(r0, bad), bad), fa, bad), sm);
      }
    });
  }
  if (S.hmix) {
    for_slots<NC>(n, [&](int j, bool ok) {
      const int64_t s = (int64_t)j * m.nC + c;
      const long long sm = sign_mask(m.eocSign[s]);
      const int64_t ie0 = ((int64_t)m.eoc[s] * L + k) * T;
#pragma unroll
      for (int t = 0; t < T; ++t) td[t] -= dflip(soft_mul(dmask(S.DF[ie0 + t], ok), fa, bad), sm);
    });
  }
  if (bad) {
#pragma unroll
    for (int t = 0; t < T; ++t)
      td[t] = cell_tend_outside(m.eoc, m.nbr, m.eocSign, S.fct ? S.A : nullptr, S.R2, S.hmix ? S.DF : nullptr, m.nC, c,
                                n, (int64_t)k * T + t, (int64_t)L * T, S.fct ? own[t] : make_double2(0.0, 0.0),
                                invAreaCell1, S.fct ? S.tLO[i * T + t] : 0.0);
  }
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const int64_t j = i * T + t;
    const double cur = S.tr_prev[j];
    switch (S.stage) {  // tracersNew += w tend; tracersPrev = tracers + w_sub tend
      case 0:
        S.trh_acc[j] = cur + mul_int(td[t], S.w_acc);
        S.tr_out[j] = cur + mul_int(td[t], S.w_sub);
        break;
      case 3:
        S.tr_new[j] = S.trh_acc[j] + mul_int(td[t], S.w_acc);
        break;
      default:
        S.trh_acc[j] = S.trh_acc[j] + mul_int(td[t], S.w_acc);
        S.tr_out[j] = cur + mul_int(td[t], S.w_sub);
    }
  }
}

Stage ocean_stage(SwState &s, int rk, double dt) {
  const double rk_w[4] = {dt / 6, dt / 3, dt / 3, dt / 6};  // apps/ocean/run.cc:15-16
  const double rk_sub[4] = {dt / 2, dt / 2, dt, 0};
  Stage S{};
  S.stage = rk, S.w_sub = rk_sub[rk], S.w_acc = rk_w[rk], S.dt = dt;
  S.fct = s.p.fct, S.hmix = s.p.hmix;
  double *trs[4] = {s.TR0, s.TRA, s.TRB, s.TRA};
  S.tr_in = trs[rk];
  S.tr_out = rk < 3 ? trs[rk + 1] : nullptr;
  S.tr_prev = s.TR0, S.trh_acc = s.TRH, S.tr_new = s.TR0;
  S.h_in = s.H[0], S.u_in = s.U[0];
  S.F = s.F, S.A = s.A, S.LO = s.LO, S.DF = s.DF, S.R2 = s.R2, S.tLO = s.tLO;
  S.hE = s.HE, S.hpi = s.HPI;
  return S;
}

template <int T> void ocean_stage_T(SwState &s, const Stage &S, cudaStream_t st) {
  const DMesh &m = s.mesh->ctx.d;
  const int L = s.L;
  cudaEvent_t *ev = s.prof_events;
  const int b0 = stage_tpb(s, 0), b1 = stage_tpb(s, 1), b2 = stage_tpb(s, 2);
  if (m.maxAdv == 10 && s.tune_unroll[0])
    k_oc_edges<T, 10><<<blocks_for((int64_t)m.nE * L, b0), b0, 0, st>>>(m, s.st, S, L);
  else
    k_oc_edges<T, 0><<<blocks_for((int64_t)m.nE * L, b0), b0, 0, st>>>(m, s.st, S, L);
  if (ev) prof_mark(ev[0], st);
  const bool c6 = m.maxEoC <= 6;
  if (c6 && s.tune_unroll[1])
    k_oc_cells<T, 6><<<blocks_for((int64_t)m.nC * L, b1), b1, 0, st>>>(m, S, L);
  else
    k_oc_cells<T, 0><<<blocks_for((int64_t)m.nC * L, b1), b1, 0, st>>>(m, S, L);
  if (ev) prof_mark(ev[1], st);
  if (c6 && s.tune_unroll[2])
    k_oc_final<T, 6><<<blocks_for((int64_t)m.nC * L, b2), b2, 0, st>>>(m, S, L);
  else
    k_oc_final<T, 0><<<blocks_for((int64_t)m.nC * L, b2), b2, 0, st>>>(m, S, L);
  if (ev) prof_mark(ev[2], st);
}

}  // namespace

void ocean_create(SwState &s) {
  const DMesh &m = s.mesh->ctx.d;
  const int64_t L = s.L, T = s.T, nC = m.nC, nE = m.nE;
  std::vector<std::pair<double **, int64_t>> bufs = {
      {&s.U[0], nE * L}, {&s.H[0], nC * L}, {&s.HE, nE * L}, {&s.HPI, nC * L},
      {&s.TR0, nC * L * T}, {&s.TRA, nC * L * T}, {&s.TRB, nC * L * T}, {&s.TRH, nC * L * T},
      {&s.F, nE * L}, {&s.A, nE * L * T}, {&s.LO, nE * L * T}, {&s.DF, nE * L * T},
      {(double **)&s.R2, 2 * nC * L * T}, {&s.tLO, nC * L * T}, {&s.SF, (int64_t)m.maxEoC * nC}};
  stat_buffers(s, bufs);
  alloc_arena(s, bufs);
  build_stat(s);
  const int64_t n = std::max<int64_t>((int64_t)m.maxAdv * nE, nE);
  k_oc_stat<<<blocks_for(n, TPB), TPB, 0, s.stream>>>(m, s.p.kappa, (double2 *)s.st.cpm1, (double *)s.st.kd);
  MPASO_CUDA(cudaGetLastError());
}

void ocean_recompute(SwState &s, double dt, cudaStream_t st);

void ocean_prepare(SwState &s, double dt, cudaStream_t st) {
  if (s.prep_dt != dt) ocean_recompute(s, dt, st);
}

// Thickness flux and 1/hProv of the stored (h, u), unconditionally (also from
// inside a stream capture, after new h / u were gathered in).
void ocean_recompute(SwState &s, double dt, cudaStream_t st) {
  const DMesh &m = s.mesh->ctx.d;
  if ((int64_t)m.nC * s.L < 1024LL * s.mesh->ctx.sms) {
    k_oc_prep<<<blocks_for(((int64_t)m.nE + m.nC) * s.L, TPB), TPB, 0, st>>>(m, s.L, s.U[0], s.H[0], s.HE, s.F,
                                                                          s.HPI, dt);
  } else {
    k_oc_prep_edges<<<blocks_for((int64_t)m.nE * s.L + (int64_t)m.maxEoC * m.nC, TPB), TPB, 0, st>>>(
        m, s.L, s.U[0], s.HE, s.F, s.SF, dt);
    k_oc_prep_cells<<<blocks_for((int64_t)m.nC * s.L, TPB), TPB, 0, st>>>(m, s.L, s.H[0], s.F, s.SF, s.HPI);
  }
  MPASO_CUDA(cudaGetLastError());
  s.prep_dt = dt;
}

void ocean_one_stage(SwState &s, int rk, double dt, cudaStream_t st) {
  const Stage S = ocean_stage(s, rk, dt);
  switch (s.T) {
    case 1: ocean_stage_T<1>(s, S, st); break;
    case 2: ocean_stage_T<2>(s, S, st); break;
    case 3: ocean_stage_T<3>(s, S, st); break;
    case 4: ocean_stage_T<4>(s, S, st); break;
    case 5: ocean_stage_T<5>(s, S, st); break;
    case 6: ocean_stage_T<6>(s, S, st); break;
    case 7: ocean_stage_T<7>(s, S, st); break;
    case 8: ocean_stage_T<8>(s, S, st); break;
    default: fail(MPASO_ERR_ARG, "ocean app needs 1..8 tracers");
  }
}

void ocean_steps(SwState &s, double dt, int nsteps, cudaStream_t st) {
  ocean_prepare(s, dt, st);
  for (int n = 0; n < nsteps; ++n)
    for (int rk = 0; rk < 4; ++rk) ocean_one_stage(s, rk, dt, st);
  MPASO_CUDA(cudaGetLastError());
}

int ocean_launches_per_step(const SwState &) { return 12; }

// A stage with the state's weights and buffers, and its launch, for callers
// that redirect some of its pointers (the adjoint's taping recompute).
Stage ocean_make_stage(SwState &s, int rk, double dt) { return ocean_stage(s, rk, dt); }
void ocean_launch_stage(SwState &s, const Stage &S, cudaStream_t st) {
  switch (s.T) {
    case 1: ocean_stage_T<1>(s, S, st); break;
    case 2: ocean_stage_T<2>(s, S, st); break;
    case 3: ocean_stage_T<3>(s, S, st); break;
    case 4: ocean_stage_T<4>(s, S, st); break;
    case 5: ocean_stage_T<5>(s, S, st); break;
    case 6: ocean_stage_T<6>(s, S, st); break;
    case 7: ocean_stage_T<7>(s, S, st); break;
    case 8: ocean_stage_T<8>(s, S, st); break;
    default: fail(MPASO_ERR_ARG, "ocean app needs 1..8 tracers");
  }
}

}  // namespace mpaso
