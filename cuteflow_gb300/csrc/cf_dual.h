/*
 * cf_dual.h -- forward-mode dual numbers for the discrete adjoint.
 *
 * Dual<N> carries a value and N directional derivatives.  The value lane performs exactly the
 * IEEE operations the plain FP64 forward performs (same order, no contraction: the kernels are
 * compiled with -fmad=false), so comparisons taken on values select the same branches as the
 * forward step, and the derivative lanes are the exact local derivatives of that branch.  The
 * templated step arithmetic (cf_flux.h) instantiated with Dual<N> therefore yields the local
 * Jacobians the reverse sweep needs (dt frozen).
 */
#ifndef CF_DUAL_H
#define CF_DUAL_H

#include "cf_flux.h"
#include "cf_xd.h"

#ifdef __CUDACC__
#define CFD_HD __host__ __device__ __forceinline__
#else
#define CFD_HD inline
#endif

namespace cf {

#ifdef __CUDACC__
using ::fabs;
using ::sqrt;
#endif

template <int N>
struct Dual {
  double v;
  double d[N];
  CFD_HD Dual() : v(0.0) {
#pragma unroll
    for (int i = 0; i < N; ++i) d[i] = 0.0;
  }
  CFD_HD Dual(double x) : v(x) {  // NOLINT: constants promote implicitly
#pragma unroll
    for (int i = 0; i < N; ++i) d[i] = 0.0;
  }
  /* the i-th independent variable with value x */
  static CFD_HD Dual var(double x, int i) {
    Dual r(x);
    r.d[i] = 1.0;
    return r;
  }
};

template <int N>
CFD_HD double val(const Dual<N>& x) { return x.v; }

template <int N>
CFD_HD Dual<N> operator-(const Dual<N>& a) {
  Dual<N> r;
  r.v = -a.v;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = -a.d[i];
  return r;
}
template <int N>
CFD_HD Dual<N> operator+(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r;
  r.v = a.v + b.v;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] + b.d[i];
  return r;
}
template <int N>
CFD_HD Dual<N> operator-(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r;
  r.v = a.v - b.v;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] - b.d[i];
  return r;
}
template <int N>
CFD_HD Dual<N> operator*(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r;
  r.v = a.v * b.v;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = fma(a.d[i], b.v, a.v * b.d[i]);
  return r;
}
/* a / b: the value lane is the IEEE quotient and the derivative lanes use the reciprocal, both
 * from the integer-pipe division of cf_xd.h (the FP64 pipe keeps the lanes' FMAs) */
template <int N>
CFD_HD Dual<N> operator/(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r;
  const double y = em_div(1.0, b.v);
  r.v = em_div(a.v, b.v);
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = fma(-r.v, b.d[i], a.d[i]) * y;
  return r;
}
/* mixed with constants */
template <int N> CFD_HD Dual<N> operator+(const Dual<N>& a, double b) { Dual<N> r = a; r.v = a.v + b; return r; }
template <int N> CFD_HD Dual<N> operator+(double a, const Dual<N>& b) { Dual<N> r = b; r.v = a + b.v; return r; }
template <int N> CFD_HD Dual<N> operator-(const Dual<N>& a, double b) { Dual<N> r = a; r.v = a.v - b; return r; }
template <int N>
CFD_HD Dual<N> operator-(double a, const Dual<N>& b) {
  Dual<N> r;
  r.v = a - b.v;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = -b.d[i];
  return r;
}
template <int N>
CFD_HD Dual<N> operator*(const Dual<N>& a, double b) {
  Dual<N> r;
  r.v = a.v * b;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] * b;
  return r;
}
template <int N>
CFD_HD Dual<N> operator*(double a, const Dual<N>& b) {
  Dual<N> r;
  r.v = a * b.v;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = a * b.d[i];
  return r;
}
template <int N>
CFD_HD Dual<N> operator/(const Dual<N>& a, double b) {
  Dual<N> r;
  r.v = a.v / b;  /* mostly constants (/ 2, / 4), which the compiler folds */
  const double y = 1.0 / b;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] * y;
  return r;
}
template <int N>
CFD_HD Dual<N> operator/(double a, const Dual<N>& b) {
  Dual<N> r;
  r.v = em_div(a, b.v);
  const double y = em_div(1.0, b.v);
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = -r.v * b.d[i] * y;
  return r;
}
/* comparisons act on values, on the ordered integer keys of cf_xd.h (the IEEE results: NaN
 * compares false, -0 equals +0), which keeps them off the FP64 pipe the derivative lanes use */
template <int N> CFD_HD bool operator<(const Dual<N>& a, const Dual<N>& b) { return xlt(a.v, b.v); }
template <int N> CFD_HD bool operator>(const Dual<N>& a, const Dual<N>& b) { return xlt(b.v, a.v); }
template <int N> CFD_HD bool operator<=(const Dual<N>& a, const Dual<N>& b) { return xle(a.v, b.v); }
template <int N> CFD_HD bool operator>=(const Dual<N>& a, const Dual<N>& b) { return xle(b.v, a.v); }
template <int N> CFD_HD bool operator<(const Dual<N>& a, double b) { return xlt_c(a.v, b); }
template <int N> CFD_HD bool operator>(const Dual<N>& a, double b) { return xgt_c(a.v, b); }
template <int N> CFD_HD bool operator<=(const Dual<N>& a, double b) { return xle_c(a.v, b); }
template <int N> CFD_HD bool operator>=(const Dual<N>& a, double b) { return xle(b, a.v); }
template <int N> CFD_HD bool operator<(double a, const Dual<N>& b) { return xgt_c(b.v, a); }
template <int N> CFD_HD bool operator>(double a, const Dual<N>& b) { return xlt_c(b.v, a); }
template <int N> CFD_HD bool lt_nonneg(const Dual<N>& a, const Dual<N>& b) { return xlt_nonneg(a.v, b.v); }
template <int N> CFD_HD bool operator!=(const Dual<N>& a, double b) { return !xeq(a.v, b); }
template <int N> CFD_HD bool operator==(const Dual<N>& a, const Dual<N>& b) { return xeq(a.v, b.v); }
template <int N> CFD_HD bool operator!=(const Dual<N>& a, const Dual<N>& b) { return !xeq(a.v, b.v); }

template <int N>
CFD_HD Dual<N> sqrt(const Dual<N>& a) {
  Dual<N> r;
  r.v = em_sqrt(a.v);
  const double y = r.v > 0.0 ? em_div(0.5, r.v) : 0.0; /* sqrt(0) only where the depth is exactly zero */
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] * y;
  return r;
}
template <int N>
CFD_HD Dual<N> fabs(const Dual<N>& a) {
  return (a.v < 0.0) ? -a : a;
}

/* the reciprocal of a depth with its derivative (the stored RN(1/h) carries none) */
template <int N>
CFD_HD Dual<N> recip_h(const Dual<N>& h, double) { return 1.0 / h; }

/* Quotient by a known reciprocal (div_rn in cf_flux.h): the value lane is the step's own
 * rounding; the lanes differentiate a / d. */
template <int N>
CFD_HD Dual<N> div_rn(const Dual<N>& a, const Dual<N>& d, const Dual<N>& y) {
  Dual<N> r;
  r.v = em_div(a.v, d.v);  /* the IEEE quotient, as div_rn's */
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = fma(-r.v, d.d[i], a.d[i]) * y.v;
  return r;
}
template <int N>
CFD_HD Dual<N> div_rn(const Dual<N>& a, double d, double y) {
  Dual<N> r;
  r.v = em_div(a.v, d);
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] * y;
  return r;
}

/* x^(-1/3): d/dx = -r / (3 x) with r = x^(-1/3) */
template <int N>
CFD_HD Dual<N> rcbrt(const Dual<N>& x) {
  Dual<N> r;
  r.v = rcbrt(x.v);
  const double k = -em_div(r.v, 3.0 * x.v);
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = x.d[i] * k;
  return r;
}

/* a b + c in one FP64 instruction (derivatives only: values round every operation) */
CFD_HD XD<true> xfma(const XD<true>& a, const XD<true>& b, const XD<true>& c) { return XD<true>(fma(a.v, b.v, c.v)); }

/* The transposed edge stage of an interior first-order HLLC edge (IFLUX 1, flux_mode 0): given the
 * adjoint weights w[10] of its two slots (side A: flux 1-3, bed x, y; then side B), the
 * contributions lamA, lamB to the adjoints of (h, hu, hv) of its two elements, i.e. J^T w for the
 * edge's Jacobian J, by the chain rule backwards through the flux's own formulas:
 *   - the rotation of both sides' frame fluxes (x1, x2, x3), with x3 = x1 v in every region, v the
 *     tangential velocity the region takes;
 *   - the HLL fluxes N / (s_R - s_L + eps) or the physical flux the region takes;
 *   - the speeds s_L = u_l - a_l p_l, s_R = u_r + a_r p_r with p = 1 or sqrt((h* + h) h* / 2) / h, and
 *     the depth h* = (h_l + h_r) / 2 - (u_r - u_l) (h_l + h_r) / (a_l + a_r) / 4; next to a dry side
 *     s = u -+ a and u +- 2 a of the wet one;
 *   - the hydrostatic reconstruction (depths pass or are clamped to 0), the change to the edge frame
 *     (u_n = (hu nx + hv ny) / h, u_t = (hv nx - hu ny) / h) and the bed sources g/2 (ha^2 - h^2) len.
 * The values repeat the step's IEEE operations (so every branch is the forward's), their products,
 * quotients and roots on the integer pipes; of the derivatives the multiply-adds are FP64
 * instructions and the products integer ones.  Returns false, and the caller differentiates the edge
 * in full, where a side's raw and masked depths differ (0 < h <= tolisec; the reference then evaluates
 * the two sides differently). */
CFD_HD bool adj_edge_hllc(const MemberDev& M, const EdgeGeo& G, const double4& UA, const double4& UB, double zml,
                          double zmr, const double w[10], double lamA[3], double lamB[3]) {
  typedef XD<true> X;
  const double g = M.gp, tolisec = M.tolisec, nx = G.nx, ny = G.ny, eps = EPS_HLLC;
  const X hA(UA.x), hB(UB.x);
  const bool wa = hA > tolisec, wb = hB > tolisec;   /* frame velocities differentiable */
  if ((!wa && hA != 0.0) || (!wb && hB != 0.0)) return false;
  const double zij = val(dmax(X(zml), X(zmr)));
  X hm, ul, vl, ur, vr;
  to_frame(hA, X(UA.y), X(UA.z), UA.w, nx, ny, tolisec, hm, ul, vl);
  to_frame(hB, X(UB.y), X(UB.z), UB.w, nx, ny, tolisec, hm, ur, vr);
  const X ul0 = ul, vl0 = vl, ur0 = ur, vr0 = vr;
  /* hydrostatic reconstruction (flux_riemann.cuf:176-181, :200-210); which variables carry a
   * derivative (a clamped or masked one is a constant of the inputs) */
  const X ea = hA + zml - zij, eb = hB + zmr - zij;
  const X ha = dmax0(ea), hb = dmax0(eb);
  X hl = wa ? ha : X(0.0), hr = hb;
  const bool pl = !(hl < tolisec), pr = !(hr < tolisec);
  if (!pl) { hl = X(0.); ul = X(0.); vl = X(0.); }
  if (!pr) { hr = X(0.); ur = X(0.); vr = X(0.); }
  const bool s_hl = pl && wa && ea > 0., s_ul = pl && wa, s_hr = pr && eb > 0., s_ur = pr && wb;
  X ghl(0.0), gul(0.0), gvl(0.0), ghr(0.0), gur(0.0), gvr(0.0);   /* adjoints (without the factor len) */
  if (!(hl < eps && hr < eps)) {
    /* the flux's values, as wave_speeds and first_order_flux<1> form them */
    const X gl = g * hl, gr = g * hr, al = sqrt(gl), ar = sqrt(gr);
    const X hs = hl + hr, du = ur - ul, as = al + ar;
    const X qd = du * hs / as;
    const X het = halve(hs) - quarter(qd);
    const bool wl = hl > eps, wr = hr > eps, both = wl && wr;
    const bool kl = both && !lt_nonneg(het, hl), kr = both && !lt_nonneg(het, hr);
    const X hll2 = hl * hl, hrr2 = hr * hr;
    const X pql = kl ? sqrt(halve(het + hl) * het / hll2) : X(1.), pqr = kr ? sqrt(halve(het + hr) * het / hrr2) : X(1.);
    X sl, sr;
    if (wl) {
      sl = ul - (both ? al * pql : al);
      sr = wr ? ur + ar * pqr : ul + twice(al);
    } else {
      sl = ur - twice(ar);
      sr = ur + ar;
    }
    const X fl1 = hl * ul, fl2 = hl * (ul * ul) + halve(gl * hl);
    const X fr1 = hr * ur, fr2 = hr * (ur * ur) + halve(gr * hr);
    const int ra = (sl > 0.) ? 0 : ((sr < 0.) ? 1 : 2);
    const int rb = (sr < 0.) ? 1 : ((sl > 0.) ? 0 : 2);
    /* s* decides which tangential velocity the HLL region carries */
    bool right_a = ra == 1, right_b = rb == 1;
    if (ra == 2 || rb == 2) {
      const X d1 = hr * (ur - sr), d0 = hl * (ul - sl), denom = d1 - d0;
      X set;
      if (fabs(denom) < eps) set = halve(ul + ur) - (hr - hl) * as / hs;
      else set = (sl * hr * (ur - sr) - sr * hl * (ul - sl)) / denom;
      if (ra == 2) right_a = !(set > 0.);
      if (rb == 2) right_b = set < 0.;
    }
    /* adjoints of x1, x2 (side A) and y1, y2 (side B, whose frame flux is (-y1, y2, y1 v) mirrored) */
    const X ta = xfma(X(w[2]), X(nx), -(X(w[1]) * ny)), tb = xfma(X(w[7]), X(nx), -(X(w[6]) * ny));
    const X ga2 = xfma(X(w[1]), X(nx), X(w[2]) * ny), gb2 = -xfma(X(w[6]), X(nx), X(w[7]) * ny);
    const X ga1 = xfma(right_a ? vr : vl, ta, X(w[0])), gb1 = -xfma(right_b ? vr : vl, tb, X(w[5]));
    X gfl1(0.0), gfl2(0.0), gfr1(0.0), gfr2(0.0), gsl(0.0), gsr(0.0), m1(0.0);
    if (ra == 2 || rb == 2) {
      const X gh1 = (ra == 2 && rb == 2) ? ga1 + gb1 : (ra == 2 ? ga1 : gb1);
      const X gh2 = (ra == 2 && rb == 2) ? ga2 + gb2 : (ra == 2 ? ga2 : gb2);
      const X y = 1.0 / (sr - sl + eps);
      const X dh = hr - hl, df = fr1 - fl1, ss = sl * sr;
      const X c1 = xfma(sl, dh, fl1), c2 = xfma(sl, df, fl2), e1 = xfma(sr, dh, -fr1), e2 = xfma(sr, df, -fr2);
      m1 = xfma(sr, c1, -(sl * fr1)) * y;
      const X m2 = xfma(sr, c2, -(sl * fr2)) * y;
      const X n1 = gh1 * y, n2 = gh2 * y;
      const X gd = -xfma(n1, m1, n2 * m2);
      gsr = xfma(n1, c1, xfma(n2, c2, gd));
      gsl = xfma(n1, e1, xfma(n2, e2, -gd));
      const X q1 = n1 * ss, q2 = n2 * ss;
      gfl1 = xfma(n1, sr, -q2);
      gfr1 = xfma(-n1, sl, q2);
      gfl2 = n2 * sr;
      gfr2 = -(n2 * sl);
      ghl = -q1;
      ghr = q1;
    }
    if (ra == 0) { gfl1 = gfl1 + ga1; gfl2 = gfl2 + ga2; }
    if (ra == 1) { gfr1 = gfr1 + ga1; gfr2 = gfr2 + ga2; }
    if (rb == 0) { gfl1 = gfl1 + gb1; gfl2 = gfl2 + gb2; }
    if (rb == 1) { gfr1 = gfr1 + gb1; gfr2 = gfr2 + gb2; }
    /* tangential velocities: x1 ta on side A, -y1 tb on side B */
    const X va = (ra == 0 ? fl1 : (ra == 1 ? fr1 : m1)) * ta, vb = -((rb == 0 ? fl1 : (rb == 1 ? fr1 : m1)) * tb);
    if (right_a == right_b) (right_a ? gvr : gvl) = va + vb;
    else { gvl = right_a ? vb : va; gvr = right_a ? va : vb; }
    /* physical fluxes: f1 = h u, f2 = h u^2 + g h^2 / 2 */
    ghl = xfma(gfl1, ul, xfma(gfl2, xfma(ul, ul, gl), ghl));
    gul = xfma(gfl1, hl, twice(gfl2 * fl1));
    ghr = xfma(gfr1, ur, xfma(gfr2, xfma(ur, ur, gr), ghr));
    gur = xfma(gfr1, hr, twice(gfr2 * fr1));
    /* speeds */
    X gal(0.0), gar(0.0);
    if (both) {
      gul = gul + gsl;
      gur = gur + gsr;
      gal = -(gsl * pql);
      gar = gsr * pqr;
      if (kl || kr) {
        /* p^2 = P = (h* + h) h* / 2 / h^2: dP/dh* = (h* + h / 2) / h^2, dP/dh = (h* / 2 - 2 P h) / h^2 */
        X ghet(0.0);
        if (kl) {
          const X gp = -(gsl * al) / (twice(pql) * hll2);
          ghet = gp * (het + halve(hl));
          ghl = xfma(gp, xfma(-twice(pql * pql), hl, halve(het)), ghl);
        }
        if (kr) {
          const X gp = gsr * ar / (twice(pqr) * hrr2);
          ghet = xfma(gp, het + halve(hr), ghet);
          ghr = xfma(gp, xfma(-twice(pqr * pqr), hr, halve(het)), ghr);
        }
        /* h* */
        const X q = quarter(ghet) / as;
        const X dq = q * du, uq = q * hs, aq = q * qd;
        const X gh = halve(ghet) - dq;
        ghl = ghl + gh;
        ghr = ghr + gh;
        gul = gul + uq;
        gur = gur - uq;
        gal = gal + aq;
        gar = gar + aq;
      }
    } else if (wl) {
      gul = gul + gsl + gsr;
      gal = twice(gsr) - gsl;
    } else {
      gur = gur + gsl + gsr;
      gar = gsr - twice(gsl);
    }
    /* celerities a = sqrt(g h): da/dh = g / (2 a) */
    const double hg = ConstOps<X>::half(g);
    if (wl) ghl = ghl + gal * hg / al;
    if (wr) ghr = ghr + gar * hg / ar;
  }
  /* to the conserved variables: d(h_m, u_n, u_t)/d(h, hu, hv) with y = RN(1/h); the bed sources
   * (source_terms.cuf:90-97): ta = g/2 (ha^2 - hA^2) len into (ta nx, ta ny) of side A, tb likewise
   * into -(tb nx, tb ny) of side B */
  const double len = G.len;
  {
    const X gu = s_ul ? gul : X(0.0), gv = s_ul ? gvl : X(0.0);
    X gh = s_hl ? ghl : X(0.0);
    gh = xfma(xfma(X(w[3]), X(nx), X(w[4]) * ny) * g, (ea > 0. ? ha : X(0.0)) - hA, gh);
    const X y = len * X(UA.w);
    lamA[0] = lamA[1] = lamA[2] = 0.0;
    if (wa) {
      lamA[0] = val(xfma(gh, X(len), -(xfma(gu, ul0, gv * vl0) * y)));
      lamA[1] = val(xfma(gu, X(nx), -(gv * ny)) * y);
      lamA[2] = val(xfma(gu, X(ny), gv * nx) * y);
    } else {
      lamA[0] = val(gh * len);
    }
  }
  {
    const X gu = s_ur ? gur : X(0.0), gv = s_ur ? gvr : X(0.0);
    X gh = s_hr ? ghr : X(0.0);   /* the B side reconstructs from the raw depth */
    gh = xfma(-(xfma(X(w[8]), X(nx), X(w[9]) * ny) * g), (eb > 0. ? hb : X(0.0)) - hB, gh);
    const X y = len * X(UB.w);
    lamB[0] = lamB[1] = lamB[2] = 0.0;
    if (wb) {
      lamB[0] = val(xfma(gh, X(len), -(xfma(gu, ur0, gv * vr0) * y)));
      lamB[1] = val(xfma(gu, X(nx), -(gv * ny)) * y);
      lamB[2] = val(xfma(gu, X(ny), gv * nx) * y);
    } else {
      lamB[0] = val(gh * len);
    }
  }
  return true;
}

/* The transposed element stage (element_core): given the adjoint L of an element's new state, its old
 * state U, its statics st = {area, n, -, RN(1/area)} and its flux and bed sums s, the adjoint own of
 * its old state (besides what comes through its edges), w of its sums and nb of its Manning n, by the
 * chain rule backwards through the formulas of friction_terms and element_core:
 *   - the update q + dt r and the clamp (a clamped element is a constant of its inputs);
 *   - r = R ri with ri = (S + sf - rc) / area, R = I or the semi-implicit matrix.  With fricimplic 1
 *     (r2, r3) solves A (r2, r3) = (ri2, ri3) - (a21, a31) ri1 with the symmetric A of entries 1 + A22,
 *     a23, 1 + A33, so with (s2, s3) = A^-1 (r2', r3') the adjoint of an entry a_ij is -s_i r_j;
 *   - all of a21, a31 are n^2 q1^(-4/3) |v| times a velocity, A22, A33, a23 the same over |v| times a
 *     product of two, sf = -g n^2 area q1^(-1/3) |v| v: their logarithmic derivatives are the same
 *     sums S, W, Z, F for every factor.
 * Only the clamp depends on a value to the last bit; that value (h = q1 + dt ri1) is the step's. */
CFD_HD void adj_element(const MemberDev& M, const double4& U, const double4& st, const Slot& s, const double4& L,
                        double dt, double4& own, Slot& w, double& nb) {
  typedef XD<true> X;
  const double area = st.x, ya = st.w;
  own = make_double4(0.0, 0.0, 0.0, 0.0);
  w.f1 = w.f2 = w.f3 = w.bx = w.by = w.q = 0.0;
  nb = 0.0;
  const bool fric = M.friction == 1;
  const X ri1 = div_rn(fric ? 0. + 0. - X(s.f1) : 0. - X(s.f1), area, ya);
  if (X(U.x) + dt * ri1 <= M.tolisec) return;
  const X q1(U.x), n(st.y), r1b = dt * X(L.x), r2b = dt * X(L.y), r3b = dt * X(L.z);
  const bool wet = fric && q1 > M.tolisec;
  X u(0.0), v(0.0), nv(0.0), iv(0.0), sf2(0.0), sf3(0.0), c(0.0), p13(0.0);
  bool fast = false;   /* |v| > tol: the matrix differs from the identity */
  if (wet) {
    u = div_rn(X(U.y), q1, X(U.w));
    v = div_rn(X(U.z), q1, X(U.w));
    nv = sqrt(u * u + v * v);
    const bool held = nv < M.tol;   /* a constant of the inputs then, as where it is 0 */
    if (held) nv = X(M.tol);
    else if (nv > 0.) iv = 1.0 / nv;
    fast = nv > M.tol;
    p13 = rcbrt(q1);
    c = M.gp * n * n * nv * area * p13;
    sf2 = -(c * u);
    sf3 = -(c * v);
  }
  X s2 = r2b, s3 = r3b, ri1b = r1b, ub(0.0), vb(0.0), nvb(0.0), S(0.0);
  if (fast && (M.fricimplic == 1 || M.fricimplic == 2)) {
    const X ri2 = div_rn(s.bx + sf2 - s.f2, area, ya), ri3 = div_rn(s.by + sf3 - s.f3, area, ya);
    const X d = ConstOps<X>::half(dt) * M.gp * n * n * p13 * U.w;
    if (M.fricimplic == 1) {
      const X e = d * iv, dn = (7.0 / 3.0) * d * nv;
      const X uu = u * u, vv = v * v;
      const X A22 = e * xfma(u, u, uu + vv), A33 = e * xfma(v, v, uu + vv), a23 = e * (u * v);
      const X a22 = 1. + A22, a33 = 1. + A33;
      const X id = 1.0 / xfma(a22, a33, -(a23 * a23));
      s2 = xfma(a33, r2b, -(a23 * r3b)) * id;
      s3 = xfma(a22, r3b, -(a23 * r2b)) * id;
      const X m1 = dn * ri1, t2 = xfma(m1, u, ri2), t3 = xfma(m1, v, ri3);
      const X r2 = xfma(a33, t2, -(a23 * t3)) * id, r3 = xfma(a22, t3, -(a23 * t2)) * id;
      const X us = xfma(u, s2, v * s3);
      ri1b = xfma(dn, us, r1b);
      const X b22 = -(s2 * r2), b33 = -(s3 * r3), b23 = -xfma(s2, r3, s3 * r2);
      /* b21 a21 + b31 a31 = ri1 dn (u s2 + v s3) */
      const X Z = m1 * us, W = xfma(b22, A22, xfma(b33, A33, b23 * a23));
      S = Z + W;
      nvb = (Z - W) * iv;
      ub = xfma(m1, s2, e * xfma(twice(u), twice(b22) + b33, v * b23));
      vb = xfma(m1, s3, e * xfma(twice(v), twice(b33) + b22, u * b23));
    } else {
      const X beta = -(twice(d) * nv), im = 1.0 / (1. - beta);
      s2 = r2b * im;
      s3 = r3b * im;
      S = xfma(s2, ri2, s3 * ri3) * beta * im;
      nvb = S * iv;
    }
  }
  const X s2y = s2 * ya, s3y = s3 * ya;
  w.f1 = val(-(ri1b * ya));
  w.f2 = val(-s2y);
  w.f3 = val(-s3y);
  w.bx = val(s2y);
  w.by = val(s3y);
  own = L;
  own.w = 0.0;
  if (wet) {
    const X F = xfma(sf2, s2y, sf3 * s3y);
    const X g = xfma(F, iv, nvb) * iv;   /* adjoint of |v| over |v| */
    ub = xfma(-c, s2y, xfma(g, u, ub));
    vb = xfma(-c, s3y, xfma(g, v, vb));
    const X k = xfma(ub, u, xfma(vb, v, xfma(X(4.0), S, F) * (1.0 / 3.0)));
    const X y(U.w);
    own.x = val(xfma(-k, y, X(L.x)));
    own.y = val(xfma(ub, y, X(L.y)));
    own.z = val(xfma(vb, y, X(L.z)));
    nb = n != 0.0 ? val(twice(F + S) / n) : 0.0;
  }
}

}  // namespace cf

#endif
