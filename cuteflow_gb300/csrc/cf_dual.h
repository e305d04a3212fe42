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

/* J^T w of one side's first-order HLLC flux (weights w of its three global components) towards a
 * differing right state, for the edges with a nearly dry side (0 < h <= tolisec, whose raw and masked
 * depths differ, so that the two sides see different states): rare, out of line, on dual numbers.
 * out: the adjoints of the left (h, u, v) and of the right one. */
#ifdef __CUDACC__
static __host__ __device__ __noinline__
#else
static inline
#endif
void adj_one_side(double g, double nx, double ny, const double l[3], const double r[3], const double w[3],
                  double out[6]) {
  typedef Dual<6> D;
  TwoFluxT<D> F;
  first_order_flux<1>(g, nx, ny, D::var(l[0], 0), D::var(l[1], 1), D::var(l[2], 2), D::var(r[0], 3), D::var(r[1], 4),
                      D::var(r[2], 5), F);
  for (int i = 0; i < 6; ++i) out[i] = fma(w[0], F.a1.d[i], fma(w[1], F.a2.d[i], w[2] * F.a3.d[i]));
}

/* One side of the transposed edge stage of an interior first-order HLLC edge (IFLUX 1, flux_mode 0):
 * given the adjoint weights w[5] of this side's slot (flux 1-3, bed x, y), and the other side running
 * beside it (EdgeSide: two lanes of the GPU), the contribution lam to the adjoint of (h, hu, hv) of
 * this side's element, by the chain rule backwards through the flux's own formulas:
 *   - the rotation of the frame flux (x1, x2, x3), with x3 = x1 v in every region, v the tangential
 *     velocity the region takes;
 *   - the HLL fluxes N / (s_R - s_L + eps) or the physical flux the region takes;
 *   - the speed s_L = u - a p with p = 1 or sqrt((h* + h) h* / 2) / h, and the depth
 *     h* = (h + h') / 2 - (u' - u) (h + h') / (a + a') / 4; next to a dry side s = u - a and u + 2 a of
 *     the wet one;
 *   - the hydrostatic reconstruction (depths pass or are clamped to 0), the change to the edge frame
 *     (u_n = (hu nx + hv ny) / h, u_t = (hv nx - hu ny) / h) and the bed source g/2 (hw^2 - h^2) len.
 * The other side's flux is this one's mirrored, so the adjoints of the HLL fluxes are the difference
 * and the sum of the two sides' weights, and what remains towards each side's own state is the same
 * code on either.  The values repeat the step's IEEE operations (so every branch is the forward's),
 * their products, quotients and roots on the integer pipes; of the derivatives the multiply-adds are
 * FP64 instructions and the products integer ones. */
struct AdjSide : EdgeSide<1, XD<true>> {
  typedef XD<true> X;
  double w[5];
  double yh;                     /* RN(1/h) of the element */
  X het, pq, hs, du, qd;
  X fg1, fg2, t, y1, m1, m2, gh, gu, gv, ga, gsl;
  bool wet, both, wl, strong, odd;
  int r, rp;                     /* region of this side's flux, and of the other side's in its own frame */

  CFD_HD void begin(const MemberDev& M, int side_, const double4& geo, const double4& U, double z, double zo,
                    const double w_[5]) {
    for (int i = 0; i < 5; ++i) w[i] = w_[i];
    yh = U.w;
    frame(M, side_, side_ ? -geo.x : geo.x, side_ ? -geo.y : geo.y, geo.z, U, z, zo);
    wet = h0 > tolisec;
  }
  CFD_HD void values1() {
    speeds1();
    odd = hraw != hr || film();  /* the other side is nearly dry, or both are films */
  }
  CFD_HD void values2() {
    const X ar = y[0];
    hs = side ? y[1] : s;
    du = side ? s : y[1];
    as_ = a + ar;
    qd = du * hs / as_;
    het = halve(hs) - quarter(qd);
    wl = h > eps();
    both = wl && hr > eps();
    strong = both && !lt_nonneg(het, h);
    pq = strong ? sqrt(halve(het + h) * het / (h * h)) : X(1.);
    sl = (wl ? u : ur) - (wl ? (both ? a * pq : a) : twice(ar));
    d0 = u - sl;
    f1 = h * u;
    f2 = h * (u * u) + halve(gh_() * h);
    d = h * d0;
    x[0] = sl;
    x[1] = d;
    x[2] = f1;
    x[3] = f2;
  }
  CFD_HD const X& gh_() const { return EdgeSide<1, XD<true>>::gh; }
  CFD_HD void values3() {
    sr = -y[0];
    s = y[1];
    fr1 = -y[2];
    fr2 = y[3];
    t2 = sr * h * d0;
    x[0] = t2;
  }
  CFD_HD void values4() {
    t2 = (side ? -d : y[0]) - (side ? s : t2);   /* as contact1 */
    x[0] = t2;
  }
  CFD_HD void reverse1() {
    const X num = side ? -y[0] : t2, denom = side ? t2 : y[0];
    if (fabs(denom) < eps()) set = halve(u + ur) - (hr - h) * as_ / hs;
    else set = num / denom;
    r = (sl > 0.) ? 0 : ((sr < 0.) ? 1 : 2);
    rp = (sr < 0.) ? 0 : ((sl > 0.) ? 1 : 2);
    const bool right = r == 1 || (r == 2 && !(set > 0.));
    t = xfma(X(w[2]), X(nx), -(X(w[1]) * ny));
    fg2 = xfma(X(w[1]), X(nx), X(w[2]) * ny);
    fg1 = xfma(right ? vr : v, t, X(w[0]));
    y1 = 1.0 / (sr - sl + eps());
    const X c1 = xfma(sl, hr - h, f1), c2 = xfma(sl, fr1 - f1, f2);
    m1 = xfma(sr, c1, -(sl * fr1)) * y1;
    m2 = xfma(sr, c2, -(sl * fr2)) * y1;
    const X c = t * (r == 0 ? f1 : (r == 1 ? fr1 : m1));
    gv = right ? X(0.0) : c;
    x[0] = fg1;
    x[1] = fg2;
    x[2] = c;
  }
  CFD_HD void reverse2() {
    /* the other side's tangential flux carries this side's v */
    if (rp == 1 || (rp == 2 && !(set < 0.))) gv = gv - y[2];
    X gf1(0.0), gf2(0.0);
    gh = X(0.0);
    gsl = X(0.0);
    if (r == 2 || rp == 2) {
      const X n1 = (rp == 2 ? (r == 2 ? fg1 - y[0] : -y[0]) : fg1) * y1;
      const X n2 = (rp == 2 ? (r == 2 ? fg2 + y[1] : y[1]) : fg2) * y1;
      const X ss = sl * sr, q2 = n2 * ss;
      gsl = xfma(n1, xfma(sr, hr - h, -fr1) + m1, n2 * (xfma(sr, fr1 - f1, -fr2) + m2));
      gf1 = xfma(n1, sr, -q2);
      gf2 = n2 * sr;
      gh = -(n1 * ss);
    }
    if (r == 0) { gf1 = gf1 + fg1; gf2 = gf2 + fg2; }
    if (rp == 1) { gf1 = gf1 - y[0]; gf2 = gf2 + y[1]; }
    /* physical flux: f1 = h u, f2 = h u^2 + g h^2 / 2 */
    gh = xfma(gf1, u, xfma(gf2, xfma(u, u, gh_()), gh));
    gu = xfma(gf1, h, twice(gf2 * f1));
    ga = X(0.0);
    X ghet(0.0);
    if (strong) {
      /* p^2 = P = (h* + h) h* / 2 / h^2: dP/dh* = (h* + h / 2) / h^2, dP/dh = (h* / 2 - 2 P h) / h^2 */
      const X gp = -(gsl * a) / (twice(pq) * (h * h));
      ghet = gp * (het + halve(h));
      gh = xfma(gp, xfma(-twice(pq * pq), h, halve(het)), gh);
    }
    x[0] = ghet;
    x[1] = gsl;
  }
  /* this side's flux alone, from its masked state towards the other one's raw reconstruction: the
   * adjoints of the two states, each in this side's frame */
  CFD_HD void one_side(double o[6]) const {
    const double l[3] = {val(h), val(u), val(v)};
    const double rr[3] = {val(hraw), val(ur), val(vr)};
    const double ww[3] = {w[0], w[1], w[2]};
    double oo[6];
    adj_one_side(g, nx, ny, l, rr, ww, oo);
    for (int i = 0; i < 6; ++i) o[i] = oo[i];
  }
  /* the adjoints of this side's own state from both one-sided evaluations: the left state of its own (a
   * constant where the depth is masked), the right state (mirrored velocities) of the other's */
  CFD_HD void join(const double own[6], const double other[6], double one[3]) const {
    one[0] = (wet ? own[0] : 0.0) + other[3];
    one[1] = own[1] - other[4];
    one[2] = own[2] - other[5];
  }
  /* one: the adjoints of this side's own state from a one-sided evaluation (adj_one_side) of both
   * fluxes, in place of the above */
  CFD_HD void reverse3(const double* one, double lam[3]) {
    if (both) {
      gu = gu + gsl;
      ga = -(gsl * pq);
      const X ghet = x[0] + y[0];
      const X q = quarter(ghet) / as_;
      gh = gh + (halve(ghet) - q * du);
      gu = xfma(q, hs, gu);
      ga = xfma(q, qd, ga);
    } else if (wl) {
      const X gsr = -y[1];       /* next to a dry side this one sets both speeds */
      gu = gu + gsl + gsr;
      ga = twice(gsr) - gsl;
    }
    if (wl) gh = gh + ga * ConstOps<X>::half(g) / a;   /* a = sqrt(g h) */
    if (dry()) gh = gu = gv = X(0.0);
    bool sh = wet && hw > 0. && !(h < tolisec), su = wet && !(h < tolisec);
    if (one) {
      gh = X(one[0]);
      gu = X(one[1]);
      gv = X(one[2]);
      sh = hw > 0. && !(hw < tolisec);
    }
    if (!sh) gh = X(0.0);
    if (!su) gu = gv = X(0.0);
    gh = xfma(xfma(X(w[3]), X(nx), X(w[4]) * ny) * g, hw - h0, gh);
    if (wet) {
      const X yl = len * X(yh);
      lam[0] = val(xfma(gh, X(len), -(xfma(gu, u, gv * v) * yl)));
      lam[1] = val(xfma(gu, X(nx), -(gv * ny)) * yl);
      lam[2] = val(xfma(gu, X(ny), gv * nx) * yl);
    } else {
      lam[0] = val(gh * len);
      lam[1] = lam[2] = 0.0;
    }
  }
};

/* The stages of both sides (P as in side_stages; P::finish: the last stage, with the one-sided evaluation for
 * the pairs that take it) */
template <class P>
CFD_HD void adj_stages(P& p) {
  p.exchange(4);
  p.each([](AdjSide& s, double*) { s.values1(); });
  p.exchange(2);
  p.each([](AdjSide& s, double*) { s.values2(); });
  p.exchange(4);
  p.each([](AdjSide& s, double*) { s.values3(); });
  p.exchange(1);
  p.each([](AdjSide& s, double*) { s.values4(); });
  p.exchange(1);
  p.each([](AdjSide& s, double*) { s.reverse1(); });
  p.exchange(3);
  p.each([](AdjSide& s, double*) { s.reverse2(); });
  p.exchange(2);
  p.finish();
}

struct AdjHostPair {
  AdjSide s[2];
  double lam[2][3];
  template <class F>
  CFD_HD void each(F&& f) {
    f(s[0], lam[0]);
    f(s[1], lam[1]);
  }
  CFD_HD void exchange(int n) {
    for (int k = 0; k < n; ++k) {
      s[0].y[k] = s[1].x[k];
      s[1].y[k] = s[0].x[k];
    }
  }
  void finish() {
    double one[2][3];
    const bool odd = s[0].odd || s[1].odd;
    if (odd) {
      double o[2][6];
      for (int k = 0; k < 2; ++k) s[k].one_side(o[k]);
      for (int k = 0; k < 2; ++k) s[k].join(o[k], o[1 - k], one[k]);
    }
    for (int k = 0; k < 2; ++k) s[k].reverse3(odd ? one[k] : nullptr, lam[k]);
  }
};

/* Both sides on the host: lamA, lamB from the weights w[10] of the two slots */
inline bool adj_edge_hllc(const MemberDev& M, const EdgeGeo& G, const double4& UA, const double4& UB, double zml,
                          double zmr, const double w[10], double lamA[3], double lamB[3]) {
  const double4 geo = make_double4(G.nx, G.ny, G.len, 0.0);
  AdjHostPair p;
  p.s[0].begin(M, 0, geo, UA, zml, zmr, w);
  p.s[1].begin(M, 1, geo, UB, zmr, zml, w + 5);
  adj_stages(p);
  for (int k = 0; k < 3; ++k) {
    lamA[k] = p.lam[0][k];
    lamB[k] = p.lam[1][k];
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
