/*
 * cf_flux.h -- per-edge and per-element arithmetic of the step, shared by the sm_103a kernels
 * (cf_kernels.cu, cf_adjoint.cu) and, compiled for the host, by the CPU test harness that checks
 * it against the oracle edge by edge.  Everything here is __host__ __device__ and FP64.
 *
 * Bit-exact reproduction.  The reference's WAF flux is discontinuous at the bit level: where
 * the reconstructed depths of an edge are equal to the last bit (still water),
 * r = dupw / (dloc + eps) (flux_riemann.cuf:876-878) changes sign with the side that
 * evaluates it, and a one-ulp change of the state moves the limiter between its branches.
 * A result "within round-off" of the reference therefore does not stay within 1e-9 of it.
 * This code evaluates every expression in the reference's order of operations, with true
 * divisions, and the kernels are compiled without FMA contraction (-fmad=false), so a step
 * on the GPU reproduces the CPU restatement of the reference bit for bit.  The second side of
 * an edge is obtained from the first by exact IEEE identities ((-a)*b = -(a*b),
 * (-a)-(-b) = b-a, commutativity), never by re-rounded arithmetic.
 *
 * Scalar type.  The state-dependent arithmetic is written once, as templates on the scalar
 * type T.  T = double is the step.  T = Dual<N> (cf_dual.h) carries N derivative lanes next to
 * a value lane that performs the same IEEE operations in the same order, so it takes the same
 * branches (wet/dry masks, wave regions, limiter cases) as the step and its lanes are the exact
 * local Jacobian of that branch: the discrete adjoint is built from it.  Geometry, time and
 * time step stay double (the adjoint holds dt fixed).
 */
#ifndef CF_FLUX_H
#define CF_FLUX_H

#include <cmath>
#include <cstring>

#include "cf_internal.h"

#ifdef __CUDACC__
#define CF_HD __host__ __device__
#define CF_INLINE __forceinline__
#else
#define CF_HD
#define CF_INLINE inline
#endif

namespace cf {

#ifndef __CUDACC__
using std::copysign;
using std::fabs;
using std::fma;
using std::fmax;
using std::frexp;
using std::ldexp;
using std::sqrt;
#endif

/* ---- loads --------------------------------------------------------------------------- */

/* Two 16-byte loads.  Plain ones: states, statics and slots are written by kernels that may still run
 * when a kernel that overlaps them begins (cf_launch.cuh), which the read-only path does not allow. */
CF_HD CF_INLINE double4 ld4(const double4* p) {
#ifdef __CUDA_ARCH__
  const double2* q = reinterpret_cast<const double2*>(p);
  const double2 a = q[0], b = q[1];
  return make_double4(a.x, a.y, b.x, b.y);
#else
  return *p;
#endif
}

/* the mesh's tables, which no kernel writes */
template <class T>
CF_HD CF_INLINE T ldro(const T* p) {
#ifdef __CUDA_ARCH__
  return __ldg(p);
#else
  return *p;
#endif
}

/* The two 32-bit words of a bit pattern, through an opaque move on the device.  A test written on
 * a double's whole 64-bit pattern, such as (b << 1) == 0 or (b & exponent) != exponent, is
 * recognised by the compiler as a comparison of the double and issued as an FP64-pipe instruction
 * (measured: one per test); on the words it stays on the integer pipes. */
CF_HD CF_INLINE void words_u(uint64_t b, uint32_t& lo, uint32_t& hi) {
#ifdef __CUDA_ARCH__
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(b));
#else
  lo = (uint32_t)b;
  hi = (uint32_t)(b >> 32);
#endif
}
/* b is the pattern of a finite double */
CF_HD CF_INLINE bool finite_u(uint64_t b) {
  uint32_t lo, hi;
  words_u(b, lo, hi);
  (void)lo;
  return (hi & 0x7ff00000u) != 0x7ff00000u;
}
/* b is the pattern of +0 or -0 */
CF_HD CF_INLINE bool zero_u(uint64_t b) {
  uint32_t lo, hi;
  words_u(b, lo, hi);
  return ((hi << 1) | lo) == 0;
}

CF_HD CF_INLINE uint64_t dbits_hd(double x) {
  uint64_t b;
  memcpy(&b, &x, sizeof(b));
  return b;
}
CF_HD CF_INLINE double dbl_hd(uint64_t b) {
  double x;
  memcpy(&x, &b, sizeof(x));
  return x;
}

CF_HD CF_INLINE bool finite_bits(double x) {
  uint64_t b;
  memcpy(&b, &x, sizeof(b));
  return finite_u(b);
}

/* value of a scalar (the Dual overload is in cf_dual.h) */
CF_HD CF_INLINE double val(double x) { return x; }

template <class T>
CF_HD CF_INLINE T dmax(const T& a, const T& b) { return (a < b) ? b : a; } /* Fortran max */
template <class T>
CF_HD CF_INLINE T dmin(const T& a, const T& b) { return (b < a) ? b : a; } /* Fortran min */

template <class T>
CF_HD CF_INLINE T dmax0(const T& x) { return dmax(T(0.0), x); }

/* a < b where b is +0 or above and not NaN (the integer type has a shorter test for that) */
template <class T>
CF_HD CF_INLINE bool lt_nonneg(const T& a, const T& b) { return a < b; }

/* Operations on an edge's constants (geometry, dt, g) in the arithmetic of the scalar type T: the
 * quotient a / d given y = RN(1/d), x / 2 and 2 x, the same results for every T.  cf_xd.h keeps them
 * off the FP64 pipe for its type. */
template <class T>
struct ConstOps {
  static CF_HD CF_INLINE double quot(double a, double d, double y);
  static CF_HD CF_INLINE double half(double x) { return x * 0.5; }
  static CF_HD CF_INLINE double dbl(double x) { return x * 2.0; }
};

/* a b where a is often exactly 0, and whether x is +-0 (cf_xd.h: without leaving the fast path) */
template <class T>
CF_HD CF_INLINE T mulz(const T& a, const T& b) { return a * b; }
CF_HD CF_INLINE bool is_zero(double x) { return x == 0.0; }

/* the value of a wave speed for its sign alone, negated for the other side: a zero stays as it is */
template <class T>
CF_HD CF_INLINE T opposite(const T& x) {
  const double v = val(x);
  return T(zero_u(dbits_hd(v)) ? v : -v);
}

/* -x of a difference x that the other side has formed: a side's own difference of equal numbers is +0 like
 * the other one's, and not its negation */
template <class T>
CF_HD CF_INLINE T mirrored(const T& x) { return 0.0 - x; }

/* 0 - x, and the first row (1, 0, 0) of the semi-implicit matrix applied to (a, b, c); cf_xd.h forms
 * them for its type without the arithmetic where that does not change the value */
template <class T>
CF_HD CF_INLINE T zero_minus(const T& x) { return 0. - x; }
template <class T>
CF_HD CF_INLINE T first_row(const T& a, const T& b, const T& c) { return 1. * a + 0. * b + 0. * c; }
/* every component finite */
template <class T>
CF_HD CF_INLINE bool finite_val(const T& x) { return finite_bits(val(x)); }

/* RN(1/d) of a denominator that several quotients share (div_rn) */
template <class T>
CF_HD CF_INLINE T recip(const T& d) { return 1.0 / d; }

/* x / 2, x / 4 and 2 x.  A scaling by a power of two rounds once whichever way it is written, so
 * these give the bits of the quotient or product they stand for; the integer-product type (cf_xd.h)
 * overloads them with an exponent change. */
template <class T>
CF_HD CF_INLINE T halve(const T& x) { return x * 0.5; }
template <class T>
CF_HD CF_INLINE T quarter(const T& x) { return x * 0.25; }
template <class T>
CF_HD CF_INLINE T twice(const T& x) { return x * 2.0; }

/* a / d rounded to nearest, given y = RN(1/d): q = RN(a y), r = a - d q (exact through the
 * FMA), RN(q + r y) (Markstein's correction step; P. Markstein, "Computation of elementary
 * functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990).  It equals the
 * IEEE quotient for finite non-zero a (no mismatch in 3e8 adversarial samples, see the tests);
 * a zero numerator is returned as q = a y, which carries the quotient's sign.  Three FP64
 * instructions instead of a full division wherever 1/d is known: for precomputed geometry,
 * and for denominators shared by several quotients (y = 1/d computed once). */
CF_HD CF_INLINE double div_rn(double a, double d, double y) {
  const double q = a * y;
  const double r = fma(-d, q, a);
  const double q1 = fma(r, y, q);
  uint64_t ab;
  memcpy(&ab, &a, sizeof(ab));
  return zero_u(ab) ? q : q1;
}

template <class T>
CF_HD CF_INLINE double ConstOps<T>::quot(double a, double d, double y) { return div_rn(a, d, y); }

/* ---- x**(-1/3) -------------------------------------------------------------------------- */

/* x^(-1/3), the Manning factor h^(-1/3) (source_terms.cuf:112-127; the reference calls pow, which
 * is not correctly rounded and differs between math libraries), as one fixed sequence of IEEE and
 * integer operations that the oracle repeats exactly, with no division:
 *   x = m 2^(3k), m in [1, 8): the exponent split in integer arithmetic (Kahan, "Computing a real
 *       cube root", 1991, splits the exponent by three the same way);
 *   a single-precision seed for m^(-1/3): a cubic in the leading mantissa bits u = 1 + f
 *       (least-squares fit of u^(-1/3) on [1, 2), relative error 2.5e-4) times 2^(-r/3), then one
 *       Newton step y <- y + y (1 - m y^3) / 3 (relative error ~2e-7);
 *   one third-order step in double precision, y <- y + y (e/3 + 2 e^2/9) with e = 1 - m y^3 (the
 *       series of (1 - e)^(-1/3) to second order; the truncation is below 1e-19 relative);
 *   y 2^(-k) by an exponent shift.
 * Rounding bound 1.2 ulp (the two products forming y^3 give e an error of 2^-52, a third of it
 * reaches y; then the final rounding); measured within 1 ulp of the exact value (tests).  Seven
 * FP64-pipe instructions.  Zero, subnormal, infinite, negative and NaN x (never reached by the
 * step, whose depths here exceed tolisec > 0) take rcbrt_special. */
struct MulFp64 {
  static CF_HD CF_INLINE double mul(double a, double b) { return a * b; }
};
template <class P = MulFp64>
CF_HD CF_INLINE double rcbrt_core(uint64_t b) {
  const uint32_t ex = (uint32_t)(b >> 52);
  const uint32_t ep = ex + 177u;            /* unbiased exponent + 1200 */
  const uint32_t k3 = ep / 3u;
  const uint32_t r = ep - 3u * k3;          /* exponent = 3 (k3 - 400) + r */
  const uint64_t frac = b & ((1ull << 52) - 1);
  const uint64_t mb = frac | ((uint64_t)(1023u + r) << 52);
  const uint32_t ub = (127u << 23) | (uint32_t)(frac >> 29);
  const uint32_t mfb = ub + (r << 23);
  double m;
  float u, mf;
  memcpy(&m, &mb, sizeof(m));
  memcpy(&u, &ub, sizeof(u));
  memcpy(&mf, &mfb, sizeof(mf));
  float y = fmaf(fmaf(fmaf(-0x1.99153cp-5f, u, 0x1.45621ap-2f), u, -0x1.9eb31ap-1f), u, 0x1.8ab91ap+0f);
  y = y * (r == 0u ? 1.0f : (r == 1u ? 0x1.965feap-1f : 0x1.428a30p-1f));
  const float e32 = fmaf(-mf, y * y * y, 1.0f);
  y = fmaf(y, e32 * 0x1.555556p-2f, y);
  const double yd = (double)y;
  const double e = fma(-m, P::mul(P::mul(yd, yd), yd), 1.0);
  const double c = P::mul(e, fma(e, 2.0 / 9.0, 1.0 / 3.0));
  const double res = fma(yd, c, yd);
  uint64_t rb;
  memcpy(&rb, &res, sizeof(rb));
  rb = (uint64_t)((int64_t)rb - ((int64_t)k3 - 400) * (int64_t)(1ull << 52));
  double out;
  memcpy(&out, &rb, sizeof(out));
  return out;
}

/* x^(-1/3) outside the normal positive numbers: +0 -> +inf, subnormal -> scaled by 2^54 into the
 * normal range (x^(-1/3) = (2^54 x)^(-1/3) 2^18, exact scalings), +inf -> 0, negative or NaN ->
 * NaN (Fortran's real power of a negative base). */
CF_HD CF_INLINE double rcbrt_special(double x) {
  if (!(x >= 0.0)) {
    const uint64_t qnan = 0x7ff8000000000000ull;
    double n;
    memcpy(&n, &qnan, sizeof(n));
    return (x != x) ? x : n;
  }
  if (x == 0.0) return 1.0 / x;
  if (x > 1.0) return 0.0;
  const double s = x * 0x1p54;
  uint64_t b;
  memcpy(&b, &s, sizeof(b));
  return rcbrt_core(b) * 0x1p18;
}

template <class P = MulFp64>
CF_HD CF_INLINE double rcbrt_of(double x) {
  uint64_t b;
  memcpy(&b, &x, sizeof(b));
  if ((uint32_t)(b >> 52) - 1u >= 2046u) return rcbrt_special(x);
  return rcbrt_core<P>(b);
}
CF_HD CF_INLINE double rcbrt(double x) { return rcbrt_of(x); }

/* ---- edge-frame states ------------------------------------------------------------------ */

/* RN(1/h) of an element's depth: the state carries it (the element kernel stores it with the
 * new depth), so the quotients by h below are Markstein's exact three-instruction form.  A
 * linearization computes it from h (cf_dual.h overloads this for its dual numbers). */
template <class T>
CF_HD CF_INLINE T recip_h(const T&, double yh) { return T(yh); }

/* Masked primitive state in the frame (n, t) of an edge (flux_riemann.cuf:105-112); yh = RN(1/h). */
template <class T>
CF_HD CF_INLINE void to_frame(T h, T hu, T hv, double yh, double nx, double ny, double tolisec, T& hm, T& un,
                              T& ut) {
  if (h > tolisec) {
    const T y = recip_h(h, yh);
    un = div_rn(hu * nx + hv * ny, h, y);
    ut = div_rn(hv * nx - hu * ny, h, y);
    hm = h;
  } else {
    hm = T(0.0);
    un = T(0.0);
    ut = T(0.0);
  }
}

/* Only the masked depth and tangential velocity (what the WAF upwind states use). */
template <class T>
CF_HD CF_INLINE void to_frame_t(T h, T hu, T hv, double yh, double nx, double ny, double tolisec, T& hm, T& ut) {
  if (h > tolisec) {
    ut = div_rn(hv * nx - hu * ny, h, recip_h(h, yh));
    hm = h;
  } else {
    hm = T(0.0);
    ut = T(0.0);
  }
}

/* Wave speeds of all solvers (flux_riemann.cuf:930-983, 753-806, 1055-1108).  Returns false
 * when both depths are below eps: the reference then reads uninitialised speeds; the flux
 * defined for that case is zero. */
template <class T>
CF_HD CF_INLINE bool wave_speeds(double g, double eps, T hl, T ul, T hr, T ur, T& sl, T& sr, T& set) {
  if (hl < eps && hr < eps) return false;
  const T al = sqrt(g * hl);
  const T ar = sqrt(g * hr);
  const T het = halve(hl + hr) - quarter((ur - ul) * (hl + hr) / (al + ar));
  T pql, pqr;
  if (lt_nonneg(het, hl)) pql = T(1.);
  else pql = (hl > eps) ? sqrt(halve(het + hl) * het / (hl * hl)) : T(0.);
  if (lt_nonneg(het, hr)) pqr = T(1.);
  else pqr = (hr > eps) ? sqrt(halve(het + hr) * het / (hr * hr)) : T(0.);
  if (hl > eps) {
    sl = ul - al * pql;
    if (hr > eps) {
      sr = ur + ar * pqr;
    } else {
      sl = ul - al;
      sr = ul + twice(al);
    }
  } else {
    sl = ur - twice(ar);
    sr = ur + ar;
  }
  const T denom = hr * (ur - sr) - hl * (ul - sl);
  if (fabs(denom) < eps) set = halve(ul + ur) - (hr - hl) * (al + ar) / (hl + hr);
  else set = (sl * hr * (ur - sr) - sr * hl * (ul - sl)) / denom;
  return true;
}

template <class T>
struct TwoFluxT {
  /* global-frame flux of side A (normal out of A) and of side B (normal out of B) */
  T a1, a2, a3, b1, b2, b3;
};
typedef TwoFluxT<double> TwoFlux;

/* Side A's global flux from the edge-frame vector x; side B's from its vector y: B's frame
 * normal is -n and its vector is the mirror (-y1, y2, y3), which reprojects to
 * -(n1 y2 - n2 y3), -(n2 y2 + n1 y3) exactly. */
template <class T>
CF_HD CF_INLINE void reproject_both(double nx, double ny, T x1, T x2, T x3, T y1, T y2, T y3, TwoFluxT<T>& F) {
  F.a1 = x1;
  F.a2 = nx * x2 - ny * x3;
  F.a3 = ny * x2 + nx * x3;
  F.b1 = -y1;
  F.b2 = -(nx * y2 - ny * y3);
  F.b3 = -(ny * y2 + nx * y3);
}

/* First-order HLLC (IFLUX 1, flux_riemann.cuf:902-1026) and the star-state HLLC of Ata et
 * al. (IFLUX 2, :1029-1182), for both sides.  Side B's evaluation is the mirror image
 * (h -> h, u_n -> -u_n, u_t -> -u_t, s_L -> -s_R, s_R -> -s_L, s_* -> -s_*): it selects a
 * region with its own tests and its vector is the mirror of an A-frame vector. */
template <int IFLUX, class T>
CF_HD CF_INLINE void first_order_flux(double g, double nx, double ny, T hl, T ul, T vl, T hr, T ur, T vr,
                                      TwoFluxT<T>& F) {
  const double eps = (IFLUX == 1) ? EPS_HLLC : EPS_RIADH;
  T sl, sr, set;
  if (!wave_speeds(g, eps, hl, ul, hr, ur, sl, sr, set)) {
    F.a1 = F.a2 = F.a3 = F.b1 = F.b2 = F.b3 = T(0.0);
    return;
  }
  const T fl1 = hl * ul, fl2 = hl * (ul * ul) + halve(g * hl * hl), fl3 = hl * ul * vl;
  const T fr1 = hr * ur, fr2 = hr * (ur * ur) + halve(g * hr * hr), fr3 = hr * ur * vr;
  T x1, x2, x3, y1, y2, y3;
  if (IFLUX == 1) {
    /* A: sl > 0 -> FL | sr < 0 -> FR | HLL with the tangential component of the upwind side
     * of s*.  B: -sr > 0 -> FR | -sl < 0 -> FL | HLL, tangential by -s*. */
    const int ra = (sl > 0.) ? 0 : ((sr < 0.) ? 1 : 2);
    const int rb = (-sr > 0.) ? 1 : ((-sl < 0.) ? 0 : 2);
    T h1 = T(0.0), h2 = T(0.0);
    if (ra == 2 || rb == 2) {
      const T den = sr - sl + eps;
    const auto yden = recip(den);
      h1 = div_rn(sr * fl1 - sl * fr1 + sl * sr * (hr - hl), den, yden);
      h2 = div_rn(sr * fl2 - sl * fr2 + sl * sr * (hr * ur - hl * ul), den, yden);
    }
    if (ra == 0) { x1 = fl1; x2 = fl2; x3 = fl3; }
    else if (ra == 1) { x1 = fr1; x2 = fr2; x3 = fr3; }
    else { x1 = h1; x2 = h2; x3 = (set > 0.) ? h1 * vl : h1 * vr; }
    if (rb == 0) { y1 = fl1; y2 = fl2; y3 = fl3; }
    else if (rb == 1) { y1 = fr1; y2 = fr2; y3 = fr3; }
    else { y1 = h1; y2 = h2; y3 = (-set > 0.) ? h1 * vr : h1 * vl; }
  } else {
    const T pl = (fabs(sl - set) > eps) ? hl * (sl - ul) / (sl - set) : T(0.0);
    const T pr = (fabs(sr - set) > eps) ? hr * (sr - ur) / (sr - set) : T(0.0);
    const T el1 = fl1 + sl * (pl - hl), el2 = fl2 + sl * (pl * set - hl * ul), el3 = fl3 + sl * (pl * vl - hl * vl);
    const T er1 = fr1 + sr * (pr - hr), er2 = fr2 + sr * (pr * set - hr * ur), er3 = fr3 + sr * (pr * vr - hr * vr);
    /* A: 0<sl FL | 0<s* & 0>sl EL | 0>s* & 0<sr ER | FR.
     * B (sl'=-sr, s*'=-s*, sr'=-sl): 0<-sr FR | 0<-s* & 0>-sr ER | 0>-s* & 0<-sl EL | FL. */
    int ra, rb;
    if (0. < sl) ra = 0;
    else if (0. < set && 0. > sl) ra = 2;
    else if (0. > set && 0. < sr) ra = 3;
    else ra = 1;
    if (0. < -sr) rb = 1;
    else if (0. < -set && 0. > -sr) rb = 3;
    else if (0. > -set && 0. < -sl) rb = 2;
    else rb = 0;
#define CF_PICK(r, a1_, a2_, a3_)                      \
  if (r == 0) { a1_ = fl1; a2_ = fl2; a3_ = fl3; }     \
  else if (r == 1) { a1_ = fr1; a2_ = fr2; a3_ = fr3; } \
  else if (r == 2) { a1_ = el1; a2_ = el2; a3_ = el3; } \
  else { a1_ = er1; a2_ = er2; a3_ = er3; }
    CF_PICK(ra, x1, x2, x3)
    CF_PICK(rb, y1, y2, y3)
#undef CF_PICK
  }
  reproject_both(nx, ny, x1, x2, x3, y1, y2, y3, F);
}

/* WAF limiter (flux_riemann.cuf:465-524).  The superbee gaps at r = 0.5, 1, 2 are kept. */
template <class T>
CF_HD CF_INLINE T waf_limiter(int ilim, T r, T c) {
  T A = T(1.);
  if (ilim == 1) {
    /* two of the branches share their arithmetic: the lanes of a warp are in all of them (WAF dam break
     * 134k 61.9 -> 59.0 us per step, with the zero products and beds below) */
    const bool low = r > 0. && r < 0.5;
    if (r <= 0.) {
      A = T(1.);
    } else if (low || (r > 1. && r < 2.)) {
      const T k = 1. - fabs(c);
      A = 1. - (low ? twice(k) : k) * r;
    } else if (r > 0.5 && r < 1.) {
      A = fabs(c);
    } else {
      A = twice(fabs(c)) - 1.;
    }
  } else if (ilim == 2) {
    if (r <= 0.) A = T(1.);
    else A = 1. - twice(1. - fabs(c)) * r / (1. + r);
  } else if (ilim == 3) {
    if (r <= 0.) A = T(1.);
    else A = 1. - (1. - fabs(c)) * r * (1. + r) / (1. + r * r);
  } else if (ilim == 4) {
    if (r <= 0.) A = T(1.);
    else if (r <= 1.) A = 1. - (1. - fabs(c)) * r;
    else A = fabs(c);
  }
  return A;
}

template <class T>
CF_HD CF_INLINE double sgn1(const T& x) { return copysign(1.0, val(x)); }

/* sgn1(x) * y, the reference's dsign(1.d0, x) * y: for every y that is not NaN the IEEE product
 * of +-1 and y is y with the sign of x multiplied in, a sign-bit flip (no FP64 instruction). */
CF_HD CF_INLINE double sgnmul(double x, double y) {
  uint64_t bx, by;
  memcpy(&bx, &x, sizeof(bx));
  memcpy(&by, &y, sizeof(by));
  by ^= bx & 0x8000000000000000ull;
  double r;
  memcpy(&r, &by, sizeof(r));
  return r;
}
template <class T>
CF_HD CF_INLINE T sgnmul(const T& x, const T& y) { return sgn1(x) * y; }

/* x, or (freeze) its value taken as a constant of the linearization; the same number either way. */
template <class T>
CF_HD CF_INLINE T held(const T& x, bool freeze) { return freeze ? T(val(x)) : x; }

/* Second-order WAF (IFLUX 3, flux_riemann.cuf:720-900) for both sides.  Inputs: the
 * reconstructed, masked edge-frame states of A (left) and B (right), the upwind
 * reconstructions (h, v) of each side, dt, and the distances d_mrl, d_mkvol (A), d_mkvoisin (B).
 * freeze_r (linearizations only) holds the limiter ratios r constant: r = dupw / (dloc + eps)
 * divides differences that are at round-off level in still water, and its derivative there
 * (~1/eps) carries no information. */
template <class T>
CF_HD CF_INLINE void waf_flux(double g, int ilim, double nx, double ny, double dt, double d_mrl, double y_mrl,
                              double d_mkvol, double y_mkvol, double d_mkvoisin, double y_mkvoisin, T hl, T ul,
                              T vl, T hr, T ur, T vr, T hl_upw, T vl_upw, T hr_upw, T vr_upw, TwoFluxT<T>& F,
                              bool freeze_r = false) {
  const double eps = EPS_SECOND;
  T sl, sr, set;
  if (!wave_speeds(g, eps, hl, ul, hr, ur, sl, sr, set)) {
    F.a1 = F.a2 = F.a3 = F.b1 = F.b2 = F.b3 = T(0.0);
    return;
  }
  const T fl1 = hl * ul, fl2 = hl * (ul * ul) + halve(g * hl * hl);
  const T fr1 = hr * ur, fr2 = hr * (ur * ur) + halve(g * hr * hr);
  const int ra = (sl > 0.) ? 0 : ((sr < 0.) ? 1 : 2);
  const int rb = (-sr > 0.) ? 1 : ((-sl < 0.) ? 0 : 2);
  T h1 = T(0.0), h2 = T(0.0);
  if (ra == 2 || rb == 2) {
    const T den = sr - sl + eps;
    const auto yden = recip(den);
    h1 = div_rn(sr * fl1 - sl * fr1 + sl * sr * (hr - hl), den, yden);
    h2 = div_rn(sr * fl2 - sl * fr2 + sl * sr * (hr * ur - hl * ul), den, yden);
  }
  const T ha1 = (ra == 0) ? fl1 : ((ra == 1) ? fr1 : h1);
  const T ha2 = (ra == 0) ? fl2 : ((ra == 1) ? fr2 : h2);
  const T hb1 = (rb == 0) ? fl1 : ((rb == 1) ? fr1 : h1);
  const T hb2 = (rb == 0) ? fl2 : ((rb == 1) ? fr2 : h2);

  const double dtoverdx = ConstOps<T>::quot(dt, d_mrl, y_mrl);
  const T cr = sr * dtoverdx, cl = sl * dtoverdx, cet = set * dtoverdx;
  const T dloc = div_rn(hr - hl, d_mrl, y_mrl);          /* delta_loc_l = delta_loc_r */
  const T dloc_et = div_rn(vr - vl, d_mrl, y_mrl);
  const T upl = div_rn(hl - hl_upw, d_mkvol, y_mkvol);     /* upwind difference of side A */
  const T upr = div_rn(hr_upw - hr, d_mkvoisin, y_mkvoisin);  /* upwind difference of side B */
  const T upvl = div_rn(vl - vl_upw, d_mkvol, y_mkvol);
  const T upvr = div_rn(vr_upw - vr, d_mkvoisin, y_mkvoisin);
  const T ret_a = held(((set > 0.) ? upvl : upvr) / (dloc_et + eps), freeze_r);

  /* side A (:854-899) */
  {
    const T den = dloc + eps;
    const auto yd = recip(den);
    const T rl = held(div_rn((sl > 0.) ? upl : upr, den, yd), freeze_r);
    const T rr = held(div_rn((sr > 0.) ? upl : upr, den, yd), freeze_r);
    const T ll = waf_limiter(ilim, rl, cl);
    const T lr = waf_limiter(ilim, rr, cr);
    const T le = waf_limiter(ilim, ret_a, cet);
    const T wl = halve(1. + sgnmul(sl, ll));
    const T wlet = halve(1. + sgnmul(set, le));
    const T wlr = halve(sgnmul(sr, lr) - sgnmul(sl, ll));
    const T wr = halve(1. - sgnmul(sr, lr));
    const T wret = halve(1. - sgnmul(set, le));
    const T fw1 = wl * fl1 + wlr * ha1 + wr * fr1;
    const T fw2 = wl * fl2 + wlr * ha2 + wr * fr2;
    const T fw3 = (wlet * vl + wret * vr) * fw1;
    F.a1 = fw1;
    F.a2 = nx * fw2 - ny * fw3;
    F.a3 = ny * fw2 + nx * fw3;
  }
  /* side B: the same formulas on the mirrored states.  Its local difference is
   * (hl - hr)/d = -dloc, its upwind differences are minus A's (for the wave it tests), the
   * tangential ones coincide; its Courant numbers are -cr, -cl, -cet. */
  {
    const T den = -dloc + eps;
    const auto yd = recip(den);
    const T rl = held(div_rn((-sr > 0.) ? -upr : -upl, den, yd), freeze_r);
    const T rr = held(div_rn((-sl > 0.) ? -upr : -upl, den, yd), freeze_r);
    /* B's tangential ratio differs from A's only when s* == 0 (or is NaN) */
    const T ret_b = (set > 0. || set < 0.) ? ret_a : held(((-set > 0.) ? upvr : upvl) / (dloc_et + eps), freeze_r);
    const T ll = waf_limiter(ilim, rl, -cr);
    const T lr = waf_limiter(ilim, rr, -cl);
    const T le = waf_limiter(ilim, ret_b, -cet);
    const T nsl = opposite(sl), nsr = opposite(sr), nset = opposite(set);
    const T wl = halve(1. + sgnmul(nsr, ll));
    const T wlet = halve(1. + sgnmul(nset, le));
    const T wlr = halve(sgnmul(nsl, lr) - sgnmul(nsr, ll));
    const T wr = halve(1. - sgnmul(nsl, lr));
    const T wret = halve(1. - sgnmul(nset, le));
    /* mirrored physical fluxes: FL' = (-fr1, fr2), FR' = (-fl1, fl2), HLL' = (-hb1, hb2) */
    const T fw1 = -(wl * fr1 + wlr * hb1 + wr * fl1);
    const T fw2 = wl * fr2 + wlr * hb2 + wr * fl2;
    const T fw3 = -(wlet * vr + wret * vl) * fw1;
    /* B's normal is -n: (fw1, -n1 fw2 + n2 fw3, -n2 fw2 - n1 fw3) */
    F.b1 = fw1;
    F.b2 = -nx * fw2 + ny * fw3;
    F.b3 = -ny * fw2 - nx * fw3;
  }
}

/* ---- MUSCL-Hancock (IFLUX 4) ----------------------------------------------------------- */

/* simple_limiter (flux_riemann.cuf:431-463) of an upwind slope r1 and a local slope r2:
 * 0 none, 1 superbee (Fortran's three-argument max / min as two nested ones), 2 van Leer,
 * 3 minmod.  Other ilimiteur values leave the reference's result unset; defined as 0. */
template <class T>
CF_HD CF_INLINE T simple_limiter(int ilim, T r1, T r2) {
  if (ilim == 1) {
    if (r2 > 0.) return dmax(T(0.), dmax(dmin(twice(r1), r2), dmin(r1, twice(r2))));
    return dmin(T(0.), dmin(dmax(twice(r1), r2), dmax(r1, twice(r2))));
  }
  if (ilim == 2) return (r1 * r2 + fabs(r1 * r2)) / (r1 + r2 + EPS_VLEER);
  if (ilim == 3) {
    if (r2 > 0.) return dmax(T(0.), dmin(r1, r2));
    return dmin(T(0.), dmax(r1, r2));
  }
  return T(0.);
}

/* Edge-frame MUSCL-Hancock flux of the side whose element is on the left
 * (solver_Riemann_muscl, flux_riemann.cuf:526-718): limited slopes of the left state (upwind
 * difference over d_up_l, local over d_mrl) and of the right state (local, upwind over
 * d_up_r), face values, the half-step predictor, then HLLC with eps = 1e-16 (single
 * precision).  Inputs are the hydrostatically reconstructed, masked states of both elements
 * and the upwind reconstructions of both sides, all in this side's frame. */
template <class T>
CF_HD CF_INLINE void muscl_side(double g, double tolisec, int ilim, double dtoverdx, double d_mrl, double y_mrl,
                                double d_up_l, double y_up_l, double d_up_r, double y_up_r, T hl, T ul, T vl, T hr,
                                T ur, T vr, T hl_upw, T ul_upw, T vl_upw, T hr_upw, T ur_upw, T vr_upw, T& x1, T& x2,
                                T& x3) {
  const double eps = EPS_SECOND;
  /* data reconstruction I (:560-609) */
  const T dloc1 = div_rn(hr - hl, d_mrl, y_mrl);
  const T dloc2 = div_rn(ur - ul, d_mrl, y_mrl);
  const T dloc3 = div_rn(vr - vl, d_mrl, y_mrl);
  const T dhl = simple_limiter(ilim, div_rn(hl - hl_upw, d_up_l, y_up_l), dloc1);
  const T hll = dmax0(hl - halve(dhl) * d_mrl);
  const T hlr = dmax0(hl + halve(dhl) * d_mrl);
  T ull, vll, ulr, vlr;
  if (hlr < tolisec || hll < tolisec) {
    ulr = vlr = ull = vll = T(0.);
  } else {
    const T dul = simple_limiter(ilim, div_rn(ul - ul_upw, d_up_l, y_up_l), dloc2);
    const T dvl = simple_limiter(ilim, div_rn(vl - vl_upw, d_up_l, y_up_l), dloc3);
    ull = ul - halve(dul) * d_mrl;
    vll = vl - halve(dvl) * d_mrl;
    ulr = ul + halve(dul) * d_mrl;
    vlr = vl + halve(dvl) * d_mrl;
  }
  const T dhr = simple_limiter(ilim, dloc1, div_rn(hr_upw - hr, d_up_r, y_up_r));
  const T hrr = dmax0(hr + halve(dhr) * d_mrl);
  const T hrl = dmax0(hr - halve(dhr) * d_mrl);
  T url, vrl, urr, vrr;
  if (hrl < tolisec || hrr < tolisec) {
    url = vrl = urr = vrr = T(0.);
  } else {
    const T dur = simple_limiter(ilim, dloc2, div_rn(ur_upw - ur, d_up_r, y_up_r));
    const T dvr = simple_limiter(ilim, dloc3, div_rn(vr_upw - vr, d_up_r, y_up_r));
    urr = ur + halve(dur) * d_mrl;
    vrr = vr + halve(dvr) * d_mrl;
    url = ur - halve(dur) * d_mrl;
    vrl = vr - halve(dvr) * d_mrl;
  }
  /* data reconstruction II (:615-621) */
  const double hdt = ConstOps<T>::half(dtoverdx), hg = ConstOps<T>::half(g);
  const T h1 = hlr + hdt * (hll * ull - hlr * ulr);
  const T u1 = ulr + hdt *
                         (hll * (ull * ull) + hg * (hll * hll) - (hlr * (ulr * ulr) + hg * (hlr * hlr)));
  const T v1 = vlr + hdt * (hll * ull * vll - hlr * ulr * vlr);
  const T h2 = hrl + hdt * (hrl * url - hrr * urr);
  const T u2 = url + hdt *
                         (hrl * (url * url) + hg * (hrl * hrl) - (hrr * (urr * urr) + hg * (hrr * hrr)));
  const T v2 = vrl + hdt * (hrl * url * vrl - hrr * urr * vrr);
  /* HLLC (:623-714) */
  T sl, sr, set;
  if (!wave_speeds(g, eps, h1, u1, h2, u2, sl, sr, set)) {
    x1 = x2 = x3 = T(0.);
    return;
  }
  if (sl > 0.) {
    x1 = h1 * u1;
    x2 = h1 * (u1 * u1) + halve(g * h1 * h1);
    x3 = h1 * u1 * v1;
  } else if (sr < 0.) {
    x1 = h2 * u2;
    x2 = h2 * (u2 * u2) + halve(g * h2 * h2);
    x3 = h2 * u2 * v2;
  } else {
    const T fl1 = h1 * u1, fl2 = h1 * (u1 * u1) + halve(g * h1 * h1);
    const T fr1 = h2 * u2, fr2 = h2 * (u2 * u2) + halve(g * h2 * h2);
    const T den = sr - sl + eps;
    const auto yden = recip(den);
    x1 = div_rn(sr * fl1 - sl * fr1 + sl * sr * (h2 - h1), den, yden);
    x2 = div_rn(sr * fl2 - sl * fr2 + sl * sr * (h2 * u2 - h1 * u1), den, yden);
    x3 = (set > 0.) ? x1 * v1 : x1 * v2;
  }
}

/* Discharge of an inlet at time t: debitglob, or a linear ramp from debitglob_start. */
CF_HD CF_INLINE double inlet_discharge(const MemberDev& M, int id, double t) {
  const double q1 = M.debit_end[id - 1];
  if (M.ramp_time > 0.0 && t < M.ramp_time) {
    const double q0 = M.debit_start[id - 1];
    return q0 + (q1 - q0) * (t / M.ramp_time);
  }
  return q1;
}

/* Boundary-edge flux of side A (flux_riemann.cuf:114-171).  surf: for phys_inflow (inlet 3),
 * calcul_surf_entree's sum of length * depth over the edge's inlet at the step's start. */
template <class T>
CF_HD CF_INLINE void boundary_flux(int iflux, const MemberDev& M, int kind, int id, double t, double nx, double ny,
                                   T h, T hu, T hv, double yh, double z, T& f1, T& f2, T& f3, T& q,
                                   double surf = 0.0) {
  const double g = M.gp, tolisec = M.tolisec;
  T hautl, vitul, vitvl;
  to_frame(h, hu, hv, yh, nx, ny, tolisec, hautl, vitul, vitvl);
  f1 = f2 = f3 = T(0.0);
  q = T(0.0);
  if (kind == -1) {
    if (M.inlet == 1) {
      f1 = hautl * vitul;
      f2 = nx * (hautl * (vitul * vitul) + halve(g * (hautl * hautl))) - ny * hautl * vitul * vitvl;
      f3 = ny * (hautl * (vitul * vitul) + halve(g * (hautl * hautl))) + nx * hautl * vitul * vitvl;
    } else if (M.inlet == 2) {
      const double debitnorm = -inlet_discharge(M, id, t) / M.long_entree[id - 1];
      f1 = T(debitnorm);
      f2 = nx * ((debitnorm * debitnorm) / (hautl + tolisec) + halve(g * (hautl * hautl)));
      f3 = ny * ((debitnorm * debitnorm) / (hautl + tolisec) + halve(g * (hautl * hautl)));
      q = T(-debitnorm);
    } else if (M.inlet == 3) {
      /* the inlet's discharge shared in proportion to depth (:127-138); the threshold is the
       * single-precision literal 1e-8 */
      const T debitnorm = (surf > (double)1e-8f) ? -(inlet_discharge(M, id, t) * hautl / surf) : T(0.0);
      f1 = debitnorm;
      f2 = nx * ((debitnorm * debitnorm) / (hautl + tolisec) + halve(g * (hautl * hautl)));
      f3 = ny * ((debitnorm * debitnorm) / (hautl + tolisec) + halve(g * (hautl * hautl)));
      q = -debitnorm;
    }
  } else if (kind == -3) {
    f2 = halve(nx * g * (hautl * hautl));
    f3 = halve(ny * g * (hautl * hautl));
  } else if (kind == -2) {
    if (M.outlet == 1) {
      if (vitul >= 0. && vitul / sqrt(g * hautl) < 1.0) {
        double ho = M.h_sortie[id - 1] - z;
        ho = dmax(0.0, ho);
        f1 = ho * vitul;
        f2 = nx * (ho * (vitul * vitul) + halve(g * (ho * ho))) - ny * ho * vitul * vitvl;
        f3 = ny * (ho * (vitul * vitul) + halve(g * (ho * ho))) + nx * ho * vitul * vitvl;
      } else {
        f2 = halve(nx * g * (hautl * hautl));
        f3 = halve(ny * g * (hautl * hautl));
      }
      q = f1;
    } else {
      /* transmissive outlet: the element is its own neighbour (:169-171), raw depth on the
       * right (:173-181); second-order schemes use first-order HLLC here (their centroid
       * distance to themselves is zero). */
      const double zij = dmax(z, z);
      T hsl = dmax0(hautl + z - zij);
      T hsr = dmax0(((iflux <= 2) ? h : hautl) + z - zij);
      T ul = vitul, vl = vitvl, ur = vitul, vr = vitvl;
      if (hsl < tolisec) { hsl = T(0.); ul = T(0.); vl = T(0.); }
      if (hsr < tolisec) { hsr = T(0.); ur = T(0.); vr = T(0.); }
      TwoFluxT<T> F;
      if (iflux == 2) first_order_flux<2>(g, nx, ny, hsl, ul, vl, hsr, ur, vr, F);
      else first_order_flux<1>(g, nx, ny, hsl, ul, vl, hsr, ur, vr, F);
      f1 = F.a1; f2 = F.a2; f3 = F.a3;
    }
  }
}

/* Upwind reconstruction (h, v) of one side from the states of its upwind elements
 * (flux_riemann.cuf:240-366): a copy of element 1's masked state when d1 < 0 (one upwind
 * element, or the first-order fallback), else the centroid-distance weighted average of two. */
template <class T>
CF_HD CF_INLINE void upwind_mix(T h1, T hu1, T hv1, double yh1, T h2, T hu2, T hv2, double yh2, double d1,
                                double d2, double ds, double ysum, double nx, double ny, double tolisec, T& hu_,
                                T& vu_) {
  T a, va;
  to_frame_t(h1, hu1, hv1, yh1, nx, ny, tolisec, a, va);
  if (T(d1) < 0.0) {
    hu_ = a;
    vu_ = va;
    return;
  }
  T b, vb;
  to_frame_t(h2, hu2, hv2, yh2, nx, ny, tolisec, b, vb);
  hu_ = div_rn(d1 * a + d2 * b, ds, ysum);
  vu_ = div_rn(d1 * va + d2 * vb, ds, ysum);
}
template <class T>
CF_HD CF_INLINE void upwind_mix(T h1, T hu1, T hv1, double yh1, T h2, T hu2, T hv2, double yh2, double d1,
                                double d2, double ysum, double nx, double ny, double tolisec, T& hu_, T& vu_) {
  upwind_mix(h1, hu1, hv1, yh1, h2, hu2, hv2, yh2, d1, d2, d1 + d2, ysum, nx, ny, tolisec, hu_, vu_);
}

/* The bed elevation of an upwind reconstruction (flux_riemann.cuf:320-366): static, so the host
 * preprocessing evaluates it once per edge side. */
CF_HD CF_INLINE double upwind_bed(double z1, double z2, double d1, double d2, double ysum) {
  return (d1 < 0.0) ? z1 : div_rn(d1 * z1 + d2 * z2, d1 + d2, ysum);
}

/* The same, loading the elements' states (w = RN(1/h)), in the edge's arithmetic type T; ds = d1 + d2
 * and
 * ysum = RN(1/ds) of a pair. */
template <class T>
CF_HD CF_INLINE void upwind_state(const double4* U, int i1, int i2, double d1, double d2, double ds, double ysum,
                                  double nx, double ny, double tolisec, T& hu_, T& vu_) {
  const double4 A1 = ld4(U + i1);
  if (T(d1) < 0.0) {
    upwind_mix(T(A1.x), T(A1.y), T(A1.z), A1.w, T(0.0), T(0.0), T(0.0), 0.0, d1, d2, ds, ysum, nx, ny, tolisec,
               hu_, vu_);
    return;
  }
  const double4 A2 = ld4(U + i2);
  upwind_mix(T(A1.x), T(A1.y), T(A1.z), A1.w, T(A2.x), T(A2.y), T(A2.z), A2.w, d1, d2, ds, ysum, nx, ny, tolisec,
             hu_, vu_);
}

/* The MUSCL form: (h, u_n, u_t) of one side's upwind reconstruction (flux_riemann.cuf:240-366
 * with the normal velocity as well). */
template <class T>
CF_HD CF_INLINE void upwind_state3(const double4* U, int i1, int i2, double d1, double d2, double ds, double ysum,
                                   double nx, double ny, double tolisec, T& hu_, T& uu_, T& vu_) {
  const double4 A1 = ld4(U + i1);
  T a, ua, va;
  to_frame(T(A1.x), T(A1.y), T(A1.z), A1.w, nx, ny, tolisec, a, ua, va);
  if (T(d1) < 0.0) {
    hu_ = a;
    uu_ = ua;
    vu_ = va;
    return;
  }
  const double4 A2 = ld4(U + i2);
  T b, ub, vb;
  to_frame(T(A2.x), T(A2.y), T(A2.z), A2.w, nx, ny, tolisec, b, ub, vb);
  hu_ = div_rn(d1 * a + d2 * b, ds, ysum);
  uu_ = div_rn(d1 * ua + d2 * ub, ds, ysum);
  vu_ = div_rn(d1 * va + d2 * vb, ds, ysum);
}

/* ---- one edge ------------------------------------------------------------------------- */

/* Static data of an interior edge beyond its normal: length, centroid distance and, for the
 * second-order scheme, the upwind distances and reciprocals. */
struct EdgeGeo {
  double nx, ny, len, d_mrl;
  double y_mrl, d_mkvol, y_mkvol, d_mkvoisin, y_mkvoisin;
  double ysum_a, ysum_b;  /* RN(1/(d1+d2)) of the upwind pairs of sides A and B */
};

/* Both sides' slot values of an interior edge: out[0..4] = side A {f1, f2, f3} * len and its
 * bed source {bx, by}; out[5..9] the same for side B.  hl_upw .. vr_upw are the upwind
 * reconstructions of sides A and B (second order only), zl_upw / zr_upw their bed elevations. */
template <int IFLUX, class T>
CF_HD CF_INLINE void interior_edge(const MemberDev& M, int ilim, int flux_mode, const EdgeGeo& G, double dt, T hA,
                                   T huA, T hvA, double zml, double yhA, T hB, T huB, T hvB, double zmr, double yhB,
                                   T hl_upw, T vl_upw, double zl_upw, T hr_upw, T vr_upw, double zr_upw, T out[10],
                                   bool freeze_r = false) {
  const double g = M.gp, tolisec = M.tolisec;
  const double nx = G.nx, ny = G.ny, len = G.len;
  const double zij = val(dmax(T(zml), T(zmr)));
  T hautl, vitul, vitvl, hautr, vitur, vitvr;
  to_frame(hA, huA, hvA, yhA, nx, ny, tolisec, hautl, vitul, vitvl);
  to_frame(hB, huB, hvB, yhB, nx, ny, tolisec, hautr, vitur, vitvr);
  /* the depths above the higher bed, of the raw depths (the bed source's, and the reconstruction of a
   * wet side).  A masked depth of 0 reconstructs to +0 on any bed: z - max(z, z') is not positive, or
   * NaN, and the max with 0 gives +0. */
  const bool wetA = hA > tolisec, wetB = hB > tolisec;
  const T ha = dmax0(hA + zml - zij), hb = dmax0(hB + zmr - zij);
  TwoFluxT<T> F;
  if (IFLUX <= 2) {
    /* hydrostatic reconstruction (:176-181, :200-210): A from its masked depth, B from its
     * raw depth; the raw and masked depths differ only for 0 < h <= tolisec, where side B's
     * own evaluation (B masked, A raw) is computed separately. */
    T hijet = wetA ? ha : T(0.0);
    T hjiet = hb;
    T ul = vitul, vl = vitvl, ur = vitur, vr = vitvr;
    if (hijet < tolisec) { hijet = T(0.); ul = T(0.); vl = T(0.); }
    if (hjiet < tolisec) { hjiet = T(0.); ur = T(0.); vr = T(0.); }
    first_order_flux<IFLUX>(g, nx, ny, hijet, ul, vl, hjiet, ur, vr, F);
    if ((!wetA && hA != 0.0) || (!wetB && hB != 0.0)) {   /* a side's masked depth differs from its raw one */
      T bl = wetB ? hb : T(0.0), br = ha;
      T bul = -vitur, bvl = -vitvr, bur = -vitul, bvr = -vitvl;
      if (bl < tolisec) { bl = T(0.); bul = T(0.); bvl = T(0.); }
      if (br < tolisec) { br = T(0.); bur = T(0.); bvr = T(0.); }
      TwoFluxT<T> Gm;
      first_order_flux<IFLUX>(g, -nx, -ny, bl, bul, bvl, br, bur, bvr, Gm);
      F.b1 = Gm.a1;
      F.b2 = Gm.a2;
      F.b3 = Gm.a3;
    }
  } else {
    /* hydrostatic reconstruction of the four states (:370-400) */
    T hijet = wetA ? ha : T(0.0);
    T hlu = dmax0(hl_upw + zl_upw - zij);
    T hjiet = wetB ? hb : T(0.0);
    T hru = dmax0(hr_upw + zr_upw - zij);
    T ul = vitul, vl = vitvl, ur = vitur, vr = vitvr, vlu = vl_upw, vru = vr_upw;
    if (hijet < tolisec) { hijet = T(0.); ul = T(0.); vl = T(0.); }
    if (hlu < tolisec) { hlu = T(0.); vlu = T(0.); }
    if (hjiet < tolisec) { hjiet = T(0.); ur = T(0.); vr = T(0.); }
    if (hru < tolisec) { hru = T(0.); vru = T(0.); }
    waf_flux(g, ilim, nx, ny, dt, G.d_mrl, G.y_mrl, G.d_mkvol, G.y_mkvol, G.d_mkvoisin, G.y_mkvoisin, hijet, ul, vl,
             hjiet, ur, vr, hlu, vlu, hru, vru, F, freeze_r);
  }
  if (flux_mode == 1) {
    F.b1 = -F.a1;
    F.b2 = -F.a2;
    F.b3 = -F.a3;
  }
  /* bed-slope source of both sides from the raw depths (source_terms.cuf:90-97) */
  const double hg = ConstOps<T>::half(g);
  const T ta = hg * (ha * ha - hA * hA) * len;
  const T tb = hg * (hb * hb - hB * hB) * len;
  out[0] = F.a1 * len;
  out[1] = F.a2 * len;
  out[2] = F.a3 * len;
  out[3] = ta * nx;
  out[4] = ta * ny;
  out[5] = F.b1 * len;
  out[6] = F.b2 * len;
  out[7] = F.b3 * len;
  out[8] = -(tb * nx);
  out[9] = -(tb * ny);
}

/* interior_edge for MUSCL-Hancock (IFLUX 4), the whole-edge form that the CPU tests hold the dry shortcut
 * against (the step goes by EdgeSide): the reference evaluates the edge from each of its
 * elements in that element's frame.  Side B's frame normal is -n, so its inputs are A's
 * frame values with the elements swapped and the velocities negated, which is what B's own
 * masking and upwind averaging produce; each side's limited reconstruction is evaluated in
 * full (its slopes are not mirror images of the other side's).  upA / upB: (h, u_n, u_t) of
 * the upwind reconstructions of sides A and B in A's frame, zl_upw / zr_upw their beds. */
template <class T>
CF_HD CF_INLINE void interior_edge_muscl(const MemberDev& M, int ilim, int flux_mode, const EdgeGeo& G, double dt,
                                         T hA, T huA, T hvA, double zml, double yhA, T hB, T huB, T hvB, double zmr,
                                         double yhB, const T upA[3], double zl_upw, const T upB[3], double zr_upw,
                                         T out[10]) {
  const double g = M.gp, tolisec = M.tolisec;
  const double nx = G.nx, ny = G.ny, len = G.len;
  const double zij = val(dmax(T(zml), T(zmr)));
  T hautl, vitul, vitvl, hautr, vitur, vitvr;
  to_frame(hA, huA, hvA, yhA, nx, ny, tolisec, hautl, vitul, vitvl);
  to_frame(hB, huB, hvB, yhB, nx, ny, tolisec, hautr, vitur, vitvr);
  /* hydrostatic reconstruction of the four states (:370-400); a masked depth reconstructs to +0 (see
   * interior_edge) */
  const T ha = dmax0(hA + zml - zij), hb = dmax0(hB + zmr - zij);
  T hijet = hA > tolisec ? ha : T(0.0);
  T hlu = dmax0(upA[0] + zl_upw - zij);
  T hjiet = hB > tolisec ? hb : T(0.0);
  T hru = dmax0(upB[0] + zr_upw - zij);
  T ul = vitul, vl = vitvl, ur = vitur, vr = vitvr;
  T ulu = upA[1], vlu = upA[2], uru = upB[1], vru = upB[2];
  if (hijet < tolisec) { hijet = T(0.); ul = T(0.); vl = T(0.); }
  if (hlu < tolisec) { hlu = T(0.); ulu = T(0.); vlu = T(0.); }
  if (hjiet < tolisec) { hjiet = T(0.); ur = T(0.); vr = T(0.); }
  if (hru < tolisec) { hru = T(0.); uru = T(0.); vru = T(0.); }
  const double dtoverdx = ConstOps<T>::quot(dt, G.d_mrl, G.y_mrl);
  TwoFluxT<T> F;
  T x1, x2, x3;
  muscl_side(g, tolisec, ilim, dtoverdx, G.d_mrl, G.y_mrl, G.d_mkvol, G.y_mkvol, G.d_mkvoisin, G.y_mkvoisin, hijet,
             ul, vl, hjiet, ur, vr, hlu, ulu, vlu, hru, uru, vru, x1, x2, x3);
  F.a1 = x1;
  F.a2 = nx * x2 - ny * x3;
  F.a3 = ny * x2 + nx * x3;
  if (flux_mode == 1) {
    F.b1 = -F.a1;
    F.b2 = -F.a2;
    F.b3 = -F.a3;
  } else {
    T y1, y2, y3;
    muscl_side(g, tolisec, ilim, dtoverdx, G.d_mrl, G.y_mrl, G.d_mkvoisin, G.y_mkvoisin, G.d_mkvol, G.y_mkvol,
               hjiet, -ur, -vr, hijet, -ul, -vl, hru, -uru, -vru, hlu, -ulu, -vlu, y1, y2, y3);
    const double mx = -nx, my = -ny;
    F.b1 = y1;
    F.b2 = mx * y2 - my * y3;
    F.b3 = my * y2 + mx * y3;
  }
  /* bed-slope source of both sides from the raw depths (source_terms.cuf:90-97) */
  const double hg = ConstOps<T>::half(g);
  const T ta = hg * (ha * ha - hA * hA) * len;
  const T tb = hg * (hb * hb - hB * hB) * len;
  out[0] = F.a1 * len;
  out[1] = F.a2 * len;
  out[2] = F.a3 * len;
  out[3] = ta * nx;
  out[4] = ta * ny;
  out[5] = F.b1 * len;
  out[6] = F.b2 * len;
  out[7] = F.b3 * len;
  out[8] = -(tb * nx);
  out[9] = -(tb * ny);
}

/* ---- one side of an edge ---------------------------------------------------------------- */

/* The limiter of one wave, out of line: a side evaluates three, and its code has to stay in the
 * instruction cache (WAF 1M: 250 us per step with the three in place, 248 called). */
#ifdef __CUDACC__
template <class T>
static __host__ __device__ __noinline__ T side_limiter(int ilim, T r, T c) { return waf_limiter(ilim, r, c); }
#else
template <class T>
inline T side_limiter(int ilim, T r, T c) { return waf_limiter(ilim, r, c); }
#endif

#ifdef __CUDACC__
#define CF_RARE static __host__ __device__ __noinline__
#else
#define CF_RARE static
#endif
/* The flux of a side with the reconstructed state (h, u, v) towards the right state (hr, ur, vr), by
 * itself, where the other side's is not its mirror image (IFLUX 1, 2): rare, out of line, in plain doubles
 * (the same bits). */
template <int IFLUX>
CF_RARE void one_sided_flux(double g, double nx, double ny, double h, double u, double v, double hr, double ur, double vr,
                            double o[3]) {
  TwoFluxT<double> F;
  first_order_flux<IFLUX>(g, nx, ny, h, u, v, hr, ur, vr, F);
  o[0] = F.a1;
  o[1] = F.a2;
  o[2] = F.a3;
}

/* +0 a b c of finite factors */
CF_HD CF_INLINE double zero_like(double a, double b, double c) {
  return dbl_hd((dbits_hd(a) ^ dbits_hd(b) ^ dbits_hd(c)) & 0x8000000000000000ull);
}

/* Both sides of an interior edge, evaluated in lockstep, each in its own frame (normal out of its own
 * element) exactly as the reference evaluates the edge from each of its elements
 * (flux_riemann.cuf:33-426), the sign of a zero wave speed included (mirrored()).  On the GPU the two sides are two neighbouring lanes; on the host two
 * objects.  What one side computes the other one needs mirrored (depths equal, normal and tangential
 * velocities negated, s_L' = -s_R, the mass flux negated: all exact), so every quantity of one side is
 * computed once, by its side, and offered to the other in x[]; after an exchange y[] holds the other
 * side's x[].  A value that both need in the same form (a sum of the two depths, the HLL quotients, the
 * contact speed's numerator and denominator) is computed by one side while the other computes a second
 * such value with the same instruction.  The stages are
 *
 *   frame      own frame state, hydrostatic reconstruction          x: h, u, v (first order: and the
 *                                                                      raw depth's reconstruction;
 *                                                                      MUSCL: the upwind h, u, v)
 *   speeds1    celerity; h + h' on side 0, u' - u on side 1         x: a, sum
 *   speeds2    s_L, the own term of s*'s denominator, own flux      x: s_L, d, f1, f2
 *   hll        own term of s*'s numerator, one HLL quotient per side;
 *              WAF: one local slope per side, both upwind slopes    x: t2, q, slope, up_h, up_v
 *   contact1   s*'s numerator on side 0, denominator on side 1      x: it
 *   contact2   s*; IFLUX 2: the own star flux                       x: its three components
 *   finish     the side's flux and bed source in the global frame
 *
 * A lane has half the code, half the live values and half the dependent chain of a thread that
 * evaluates a whole edge, for the ~6 FP64 sums per edge that both sides repeat: WAF 201k triangles
 * (fully wet), the edge kernel: 141 us with 608 local memory instructions per 32 edges -> 120 us with
 * 232 (117 with the quotients by known reciprocals). */
template <int IFLUX, class T>
struct EdgeSide {
  int side;                      /* 0: the edge's first element (its normal points out of it), 1: the second */
  double g, tolisec, nx, ny, len;
  T x[6], y[6];
  T h0, hw;                      /* own raw depth; the raw depth's reconstruction */
  T h, u, v;                     /* reconstructed, masked state, own frame */
  T hr, ur, vr;                  /* the other side's, in the own frame */
  T gh, a, s, as_, sl, sr, d0, f1, f2, fr1, fr2;
  T t2, d, q1, q2, set;          /* q1, q2: HLL mass and momentum flux */
  T hup, uup, vup, sloc, sloct, up_h, up_v, upr_h, upr_v;   /* WAF */
  T e1, e2, e3;                  /* IFLUX 2 */
  double dt, d_mrl, y_mrl, d_up, y_up;
  bool thin;                     /* neither reconstructed depth above eps */
  T hraw;                        /* first order: the other side's reconstruction from its raw depth */

  static constexpr CF_HD CF_INLINE double eps() { return IFLUX == 1 ? EPS_HLLC : IFLUX == 2 ? EPS_RIADH : EPS_SECOND; }
  /* both reconstructed depths below eps: zero flux */
  CF_HD CF_INLINE bool dry() const { return thin && h < eps() && hr < eps(); }
  /* a depth of exactly eps and none above: the reference's wave speeds of the two sides are then not mirror
   * images of one another (each takes the right state's for both), so that each side evaluates its own.  (Not
   * so with WAF, whose eps is a depth of 1e-16: the code of the case alone cost its step 2 % in spilled
   * registers, 201k triangles 149 -> 153 us.) */
  CF_HD CF_INLINE bool film() const { return IFLUX <= 2 && thin && !(h < eps() && hr < eps()); }

  /* U: own state; z, zo: beds of the own and of the other element */
  CF_HD CF_INLINE void frame(const MemberDev& M, int side_, double nx_, double ny_, double len_, const double4& U,
                             double z, double zo) {
    side = side_;
    g = M.gp;
    tolisec = M.tolisec;
    nx = nx_;
    ny = ny_;
    len = len_;
    h0 = T(U.x);
    T hm;
    to_frame(h0, T(U.y), T(U.z), U.w, nx, ny, tolisec, hm, u, v);
    const bool wet = h0 > tolisec;
    const double zij = val(dmax(T(z), T(zo)));
    hw = dmax0(h0 + z - zij);     /* a masked depth reconstructs to +0 (see interior_edge) */
    h = wet ? hw : T(0.0);
    if (h < tolisec) { h = T(0.); u = T(0.); v = T(0.); }
    x[0] = h;
    x[1] = u;
    x[2] = v;
    /* the other side reconstructs this one from its raw depth (:176-181), with the masked velocities */
    if (IFLUX <= 2) x[3] = hw < tolisec ? T(0.) : hw;
  }
  /* second order: the side's upwind reconstruction from its upwind elements i1, i2 (distances d1, d2;
   * d1 < 0: a copy of i1; bed zu), the time step and the distances to the other element and to the
   * upwind reconstruction */
  CF_HD CF_INLINE void upwind(const double4* U, int i1, int i2, double d1, double d2, double zu, double z, double zo,
                              double dt_, double d_mrl_, double y_mrl_, double d_up_, double y_up_) {
    dt = dt_;
    d_mrl = d_mrl_;
    y_mrl = y_mrl_;
    d_up = d_up_;
    y_up = y_up_;
    /* of a pair d_up = (d1 + d2) / 2, so d1 + d2 and its reciprocal are exact scalings */
    const double ds = ConstOps<T>::dbl(d_up), ysum = ConstOps<T>::half(y_up);
    T hu_;
    if (IFLUX == 4) upwind_state3(U, i1, i2, d1, d2, ds, ysum, nx, ny, tolisec, hu_, uup, vup);
    else upwind_state(U, i1, i2, d1, d2, ds, ysum, nx, ny, tolisec, hu_, vup);
    hup = dmax0(hu_ + zu - val(dmax(T(z), T(zo))));
    if (hup < tolisec) { hup = T(0.); vup = T(0.); uup = T(0.); }
    if (IFLUX == 4) {
      x[3] = hup;
      x[4] = uup;
      x[5] = vup;
    }
  }
  CF_HD CF_INLINE void speeds1() {
    hr = y[0];
    ur = -y[1];
    vr = -y[2];
    if (IFLUX <= 2) hraw = y[3];
    thin = !(h > eps()) && !(hr > eps());
    gh = g * h;
    a = sqrt(gh);
    s = (side ? ur : h) + (side ? -u : hr);
    x[0] = a;
    x[1] = s;
  }
  CF_HD CF_INLINE void speeds2() {
    const T ar = y[0];
    const T hs = side ? y[1] : s, du = side ? s : y[1];
    as_ = a + ar;
    const T het = halve(hs) - quarter(du * hs / as_);
    const bool wl = h > eps(), wr = hr > eps();
    T pq;
    if (lt_nonneg(het, h)) pq = T(1.);
    else pq = wl ? sqrt(halve(het + h) * het / (h * h)) : T(0.);
    const T sub = wl ? (wr ? a * pq : a) : twice(ar);
    sl = (wl ? u : ur) - sub;
    d0 = u - sl;
    f1 = h * u;
    f2 = h * (u * u) + halve(gh * h);
    d = h * d0;
    x[0] = sl;
    x[1] = d;
    x[2] = f1;
    x[3] = f2;
  }
  CF_HD CF_INLINE void hll() {
    sr = IFLUX == 3 ? mirrored(y[0]) : -y[0];   /* only WAF looks at the sign of a zero speed */
    s = y[1];                      /* the other side's denominator term, negated in the own frame */
    fr1 = -y[2];
    fr2 = y[3];
    t2 = sr * h * d0;
    const T den = sr - sl + eps();
    const T diff = (side ? fr1 : hr) - (side ? f1 : h);
    const T num = sr * (side ? f2 : f1) - sl * (side ? fr2 : fr1) + sl * sr * diff;
    q1 = num / den;
    x[0] = t2;
    x[1] = q1;
    if (IFLUX == 3) {
      sloc = div_rn((side ? vr : hr) - (side ? v : h), d_mrl, y_mrl);
      up_h = div_rn(h - hup, d_up, y_up);
      up_v = div_rn(v - vup, d_up, y_up);
      x[2] = sloc;
      x[3] = up_h;
      x[4] = up_v;
    }
  }
  CF_HD CF_INLINE void contact1() {
    q2 = side ? q1 : y[1];
    q1 = side ? -y[1] : q1;
    if (IFLUX == 3) {
      sloct = side ? sloc : y[2];
      sloc = side ? -y[2] : sloc;
      upr_h = -y[3];
      upr_v = y[4];
    }
    /* side 0: (s_L h' (u' - s_R)) - (s_R h (u - s_L)); side 1: h' (u' - s_R) - h (u - s_L) of side 0 */
    t2 = (side ? -d : y[0]) - (side ? s : t2);
    x[0] = t2;
  }
  CF_HD CF_INLINE void contact2() {
    const T num = side ? (IFLUX == 3 ? mirrored(y[0]) : -y[0]) : t2, denom = side ? t2 : y[0];
    if (fabs(denom) < eps()) set = halve(u + ur) - (hr - h) * as_ / (h + hr);
    else set = num / denom;
    if (IFLUX == 2) {
      const T f3 = f1 * v;
      const T p = (fabs(sl - set) > eps()) ? h * (-d0) / (sl - set) : T(0.0);
      e1 = f1 + sl * (p - h);
      e2 = f2 + sl * (p * set - f1);
      e3 = f3 + sl * (p * v - h * v);
      x[0] = e1;
      x[1] = e2;
      x[2] = e3;
    }
  }
  /* the side's flux (times the length) and bed source, global frame */
  CF_HD CF_INLINE void finish(int ilim, T out[5]) {
    T x1, x2, x3;
    const int r = (sl > 0.) ? 0 : ((sr < 0.) ? 1 : 2);
    if (IFLUX == 1) {
      x1 = r == 0 ? f1 : (r == 1 ? fr1 : q1);
      x2 = r == 0 ? f2 : (r == 1 ? fr2 : q2);
      x3 = x1 * (r == 0 ? v : (r == 1 ? vr : (set > 0.) ? v : vr));
    } else if (IFLUX == 2) {
      /* 0 < s_L: F_L; 0 < s* and 0 > s_L: star left; 0 > s* and 0 < s_R: star right; else F_R */
      const int k = (0. < sl) ? 0 : ((0. < set && 0. > sl) ? 2 : ((0. > set && 0. < sr) ? 3 : 1));
      x1 = k == 0 ? f1 : (k == 1 ? fr1 : (k == 2 ? e1 : -y[0]));
      x2 = k == 0 ? f2 : (k == 1 ? fr2 : (k == 2 ? e2 : y[1]));
      x3 = k == 2 ? e3 : (k == 3 ? y[2] : (k == 0 ? f1 * v : fr1 * vr));
    } else {
      const T m1 = r == 0 ? f1 : (r == 1 ? fr1 : q1);
      const T m2 = r == 0 ? f2 : (r == 1 ? fr2 : q2);
      const double dtoverdx = ConstOps<T>::quot(dt, d_mrl, y_mrl);
      const T den = sloc + eps();
      const auto yd = recip(den);
      const T rl = div_rn((sl > 0.) ? up_h : upr_h, den, yd);
      const T rr = div_rn((sr > 0.) ? up_h : upr_h, den, yd);
      const T re = ((set > 0.) ? up_v : upr_v) / (sloct + eps());
      const T ll = sgnmul(sl, side_limiter(ilim, rl, sl * dtoverdx));
      const T lr = sgnmul(sr, side_limiter(ilim, rr, sr * dtoverdx));
      const T le = sgnmul(set, side_limiter(ilim, re, set * dtoverdx));
      const T wl = halve(1. + ll), wlr = halve(lr - ll), wr = halve(1. - lr);
      /* a limiter of 1 (a ratio not above 0) makes the weight of its wave's side 0 */
      x1 = mulz(wl, f1) + wlr * m1 + mulz(wr, fr1);
      x2 = mulz(wl, f2) + wlr * m2 + mulz(wr, fr2);
      x3 = (halve(1. + le) * v + halve(1. - le) * vr) * x1;
    }
    out[0] = x1;
    out[1] = nx * x2 - ny * x3;
    out[2] = ny * x2 + nx * x3;
    if (dry()) out[0] = out[1] = out[2] = T(0.0);
    if (IFLUX <= 2 && (hraw != hr || film())) {
      /* a nearly dry other side at rest (0 < h <= tolisec), whose raw depth reaches the higher bed */
      double o[3];
      one_sided_flux<IFLUX>(g, nx, ny, val(h), val(u), val(v), val(hraw), val(ur), val(vr), o);
      out[0] = T(o[0]);
      out[1] = T(o[1]);
      out[2] = T(o[2]);
    }
  }
  /* MUSCL-Hancock: the flux of this side from the exchanged states; d_upr, y_upr: the other side's
   * upwind distance */
  CF_HD CF_INLINE void muscl(int ilim, double d_upr, double y_upr, T out[5]) {
    T x1, x2, x3;
    muscl_side(g, tolisec, ilim, ConstOps<T>::quot(dt, d_mrl, y_mrl), d_mrl, y_mrl, d_up, y_up, d_upr, y_upr, h, u, v,
               y[0], -y[1], -y[2], hup, uup, vup, y[3], -y[4], -y[5], x1, x2, x3);
    out[0] = x1;
    out[1] = nx * x2 - ny * x3;
    out[2] = ny * x2 + nx * x3;
  }
  CF_HD CF_INLINE void bed(T out[5]) {
    const T d2 = hw * hw - h0 * h0;
    if (is_zero(d2) && finite_bits(g) && finite_bits(len) && finite_bits(nx) && finite_bits(ny)) {
      /* a side on the higher bed (x - x is +0): the products' zeros, with their signs */
      out[3] = T(zero_like(g, len, nx));
      out[4] = T(zero_like(g, len, ny));
      return;
    }
    const T t = ConstOps<T>::half(g) * d2 * len;
    out[3] = t * nx;
    out[4] = t * ny;
  }
};

/* The stages of both sides of an edge.  P holds the sides at hand: the lane's own one on the GPU
 * (exchange: shuffles with the neighbouring lane), both on the host. */
template <int IFLUX, class P>
CF_HD CF_INLINE void side_stages(P& p, int ilim, double d_up0, double y_up0, double d_up1, double y_up1) {
  using S = typename P::Side;
  if (IFLUX == 4) {
    p.exchange(6);
    p.each([&](S& s, typename P::T* out) {
      s.muscl(ilim, s.side ? d_up0 : d_up1, s.side ? y_up0 : y_up1, out);
      s.bed(out);
    });
  } else {
    p.exchange(IFLUX == 3 ? 3 : 4);
    p.each([&](S& s, typename P::T*) { s.speeds1(); });
    p.exchange(2);
    p.each([&](S& s, typename P::T*) { s.speeds2(); });
    p.exchange(4);
    p.each([&](S& s, typename P::T*) { s.hll(); });
    p.exchange(IFLUX == 3 ? 5 : 2);
    p.each([&](S& s, typename P::T*) { s.contact1(); });
    p.exchange(1);
    p.each([&](S& s, typename P::T*) { s.contact2(); });
    if (IFLUX == 2) p.exchange(3);
    p.each([&](S& s, typename P::T* out) {
      s.finish(ilim, out);
      s.bed(out);
    });
  }
}

/* The inputs of one side of interior edge e: its element's state U, normal out of that element */
template <int IFLUX, class T>
CF_HD CF_INLINE void side_load(const StepArgs& a, const MemberDev& M, int e, int side, const double4& geo,
                               const double4& U, double dt, EdgeSide<IFLUX, T>& s) {
  const double2 z = ldro(reinterpret_cast<const double2*>(a.ez + e));        /* bed of A, of B */
  const double zo = side ? z.x : z.y, zs = side ? z.y : z.x;
  const double nx = side ? -geo.x : geo.x, ny = side ? -geo.y : geo.y;
  s.frame(M, side, nx, ny, geo.z, U, zs, zo);
  if (IFLUX >= 3) {
    const double zu = ldro(reinterpret_cast<const double*>(a.ez + e) + 2 + side);
    const int2 up = ldro(reinterpret_cast<const int2*>(a.eupw + e) + side);
    const double2 dw = ldro(reinterpret_cast<const double2*>(a.ewts + e) + side);
    const double4 dk = ld4(a.edk + e);
    const double yi = ldro(reinterpret_cast<const double*>(a.einv + e));
    s.upwind(a.Uin, up.x, up.y, dw.x, dw.y, zu, zs, zo, dt, geo.w, yi, side ? dk.y : dk.x, side ? dk.w : dk.z);
  }
}

/* Both sides of an edge, one after another (host) */
template <int IFLUX, class T_>
struct HostPair {
  using T = T_;
  using Side = EdgeSide<IFLUX, T>;
  Side s[2];
  T out[2][5];
  template <class F>
  CF_HD void each(F&& f) {
    f(s[0], out[0]);
    f(s[1], out[1]);
  }
  CF_HD void exchange(int n) {
    for (int k = 0; k < n; ++k) {
      s[0].y[k] = s[1].x[k];
      s[1].y[k] = s[0].x[k];
    }
  }
};

/* Static data of edge e in the form interior_edge takes. */
CF_HD CF_INLINE EdgeGeo edge_geo(const StepArgs& a, int e, bool second, const double4& geo) {
  EdgeGeo G;
  G.nx = geo.x;
  G.ny = geo.y;
  G.len = geo.z;
  G.d_mrl = geo.w;
  G.y_mrl = G.d_mkvol = G.y_mkvol = G.d_mkvoisin = G.y_mkvoisin = G.ysum_a = G.ysum_b = 0.0;
  if (second) {
    const double4 dk = ld4(a.edk + e);    /* d_mkvol, d_mkvoisin and their reciprocals */
    const double4 yi = ld4(a.einv + e);   /* 1/d_mrl, 1/(d1+d2) of A and of B */
    G.y_mrl = yi.x;
    G.d_mkvol = dk.x;
    G.y_mkvol = dk.z;
    G.d_mkvoisin = dk.y;
    G.y_mkvoisin = dk.w;
    G.ysum_a = yi.y;
    G.ysum_b = yi.z;
  }
  return G;
}
CF_HD CF_INLINE EdgeGeo edge_geo(const StepArgs& a, int e, bool second) { return edge_geo(a, e, second, ld4(a.egeo + e)); }

/* One slot's six values.  On the device three 16-byte stores: every slot array starts on a
 * 256-byte boundary (cudaMalloc, the no-allocation scratch) and a slot is 48 bytes, so every slot
 * starts on a 16-byte boundary.  On the host (the CPU harness) plain stores. */
CF_HD CF_INLINE void store_slot(Slot* p, double f1, double f2, double f3, double bx, double by, double q) {
#ifdef __CUDA_ARCH__
  double2* d = reinterpret_cast<double2*>(p);
  d[0] = make_double2(f1, f2);
  d[1] = make_double2(f3, bx);
  d[2] = make_double2(by, q);
#else
  p->f1 = f1;
  p->f2 = f2;
  p->f3 = f3;
  p->bx = bx;
  p->by = by;
  p->q = q;
#endif
}

/* ---- dry regions ------------------------------------------------------------------------ */

/* The two slots of an interior edge whose elements both hold the depth +0 (bit pattern 0), written
 * without evaluating the edge.  The general evaluation gives, for any bed elevations and any upwind
 * states:
 *   - masked depths 0, hydrostatic depths max(0, (+0 + z) - max(z, z')) = +0 (the difference is
 *     <= 0 or NaN, and max(0, .) returns the +0 operand); the first-order and WAF schemes
 *     (IFLUX 1-3) then see both depths below eps and assign +0 to every component of both sides'
 *     flux vectors (the second first-order evaluation is skipped: masked and raw depths agree);
 *   - MUSCL-Hancock (IFLUX 4): the local slopes are (+0 - +0) / d = +0, each limited slope is +0 (the
 *     limiters return their +0 operand for a +0 local slope and an upwind slope of either sign; a
 *     NaN slope of van Leer's 0 / 0 is removed by the max with 0), so the face depths, the clamped
 *     face velocities and the predicted states are +0 and the wave-speed routine gives the frame
 *     flux (+0, +0, +0); rotated back, a2 = nx 0 - ny 0, a3 = ny 0 + nx 0 (side B with -n), signed
 *     zeros formed here by the same operations (the time step must be finite);
 *   - with flux_mode 1 side B's fluxes are the negated side A's;
 *   - the bed source (g/2 (ha^2 - h^2)) len with ha = h = +0: (g/2 * +0) * len, a zero with the
 *     sign of g times the sign of len, then times nx, ny (side B negated).
 * Every product of a zero and a finite number is the zero with the product of the signs, so the
 * slots are these signed zeros whenever g, len, nx and ny are finite; otherwise (returns false)
 * the caller evaluates the edge. */
template <int IFLUX>
CF_HD CF_INLINE bool dry_edge_ok(double g, const double4& geo, double dt) {
  return finite_u(dbits_hd(g)) & finite_u(dbits_hd(geo.x)) & finite_u(dbits_hd(geo.y)) & finite_u(dbits_hd(geo.z)) &
         (IFLUX != 4 || finite_u(dbits_hd(dt)));
}
/* the slot of one side (0 or 1) when dry_edge_ok holds */
template <int IFLUX>
CF_HD CF_INLINE void dry_slot(double g, int flux_mode, const double4& geo, int side, Slot* p) {
  const uint64_t S = 0x8000000000000000ull;
  const uint64_t bg = dbits_hd(g), bnx = dbits_hd(geo.x), bny = dbits_hd(geo.y), bl = dbits_hd(geo.z);
  const uint64_t sl = bl & S;                              /* the sign of len */
  const uint64_t st = (bg & S) ^ sl ^ (side ? S : 0);      /* ta = tb = (g/2 * +0) * len, side B negated */
  /* the flux vector (before * len): the frame flux rotated by n, side B's by -n */
  uint64_t f1 = 0, f2 = 0, f3 = 0;
  const bool neg = side && flux_mode == 1;                 /* minus side A's */
  if (IFLUX == 4) {
    const bool mirror = side && !neg;
    const double x = (mirror ? -geo.x : geo.x) * 0.0, y = (mirror ? -geo.y : geo.y) * 0.0;
    f2 = dbits_hd(x - y);
    f3 = dbits_hd(y + x);
  }
  const uint64_t sf = sl ^ (neg ? S : 0);
  store_slot(p, dbl_hd((f1 & S) ^ sf), dbl_hd((f2 & S) ^ sf), dbl_hd((f3 & S) ^ sf), dbl_hd(st ^ (bnx & S)),
             dbl_hd(st ^ (bny & S)), 0.0);
}
template <int IFLUX>
CF_HD CF_INLINE bool dry_edge_slots(double g, int flux_mode, const double4& geo, Slot* sa, double dt = 0.0) {
  if (!dry_edge_ok<IFLUX>(g, geo, dt)) return false;
  dry_slot<IFLUX>(g, flux_mode, geo, 0, sa);
  dry_slot<IFLUX>(g, flux_mode, geo, 1, sa + 1);
  return true;
}

/* An element area for which a dry element's update is exact zeros: a positive normal number (the
 * sign bit fails the test). */
CF_HD CF_INLINE bool area_ok(double area) {
  uint32_t lo, hi;
  words_u(dbits_hd(area), lo, hi);
  (void)lo;
  return (hi >> 20) - 1u < 2046u;
}

/* The conditions on the element's state and the member under which a dry element's update is
 * (+0, +0, +0, +0), besides area_ok: its depth is +-0, its discharges are finite, dt is finite and
 * tolisec >= 0. */
CF_HD CF_INLINE bool dry_state_ok(const MemberDev& M, const double4& U, double dt) {
  uint32_t tlo, thi;
  words_u(dbits_hd(M.tolisec), tlo, thi);
  /* +0..+inf: sign clear, magnitude at most the infinity's */
  const bool tol_ok = (thi >> 31) == 0 && (thi < 0x7ff00000u || (thi == 0x7ff00000u && tlo == 0));
  return zero_u(dbits_hd(U.x)) && tol_ok && finite_u(dbits_hd(U.y)) && finite_u(dbits_hd(U.z)) &&
         finite_u(dbits_hd(dt));
}

/* The conditions on the element itself under which a dry element's update is (+0, +0, +0, +0). */
CF_HD CF_INLINE bool dry_element_state(const MemberDev& M, const double4& U, const double4& st, double dt) {
  return area_ok(st.x) && dry_state_ok(M, U, dt);
}

/* True when the general update of an element provably returns the state (+0, +0, +0, +0) without
 * flagging it non-finite: dry_element_state holds and every flux and bed-source component of its
 * three slots is +-0.  Then every residual (0 + 0 - rc) / area and (sb + sf - rc) / area is +0 (the
 * friction source of a dry element is +0), each new component is the old one plus +-0 (finite),
 * and the new depth +-0 <= tolisec clamps the state to +0. */
CF_HD CF_INLINE bool dry_element(const MemberDev& M, const double4& U, const double4& st, const Slot& s0,
                                 const Slot& s1, const Slot& s2, double dt) {
  const uint64_t z = (dbits_hd(s0.f1) | dbits_hd(s0.f2) | dbits_hd(s0.f3) | dbits_hd(s0.bx) | dbits_hd(s0.by) |
                      dbits_hd(s1.f1) | dbits_hd(s1.f2) | dbits_hd(s1.f3) | dbits_hd(s1.bx) | dbits_hd(s1.by) |
                      dbits_hd(s2.f1) | dbits_hd(s2.f2) | dbits_hd(s2.f3) | dbits_hd(s2.bx) | dbits_hd(s2.by)) << 1;
  return z == 0 && dry_element_state(M, U, st, dt);
}

/* True when an element's three slots are signed zeros without reading them: nb (cnbr) flags three
 * interior edges with finite normals and lengths (and an area for which area_ok holds), the
 * member's g is finite, and the element and its three neighbours have depth +0 (bits 0), so that
 * every one of its edges took the edge kernel's dry shortcut (edge_body, dry_edge_slots; the
 * element kernel reads the same state and dt).  With dry_state_ok it gives dry_element's answer. */
template <class Ld>
CF_HD CF_INLINE bool dry_neighbourhood(const MemberDev& M, const int4& nb, const double4& U, Ld h_of) {
  if (!(nb.w && dbits_hd(U.x) == 0 && finite_u(dbits_hd(M.gp)))) return false;
  return (dbits_hd(h_of(nb.x)) | dbits_hd(h_of(nb.y)) | dbits_hd(h_of(nb.z))) == 0;
}

/* The slot of boundary edge e (kind ab.y < 0) */
template <int IFLUX>
CF_HD CF_INLINE void boundary_slot(const StepArgs& a, const MemberDev& M, int e, int2 ab, const double4& geo,
                                   const double4& UA, double t, const double* surf) {
  const double len = geo.z;
  const int id = ldro(a.ebid + e);
  const double sf = (surf && ab.y == -1 && M.inlet == 3 && id >= 1 && id <= M.nin) ? surf[id - 1] : 0.0;
  double f1, f2, f3, q;
  boundary_flux(IFLUX, M, ab.y, id, t, geo.x, geo.y, UA.x, UA.y, UA.z, UA.w, ldro(reinterpret_cast<const double*>(a.ez + e)),
                f1, f2, f3, q, sf);
  store_slot(a.slots + 2 * (size_t)e, f1 * len, f2 * len, f3 * len, 0.0, 0.0, q * len);
}

/* Whether the edge at position pos of the order in which a kernel takes its edges forms its products on
 * the integer pipes, by the tuning mask: one answer for each 32 consecutive positions. */
CF_HD CF_INLINE bool int_products(int32_t mask, int pos) { return (mask >> ((pos % TILE_E) >> 5)) & 1; }

/* A side's flux times the length, and its bed source, into its slot */
template <class T>
CF_HD CF_INLINE void store_side(Slot* p, const T out[5], double len) {
  store_slot(p, val(out[0] * len), val(out[1] * len), val(out[2] * len), val(out[3]), val(out[4]), 0.0);
}

/* Interior edge e on the host, whatever its depths: the stages that the edge kernel runs on two lanes */
template <int IFLUX, class T = double>
inline void edge_interior(const StepArgs& a, const MemberDev& M, int e, double dt) {
  const int2 ab = a.ecell[e];
  const double4 geo = a.egeo[e];
  Slot* sa = a.slots + 2 * (size_t)e;
  HostPair<IFLUX, T> p;
  side_load(a, M, e, 0, geo, a.Uin[ab.x], dt, p.s[0]);
  side_load(a, M, e, 1, geo, a.Uin[ab.y], dt, p.s[1]);
  const double4 dk = IFLUX >= 3 ? a.edk[e] : make_double4(0.0, 0.0, 0.0, 0.0);
  side_stages<IFLUX>(p, a.ilimiteur, dk.x, dk.z, dk.y, dk.w);
  if (a.flux_mode == 1)
    for (int k = 0; k < 3; ++k) p.out[1][k] = -p.out[0][k];
  store_side(sa, p.out[0], geo.z);
  store_side(sa + 1, p.out[1], geo.z);
}

/* Fluxes (times the edge length) and bed sources of edge e into its two slots, from the state U of step
 * n, on the host. */
template <int IFLUX, class T = double>
inline void edge_body(const StepArgs& a, const MemberDev& M, int e, double dt, double t, const double* surf = nullptr) {
  const int2 ab = a.ecell[e];
  const double4 geo = a.egeo[e], UA = a.Uin[ab.x];
  if (ab.y < 0) {
    boundary_slot<IFLUX>(a, M, e, ab, geo, UA, t, surf);
    return;
  }
  Slot* sa = a.slots + 2 * (size_t)e;
  const double4 UB = a.Uin[ab.y];
  /* an edge between two dry elements (most of a flood plain that the water has not reached) */
  if ((dbits_hd(UA.x) | dbits_hd(UB.x)) == 0 && dry_edge_slots<IFLUX>(M.gp, a.flux_mode, geo, sa, dt)) return;
  edge_interior<IFLUX, T>(a, M, e, dt);
}

/* ---- one element ------------------------------------------------------------------------ */

/* CFL time step of one element (cfl_condition.cuf:20-37); cflL = cfl * L_cfl. */
CF_HD CF_INLINE double cfl_dt_elem(const MemberDev& M, double cflL, double h, double hu, double hv, double yh) {
  double d = 1000000.0;
  if (h > M.tolisec) {
    const double vu = div_rn(hu, h, yh), vv = div_rn(hv, h, yh);
    const double nv = sqrt(vu * vu + vv * vv);
    const double vmax = dmax(0.01, nv + sqrt(M.gp * fabs(h)));
    d = dmin(cflL / vmax, 1000000.0);
  }
  if (M.is_dt_constant == 1) d = M.constant_dt;
  return d;
}

/* Manning friction of one element (source_terms.cuf:102-210): the source (sf2, sf3) of its
 * state q and the entries m = {m4, m5, m6, m7, m8, m9} of the rows 2 and 3 of the
 * semi-implicit matrix (I - dt/2 J)^-1 (row 1 is (1, 0, 0)).  A dry element, or
 * fricimplic 0, gives m = {0, 1, 0, 0, 0, 1}. */
template <class T>
CF_HD CF_INLINE void friction_terms(const MemberDev& M, double area, double dt, T manning, T q1, T q2, T q3, T& sf2,
                                    T& sf3, T m[6], double yq1) {
  const double gp = M.gp, tolisec = M.tolisec, tol = M.tol;
  sf2 = T(0.);
  sf3 = T(0.);
  m[0] = T(0.); m[1] = T(1.); m[2] = T(0.); m[3] = T(0.); m[4] = T(0.); m[5] = T(1.);
  if (q1 > tolisec) {
    const T yq = recip_h(q1, yq1);
    const T vitu = div_rn(q2, q1, yq), vitv = div_rn(q3, q1, yq);
    T normvit = sqrt(vitu * vitu + vitv * vitv);
    if (normvit < tol) normvit = T(tol);
    const T p13 = rcbrt(q1);                /* q1**(-1/3) */
    sf2 = -(gp * manning * manning * vitu * normvit * area * p13);
    sf3 = -(gp * manning * manning * vitv * normvit * area * p13);
    if (normvit > tol) {
      const T p43 = div_rn(p13, q1, yq);     /* q1**(-4/3) */
      if (M.fricimplic == 1) {
        const auto yn = recip(normvit);
        const T dtgn2h = T(ConstOps<T>::half(dt)) * gp * manning * manning * p43;
        const T af21 = -(7.0 / 3.0 * dtgn2h * vitu * normvit);
        const T af22 = 1.0 + div_rn(dtgn2h * (twice(vitu * vitu) + vitv * vitv), normvit, yn);
        const T af23 = div_rn(dtgn2h * vitu * vitv, normvit, yn);
        const T af31 = -(7.0 / 3.0 * dtgn2h * vitv * normvit);
        const T af32 = af23;
        const T af33 = 1.0 + div_rn(dtgn2h * (vitu * vitu + twice(vitv * vitv)), normvit, yn);
        const T detaf = af22 * af33 - af23 * af32;
        const auto yd = recip(detaf);
        m[0] = div_rn(-(af21 * af33 - af23 * af31), detaf, yd);
        m[1] = div_rn(af33, detaf, yd);
        m[2] = div_rn(-af23, detaf, yd);
        m[3] = div_rn(af21 * af32 - af22 * af31, detaf, yd);
        m[4] = div_rn(-af32, detaf, yd);
        m[5] = div_rn(af22, detaf, yd);
      } else if (M.fricimplic == 2) {
        const T beta = -(dt * gp * manning * manning * normvit * p43);
        const T detaf = (1. - beta) * (1. - beta);
        m[1] = (1. - beta) / detaf;
        m[5] = (1. - beta) / detaf;
      }
    }
  }
}

/* Sources, friction and update of one element (source_terms.cuf:33-211,
 * finite_volumes_method.cuf:283-303) from its state q, the sums rc of its three edge fluxes
 * and sb of its bed sources, its area (and RN(1/area)) and its Manning n.  The wet/dry clamp
 * of the new depth is part of the map. */
template <class T>
CF_HD CF_INLINE void element_core(const MemberDev& M, double area, double yarea, T manning, T q1, T q2, T q3, T rc1,
                                  T rc2, T rc3, T sb2, T sb3, double dt, T& h, T& hu, T& hv, bool& nonfinite,
                                  double yq1) {
  T r1, r2, r3;
  if (M.friction == 1) {
    T sf2, sf3, m[6];
    friction_terms(M, area, dt, manning, q1, q2, q3, sf2, sf3, m, yq1);
    const T ri1 = div_rn(zero_minus(rc1), area, yarea);   /* 0 + 0 - rc1 */
    const T ri2 = div_rn(sb2 + sf2 - rc2, area, yarea);
    const T ri3 = div_rn(sb3 + sf3 - rc3, area, yarea);
    if (M.fricimplic == 1 || M.fricimplic == 2) {
      r1 = first_row(ri1, ri2, ri3);
      r2 = m[0] * ri1 + m[1] * ri2 + m[2] * ri3;
      r3 = m[3] * ri1 + m[4] * ri2 + m[5] * ri3;
    } else {
      r1 = ri1;
      r2 = ri2;
      r3 = ri3;
    }
  } else {
    r1 = div_rn(zero_minus(rc1), area, yarea);
    r2 = div_rn(sb2 - rc2, area, yarea);
    r3 = div_rn(sb3 - rc3, area, yarea);
  }
  h = q1 + dt * r1;
  hu = q2 + dt * r2;
  hv = q3 + dt * r3;
  nonfinite = !(finite_bits(val(h)) && finite_bits(val(hu)) && finite_bits(val(hv)));
  if (h <= M.tolisec) {
    h = T(0.);
    hu = T(0.);
    hv = T(0.);
  }
}

/* The element kernel's general body (element_update without its dry-region shortcut). */
template <class S = double>
CF_HD CF_INLINE double4 element_update_full(const MemberDev& M, const double4 U, const double4 st, const Slot& s0,
                                            const Slot& s1, const Slot& s2, double dt, bool& nonfinite) {
  /* fixed-order sums over the three edges (flux_riemann.cuf:411-426, source_terms.cuf:54-100) */
  const double rc1 = s0.f1 + s1.f1 + s2.f1;
  const double rc2 = s0.f2 + s1.f2 + s2.f2;
  const double rc3 = s0.f3 + s1.f3 + s2.f3;
  const double sb2 = s0.bx + s1.bx + s2.bx;
  const double sb3 = s0.by + s1.by + s2.by;
  S h, hu, hv;
  element_core(M, st.x, st.w, S(st.y), S(U.x), S(U.y), S(U.z), S(rc1), S(rc2), S(rc3), S(sb2), S(sb3), dt, h, hu,
               hv, nonfinite, U.w);
  /* the new state carries RN(1/h) for the next step's quotients by h */
  const double hn = val(h);
  return make_double4(hn, val(hu), val(hv), hn > 0.0 ? val(S(1.0) / h) : 0.0);
}

/* The element kernel's body: st = {area, manning n, cfl*L_cfl, 1/area}.  Returns the new
 * state; sets *nonfinite when it is not finite. */
template <class S = double>
CF_HD CF_INLINE double4 element_update(const MemberDev& M, const double4 U, const double4 st, const Slot& s0,
                                       const Slot& s1, const Slot& s2, double dt, bool& nonfinite) {
  if (dry_element(M, U, st, s0, s1, s2, dt)) {
    /* a dry element that no water reaches this step (its edges carry no flux) */
    nonfinite = false;
    return make_double4(0.0, 0.0, 0.0, 0.0);
  }
  return element_update_full<S>(M, U, st, s0, s1, s2, dt, nonfinite);
}

/* ---- one momentum component of an element ------------------------------------------------- */

/* The update of an element (element_update_full) by two lanes in lockstep, one for each component of the
 * momentum: comp 0 works on hu, comp 1 on hv, with the same formulas under the exchange of the two, and
 * both carry the depth.  x[] is offered to the other lane, y[] is what it offers (as EdgeSide).
 * Stages: velocity (x: u, u^2); friction (x: diagonal entry, first-column entry, ri); update. */
template <class T>
struct ElemSide {
  int comp;
  T x[3], y[3];
  T q1, q, rc1, rcq, sb, vel, sq, ri, ri1, diag, a1, a23, h, qn;
  bool wet, fast, impl;

  /* U: the state; rc1_, rcq_, sb_: the sums of the depth flux, of this component's flux and bed source */
  CF_HD CF_INLINE void velocity(const MemberDev& M, int comp_, const double4& U, double rc1_, double rcq_, double sb_) {
    comp = comp_;
    q1 = T(U.x);
    q = T(comp ? U.z : U.y);
    rc1 = T(rc1_);
    rcq = T(rcq_);
    sb = T(sb_);
    wet = M.friction == 1 && q1 > M.tolisec;
    vel = sq = T(0.0);
    if (wet) {
      vel = div_rn(q, q1, recip_h(q1, U.w));
      sq = vel * vel;
    }
    x[0] = vel;
    x[1] = sq;
  }
  CF_HD CF_INLINE void friction(const MemberDev& M, const double4& U, const double4& st, double dt) {
    const double gp = M.gp, area = st.x, tol = M.tol;
    T sf = T(0.0);
    fast = false;
    impl = M.friction == 1 && (M.fricimplic == 1 || M.fricimplic == 2);
    diag = T(1.0);
    a1 = T(0.0);
    a23 = T(0.0);
    if (wet) {
      const T n = T(st.y), ot = y[0];
      T nv = sqrt(sq + y[1]);
      if (nv < tol) nv = T(tol);
      const T p13 = rcbrt(q1);
      sf = -(gp * n * n * vel * nv * area * p13);
      fast = impl && nv > tol;
      if (fast) {
        const T p43 = div_rn(p13, q1, recip_h(q1, U.w));
        if (M.fricimplic == 1) {
          const auto yn = recip(nv);
          const T d = T(ConstOps<T>::half(dt)) * gp * n * n * p43;
          diag = 1.0 + div_rn(d * (twice(sq) + y[1]), nv, yn);
          a1 = -(7.0 / 3.0 * d * vel * nv);
          a23 = div_rn(d * (comp ? ot : vel) * (comp ? vel : ot), nv, yn);
        } else {
          const T beta = -(dt * gp * n * n * nv * p43);
          diag = (1. - beta) / ((1. - beta) * (1. - beta));
        }
      }
    }
    if (M.friction == 1) {
      ri1 = div_rn(zero_minus(rc1), area, st.w);
      ri = div_rn(sb + sf - rcq, area, st.w);
    } else {
      ri1 = div_rn(zero_minus(rc1), area, st.w);
      ri = div_rn(sb - rcq, area, st.w);
    }
    x[0] = diag;
    x[1] = a1;
    x[2] = ri;
  }
  /* the new depth and momentum component; false when one is not finite */
  CF_HD CF_INLINE bool update(const MemberDev& M, double dt) {
    const T ro = y[2];
    T r1 = ri1, r = ri;
    if (impl) {
      r1 = first_row(ri1, ri, ro);
      if (fast && M.fricimplic == 1) {
        const T det = diag * y[0] - a23 * a23;
        const auto yd = recip(det);
        /* the other side's row is the same with the roles exchanged: -(a b - c) = c - a b */
        const T ma = div_rn(a23 * y[1] - a1 * y[0], det, yd);
        const T own = div_rn(y[0], det, yd) * ri, oth = div_rn(-a23, det, yd) * ro;
        r = ma * ri1 + (comp ? oth : own) + (comp ? own : oth);
      } else if (fast) {
        r = first_row(diag * ri, ri1, ro);
      } else {
        r = first_row(ri, ri1, ro);
      }
    }
    h = q1 + dt * r1;
    qn = q + dt * r;
    const bool ok = finite_val(h) && finite_val(qn);
    if (h <= M.tolisec) {
      h = T(0.);
      qn = T(0.);
    }
    return ok;
  }
};

/* element_update_full by its two components, on the host */
template <class T>
inline double4 element_update_pair(const MemberDev& M, const double4& U, const double4& st, const Slot& s0,
                                   const Slot& s1, const Slot& s2, double dt, bool& nonfinite) {
  ElemSide<T> e[2];
  e[0].velocity(M, 0, U, s0.f1 + s1.f1 + s2.f1, s0.f2 + s1.f2 + s2.f2, s0.bx + s1.bx + s2.bx);
  e[1].velocity(M, 1, U, s0.f1 + s1.f1 + s2.f1, s0.f3 + s1.f3 + s2.f3, s0.by + s1.by + s2.by);
  auto swap = [&](int n) {
    for (int k = 0; k < n; ++k) {
      e[0].y[k] = e[1].x[k];
      e[1].y[k] = e[0].x[k];
    }
  };
  swap(2);
  e[0].friction(M, U, st, dt);
  e[1].friction(M, U, st, dt);
  swap(3);
  const bool ok0 = e[0].update(M, dt), ok1 = e[1].update(M, dt);
  nonfinite = !(ok0 && ok1);
  const double h = val(e[0].h);
  return make_double4(h, val(e[0].qn), val(e[1].qn), h > 0.0 ? val(T(1.0) / e[0].h) : 0.0);
}

}  // namespace cf

#endif
