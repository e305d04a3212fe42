/*
 * cf_xd.h -- binary64 arithmetic that keeps GB300's FP64 pipe for the operations only it can do.
 *
 * GB300 issues one FP64 instruction per warp and SM sub-partition in 76 cycles (64 when it reads one
 * register pair fewer; 5.0e11/s on 152 SMs), a 32-bit integer one in 2 (shifts, logic, additions,
 * IMAD; 64 lanes per clock and SM on each of two pipes) and a 32 x 32 -> 64 multiply-add in 4, beside
 * the FP64 pipe.  So integer sequences of up to ~40 instructions that give the IEEE result exactly
 * replace FP64 instructions at a profit:
 *
 *   comparisons  on the words of the patterns (-0 = +0, NaN compares false), 4 to 6 instructions
 *                against a constant;
 *   products     x * y by four 32-bit multiply-adds of the significands (em_mul, 31);
 *   quotients    a / b by a two-digit long division with a float reciprocal seed (em_div, 44);
 *   roots        sqrt(x) by a two-digit root extraction the same way (em_sqrt, 55);
 *   scalings     x / 2, x / 4, 2 x, negation, |x| and sign transfers as operations on the high word.
 * Each takes the FP64 instruction (out of line, so that the compiler does not evaluate it
 * speculatively on the fast path) wherever the integer path does not cover the case: exponents
 * outside the window of xwindow (zero operands of a product and zero numerators are covered), a tie
 * of a product, subnormal, infinite and NaN operands.
 *
 * XD<MUL> is a double that compares on integers and, with MUL, multiplies, divides (div_rn
 * included) and takes square roots with em_mul, em_div and em_sqrt; sums stay FP64
 * instructions.  Every result is the IEEE binary64 result of the same operation, so code
 * instantiated on XD<...> rounds exactly like the same code on double; which warps use the
 * integer arithmetic is a tuning choice, not a numerical one.
 *
 * What is expanded in place and what is called is a matter of the instruction cache: products and
 * quotients are in place (a call costs ~13 instructions), roots, the products and quotients outside the
 * fast path and the limiter are called.  WAF 201k triangles / dam break 134k, us per step, when it was decided: 154 / 65;
 * with the uncovered products in place 162 / 65; with every quotient called 156 / 66; with every
 * product called too 173 / 74.
 */
#ifndef CF_XD_H
#define CF_XD_H

#include "cf_flux.h"

#ifdef __CUDACC__
#define XD_HD __host__ __device__ __forceinline__
#define XD_NOINLINE static __host__ __device__ __noinline__
#else
#define XD_HD inline
#define XD_NOINLINE static __attribute__((noinline))
#endif
#define XD_FN_MUL XD_HD
#define XD_FN_DIV XD_HD
#define XD_FN_DIVY XD_HD
#define XD_FN_SQRT XD_NOINLINE

namespace cf {

using ::fabs;
using ::sqrt;

XD_HD uint64_t xbits(double x) {
  uint64_t b;
  memcpy(&b, &x, sizeof(b));
  return b;
}
XD_HD double xdbl(uint64_t b) {
  double x;
  memcpy(&x, &b, sizeof(x));
  return x;
}

/* The 32-bit words of a double and back.  On the device opaque register moves: the bit operations
 * then work on the registers of the value as they are, and the compiler neither turns them into FP64
 * instructions nor forms an FP64 sum a second time for its bits. */
XD_HD void xwords(double x, uint32_t& lo, uint32_t& hi) {
#ifdef __CUDA_ARCH__
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(x));
#else
  const uint64_t b = xbits(x);
  lo = (uint32_t)b;
  hi = (uint32_t)(b >> 32);
#endif
}
XD_HD double xjoin(uint32_t lo, uint32_t hi) {
#ifdef __CUDA_ARCH__
  double x;
  asm("mov.b64 %0, {%1, %2};" : "=d"(x) : "r"(lo), "r"(hi));
  return x;
#else
  return xdbl(((uint64_t)hi << 32) | lo);
#endif
}
XD_HD uint32_t xmulhi32(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
/* words (lo, hi) shifted left (right) by n in 0..31: the high (low) word of the result */
XD_HD uint32_t xshl(uint32_t lo, uint32_t hi, uint32_t n) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, n);
#else
  return (uint32_t)(((((uint64_t)hi << 32) | lo) << n) >> 32);
#endif
}
XD_HD uint32_t xshr(uint32_t lo, uint32_t hi, uint32_t n) {
#ifdef __CUDA_ARCH__
  return __funnelshift_r(lo, hi, n);
#else
  return (uint32_t)((((uint64_t)hi << 32) | lo) >> n);
#endif
}
/* (hi + e, lo + r): a rounding increment (or last digit) and the exponent and sign word join the
 * significand in one carry chain */
XD_HD double xround(uint32_t lo, uint32_t r, uint32_t hi, uint32_t e) {
#ifdef __CUDA_ARCH__
  uint32_t l, h;
  asm("add.cc.u32 %0, %2, %3;\n\taddc.u32 %1, %4, %5;" : "=r"(l), "=r"(h) : "r"(lo), "r"(r), "r"(hi), "r"(e));
  return xjoin(l, h);
#else
  const uint64_t s = (uint64_t)lo + r;
  return xjoin((uint32_t)s, hi + e + (uint32_t)(s >> 32));
#endif
}
XD_HD uint64_t xpair(uint32_t lo, uint32_t hi) { return ((uint64_t)hi << 32) | lo; }
/* q (bh, bl) modulo 2^64.  (Differences of such products are plain 64-bit subtractions: written as
 * sub.cc / subc with a shifted low word, the borrow came out wrong where that word was zero.) */
XD_HD uint64_t xmulw(uint32_t q, uint32_t bl, uint32_t bh) {
  const uint64_t p = (uint64_t)q * bl;
  return xpair((uint32_t)p, (uint32_t)(p >> 32) + q * bh);
}
/* both high words have exponent fields in [767, 1278] (2^-256 .. 2^256): the window in which products
 * and quotients are normal numbers whatever the significands */
XD_HD bool xwindow(uint32_t ah, uint32_t bh) {
  const uint32_t k = 0u - (767u << 21);
  return (((ah * 2u + k) | (bh * 2u + k)) & 0xc0000000u) == 0;
}

/* the FP64 instruction, for the operands and results the integer path does not cover (out of line, so
 * that it is not evaluated speculatively on the fast path) */
XD_NOINLINE double xmul_slow(double a, double b) { return a * b; }

/* m + p + 2^32 v as three words: m the middle sum of a product, v its high part, p the high word of its
 * low part */
XD_HD void xadd3(uint64_t m, uint32_t p, uint64_t v, uint32_t& w0, uint32_t& w1, uint32_t& w2) {
#ifdef __CUDA_ARCH__
  asm("{\n\t.reg .u32 a, b, c, d;\n\tmov.b64 {a, b}, %3;\n\tmov.b64 {c, d}, %4;\n\t"
      "add.cc.u32 %0, a, %5;\n\taddc.cc.u32 %1, c, b;\n\taddc.u32 %2, d, 0;\n\t}"
      : "=r"(w0), "=r"(w1), "=r"(w2) : "l"(m), "l"(v), "r"(p));
#else
  const uint64_t t = m + p, u = v + (t >> 32);   /* m < 2^55 */
  w0 = (uint32_t)t;
  w1 = (uint32_t)u;
  w2 = (uint32_t)(u >> 32);
#endif
}

/* a * b, round to nearest even, in integer arithmetic.  The 53-bit significands are multiplied as
 * 21 + 32 bit words: the middle sum stays below 2^55, and of the lowest product only the high word is
 * formed.  With the product in [2^104, 2^106), top tells its length; the result is its leading 53 bits
 * plus the next one (round half up; where the bits after that one that are formed are all zero it may
 * be a tie, which goes to the FP64 instruction with the operands outside the window).
 * Shifts to the left by a variable and the exponent's constants are written as multiply-adds, which
 * spreads the work evenly over the two integer pipes. */
XD_HD double em_mul_fast(double a, double b, bool& bad) {
  uint32_t al, ah, bl, bh;
  xwords(a, al, ah);
  xwords(b, bl, bh);
  const uint32_t ma = (ah & 0xfffffu) | 0x100000u, mb = (bh & 0xfffffu) | 0x100000u;
  uint64_t m = (uint64_t)ma * bl;
  m = (uint64_t)al * mb + m;
  uint32_t w0, w1, w2;
  xadd3(m, xmulhi32(al, bl), (uint64_t)ma * mb, w0, w1, w2);
  const uint32_t top = w2 >> 9;                       /* 1: the product is at least 2^105 */
  const uint32_t rest = xshl(0u, w0, 12u - top);      /* the bits after the 53rd, round bit first */
  const uint32_t e = (ah - ma) + (bh - mb) + (top * 0x100000u - (1022u << 20));
  bad = !xwindow(ah, bh) || rest == 0x80000000u;
  return xround(xshr(w0, w1, 20u + top), rest >> 31, xshr(w1, w2, 20u + top), e);
}
/* a * b where em_mul_fast does not cover it: a signed zero for a zero and a finite operand, else FP64 */
XD_NOINLINE double em_mul_rest(double a, double b) {
  uint32_t al, ah, bl, bh;
  xwords(a, al, ah);
  xwords(b, bl, bh);
  if (((((ah << 1) | al) == 0) | (((bh << 1) | bl) == 0)) & ((~ah & 0x7ff00000u) != 0) & ((~bh & 0x7ff00000u) != 0))
    return xjoin(0u, (ah ^ bh) & 0x80000000u);
  return xmul_slow(a, b);
}
XD_FN_MUL double em_mul(double a, double b) {
  bool bad;
  double r = em_mul_fast(a, b, bad);
  if (__builtin_expect(bad, 0)) r = em_mul_rest(a, b);
  return r;
}

/* Quotients outside the integer path: a signed zero for a zero over a normal number, else FP64 */
XD_NOINLINE double xdiv_slow(double a, double b) {
  uint32_t al, ah, bl, bh;
  xwords(a, al, ah);
  xwords(b, bl, bh);
  if (((ah << 1) | al) == 0 && ((bh >> 20) & 0x7ffu) - 1u < 2046u) return xjoin(0u, (ah ^ bh) & 0x80000000u);
  return a / b;
}

/* bits of an approximation to 1/f, f in (1, 2]: on the device the single-precision reciprocal
 * (rcp.approx.ftz.f32, error at most one unit in the last place); on the host the IEEE float
 * quotient moved by -1, 0 or +1 unit, so host runs exercise the device's error bound */
XD_HD uint32_t xrcp_seed(uint32_t fb, uint32_t salt) {
#ifdef __CUDA_ARCH__
  (void)salt;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fb)));
  return __float_as_uint(r);
#else
  float f;
  memcpy(&f, &fb, sizeof(f));
  const float r = 1.0f / f;
  uint32_t rb;
  memcpy(&rb, &r, sizeof(rb));
  return f == 2.0f ? rb : rb + salt % 3u - 1u;
#endif
}

/* a / b rounded to nearest, in integer arithmetic, by two digits of a long division.  With A, B the
 * significands (2^52 <= A, B < 2^53) and t = (A < B), the result's significand is RN(q),
 * q = A 2^(52 + t) / B in [2^52, 2^53).  Write R* = 2^84 / B (in (2^31, 2^32]) and b = B 2^8.
 *  1. R0 < R*: a float reciprocal of B's leading 24 bits plus one, less 512: R* - R0 <= 1280.
 *  2. R1 = R0 (1 + e), e = 1 - R0 / R* to 31 bits, lowered by 4 units: R* - 5.01 <= R1 <= R*.
 *     Where RN(1/b) is known (em_div_y) R1 is its leading 32 bits after one unit in the last place is
 *     taken off: R* - 1.01 <= R1 <= R* (also for a power of two, whose R* is 2^32).
 *  3. q1 = floor(X R1 / 2^32), X the leading 32 bits of A 2^(10 + t): 0 <= A 2^(30 + t) / B - q1 <=
 *     7.02, so the remainder r1 = A 2^(38 + t) - q1 b is in [0, 7.02 b), below 2^64: formed exactly
 *     modulo 2^64.
 *  4. q2 = floor(r1 R1 / 2^70) from r1's high word: 0 <= r1 2^22 / b - q2 < 1.11.  Q = q1 2^22 + q2
 *     is then within [q - 1.11, q], and RN(q) = Q + 1 exactly when 2 (r1 2^22 - q2 b) > b: the sign
 *     of (2 q2 + 1) b - r1 2^23, again exact modulo 2^64.  (A quotient of two 53-bit numbers is
 *     never a tie.)
 * Only the seed is approximate, and its error is inside the bounds above; every result is the IEEE
 * quotient. */
XD_HD double xquot(uint32_t al, uint32_t ah, uint32_t ma, uint32_t bl, uint32_t bh, uint32_t mb, uint32_t R1) {
  /* 3. */
  const bool lt = (((uint64_t)ma << 32) | al) < (((uint64_t)mb << 32) | bl);
  const uint32_t X = xshl(al, ma, lt ? 11u : 10u);
  const uint32_t b8l = bl << 8, b8h = xshl(bl, mb, 8);
  const uint32_t q1 = xmulhi32(X, R1);
  const uint64_t r1 = xpair(0u, al << (lt ? 7u : 6u)) - xmulw(q1, b8l, b8h);
  /* 4. */
  const uint32_t q2 = xmulhi32((uint32_t)(r1 >> 32), R1) >> 6;
  const uint32_t D = (uint32_t)((xmulw(2u * q2 + 1u, b8l, b8h) - (r1 << 23)) >> 32);
  const uint32_t e = (ah - ma) - (bh - mb) + (lt ? (1021u << 20) : (1022u << 20));
  return xround(q1 << 22, q2 + (D >> 31), q1 >> 10, e);
}
XD_HD uint32_t xsig(uint32_t h) { return (h & 0xfffffu) | 0x100000u; }   /* high word of a significand */

XD_FN_DIV double em_div(double a, double b) {
  uint32_t al, ah, bl, bh;
  xwords(a, al, ah);
  xwords(b, bl, bh);
  if (__builtin_expect(!xwindow(ah, bh), 0)) return xdiv_slow(a, b);
  const uint32_t mb = xsig(bh);
  /* 1., 2. */
  const uint32_t bn = xshl(bl, mb, 11);               /* B's leading 32 bits */
  const uint32_t R0 = xrcp_seed((bn >> 8) + 0x3f000001u, bl) * 256u + (0x80000000u - 0x200u);
  const uint32_t d2 = xmulhi32(bn, R0) * 0xfffffffeu - 4u;
  return xquot(al, ah, xsig(ah), bl, bh, mb, xmulhi32(R0, d2) + R0);
}
/* the same with y = RN(1/b) at hand */
XD_FN_DIVY double em_div_y(double a, double b, double y) {
  uint32_t al, ah, bl, bh, yl, yh;
  xwords(a, al, ah);
  xwords(b, bl, bh);
  xwords(y, yl, yh);
  if (__builtin_expect(!xwindow(ah, bh), 0)) return xdiv_slow(a, b);
  yh -= yl == 0 ? 1u : 0u;
  return xquot(al, ah, xsig(ah), bl, bh, xsig(bh), xshl(yl - 1u, xsig(yh), 11));
}

/* the FP64 square root, for the operands the integer path does not cover; zeros are their own roots */
XD_NOINLINE double xsqrt_slow(double x) {
  uint32_t lo, hi;
  xwords(x, lo, hi);
  if (((hi << 1) | lo) == 0) return x;
  return ::sqrt(x);
}

/* bits of an approximation to 1/sqrt(f), f in (1, 4], within [1/2, 1 - 2^-24]: rsqrt.approx.ftz.f32 on
 * the device (relative error below 2^-22.9); on the host the quotient of 1 and the float root moved
 * by -1, 0 or +1 unit */
XD_HD uint32_t xrsqrt_seed(uint32_t fb, uint32_t salt) {
  uint32_t gb;
#ifdef __CUDA_ARCH__
  (void)salt;
  float g;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(g) : "f"(__uint_as_float(fb)));
  gb = __float_as_uint(g);
#else
  float f;
  memcpy(&f, &fb, sizeof(f));
  const float g = 1.0f / std::sqrt(f);
  memcpy(&gb, &g, sizeof(gb));
  gb = gb + salt % 3u - 1u;
#endif
  gb = gb > 0x3f7fffffu ? 0x3f7fffffu : gb;
  return gb < 0x3f000000u ? 0x3f000000u : gb;
}

/* sqrt(x) rounded to nearest, in integer arithmetic (positive normal x), by two digits.  With X the
 * significand and p the parity of the unbiased exponent, the result's significand is RN(s),
 * s = sqrt(Y), Y = X 2^(52 + p) in [2^104, 2^106).  Write f = X 2^(p - 52) in [1, 4) and
 * G* = 2^32 / sqrt(f).
 *  1. G0 < G*: a float reciprocal root of f's leading 24 bits plus one, less 1024 units.
 *  2. G1 = G0 (1 + (1 - f g^2) / 2) to 31 bits, lowered by 6 units: G* - 8 <= G1 <= G*.
 *  3. s1 = floor(F G1 / 2^32), F the leading 32 bits of f: 0 <= sqrt(f) 2^30 - s1 <= 10, and the
 *     remainder r1 = X 2^(8 + p) - s1^2 is in [0, 2^35.4).
 *  4. s2 = floor(r1 G1 / 2^41) from r1's leading 32 bits: S = s1 2^22 + s2 has 0 <= s - S < 1.41 (the
 *     square of s2 adds at most 0.19), and RN(s) = S + 1 exactly when Y - S^2 > S: the sign of
 *     S^2 + S - Y modulo 2^64.  (s is never halfway between two integers.)
 * Every result is the IEEE root. */
XD_FN_SQRT double em_sqrt(double x) {
  uint32_t xl, xh;
  xwords(x, xl, xh);
  if (xh - 0x100000u >= 0x7fe00000u) return xsqrt_slow(x);   /* zero, subnormal, negative, inf, NaN */
  const uint32_t xm = (xh & 0xfffffu) | 0x100000u;
  const uint32_t p = (~xh >> 20) & 1u;
  /* 1., 2. */
  const uint32_t F = xshr(xl, xm, 22u - p);
  const uint32_t G0 = xrsqrt_seed(xshr(xl, xm, 29) + 0x3f000001u + (p << 23), xl) * 256u + (0x80000000u - 0x400u);
  const uint32_t t = xmulhi32(xmulhi32(G0, G0), F);
  const uint32_t G1 = xmulhi32(G0, 0x7ffffffau - 2u * t) + G0;
  /* 3. */
  const uint32_t s1 = xmulhi32(F, G1);
  const uint64_t r1 = (((((uint64_t)xm << 32) | xl) << 8) << p) - (uint64_t)s1 * s1;
  /* 4. */
  const uint32_t s2 = xmulhi32((uint32_t)(r1 >> 4), G1) >> 5;
  const uint64_t S = (uint64_t)s1 * (1u << 22) + s2;
  const uint64_t D = S * S + S - ((uint64_t)(xl << (20u + p)) << 32);
  const uint32_t e = (((xh + (1023u << 20)) >> 1) & 0x7ff00000u) - 0x100000u;
  return xround((uint32_t)S, (uint32_t)(D >> 63), (uint32_t)(S >> 32), e);
}

/* Comparisons on the words of the patterns: the IEEE results, on the integer pipes.
 *
 * Against a finite constant c of +0 or above the pattern of x compares as a signed integer (a negative x is
 * below every c, a NaN of positive sign above them all, so that one NaN sign is left to exclude). */
XD_HD bool xzero(double x) {
  uint32_t lo, hi;
  xwords(x, lo, hi);
  return ((hi << 1) | lo) == 0;
}
XD_HD bool xcmp_const(uint32_t ch) { return ch < 0x7ff00000u; }   /* c: not negative, finite */
XD_HD long long xsword(uint32_t lo, uint32_t hi) { return (long long)(((uint64_t)hi << 32) | lo); }
XD_HD bool xnan(uint32_t lo, uint32_t hi) { return (((uint64_t)(hi & 0x7fffffffu) << 32) | lo) > 0x7ff0000000000000ull; }
/* ordered integer key of a non-NaN double: order of the values, -0 and +0 equal */
XD_HD long long xkey(uint32_t lo, uint32_t hi) {
  const uint32_t s = (uint32_t)((int32_t)hi >> 31);
  return (long long)((((uint64_t)((hi & 0x7fffffffu) ^ s)) << 32) | (lo ^ s)) - (long long)(int32_t)s;
}
XD_HD bool xlt(double a, double b) {
  uint32_t al, ah, bl, bh;
  xwords(a, al, ah);
  xwords(b, bl, bh);
  return !(xnan(al, ah) | xnan(bl, bh)) & (xkey(al, ah) < xkey(bl, bh));
}
XD_HD bool xle(double a, double b) {
  uint32_t al, ah, bl, bh;
  xwords(a, al, ah);
  xwords(b, bl, bh);
  return !(xnan(al, ah) | xnan(bl, bh)) & (xkey(al, ah) <= xkey(bl, bh));
}
XD_HD bool xeq(double a, double b) {
  uint32_t al, ah, bl, bh;
  xwords(a, al, ah);
  xwords(b, bl, bh);
  return !(xnan(al, ah) | xnan(bl, bh)) & (xkey(al, ah) == xkey(bl, bh));
}
/* x < c, x > c, x <= c for the constants of the flux code (0, 1/2, 1, 2, eps, tolisec, tol): the
 * test of c folds away for a literal and is the same for every thread otherwise */
XD_HD bool xlt_c(double x, double c) {
  const uint64_t bc = xbits(c);
  if (!xcmp_const((uint32_t)(bc >> 32))) return xlt(x, c);
  uint32_t lo, hi;
  xwords(x, lo, hi);
  const long long sx = xsword(lo, hi);
  if (bc == 0) return (uint64_t)sx - 0x8000000000000001ull < 0x7ff0000000000000ull;
  return (sx < (long long)bc) & ((uint64_t)sx <= 0xfff0000000000000ull);
}
XD_HD bool xgt_c(double x, double c) {
  const uint64_t bc = xbits(c);
  if (!xcmp_const((uint32_t)(bc >> 32))) return xlt(c, x);
  uint32_t lo, hi;
  xwords(x, lo, hi);
  const long long sx = xsword(lo, hi);
  return (sx > (long long)bc) & (sx <= 0x7ff0000000000000ll);
}
/* x < b for a b of +0 .. +inf that is not a literal: as xlt_c, and -0 is not below +0 */
XD_HD bool xlt_nonneg(double x, double b) {
  uint32_t lo, hi, bl, bh;
  xwords(x, lo, hi);
  xwords(b, bl, bh);
  const long long sx = xsword(lo, hi), sb = xsword(bl, bh);
  return (sx < sb) & ((uint64_t)sx <= 0xfff0000000000000ull) & ((hi != 0x80000000u) | (((bl | bh | lo)) != 0));
}
XD_HD bool xle_c(double x, double c) {
  const uint64_t bc = xbits(c);
  if (!xcmp_const((uint32_t)(bc >> 32))) return xle(x, c);
  uint32_t lo, hi;
  xwords(x, lo, hi);
  const long long sx = xsword(lo, hi);
  return (sx <= (long long)bc) & ((uint64_t)sx <= 0xfff0000000000000ull);
}

template <bool MUL>
struct XD {
  double v;
  XD_HD XD() : v(0.0) {}
  XD_HD XD(double x) : v(x) {}  // NOLINT: constants promote implicitly
};

template <bool MUL>
XD_HD double val(const XD<MUL>& x) { return x.v; }

template <bool MUL>
XD_HD double xd_mul(double a, double b) {
  if (MUL) return em_mul(a, b);
  return a * b;
}
template <bool MUL>
XD_HD double xd_div(double a, double b) {
  if (MUL) return em_div(a, b);
  return a / b;
}

#define CF_XD_BIN(op, expr)                                                                               \
  template <bool MUL> XD_HD XD<MUL> operator op(const XD<MUL>& a, const XD<MUL>& b) { double x = a.v, y = b.v; return XD<MUL>(expr); } \
  template <bool MUL> XD_HD XD<MUL> operator op(const XD<MUL>& a, double y) { double x = a.v; return XD<MUL>(expr); } \
  template <bool MUL> XD_HD XD<MUL> operator op(double x, const XD<MUL>& b) { double y = b.v; return XD<MUL>(expr); }
CF_XD_BIN(+, x + y)
CF_XD_BIN(-, x - y)
CF_XD_BIN(*, xd_mul<MUL>(x, y))
CF_XD_BIN(/, xd_div<MUL>(x, y))
#undef CF_XD_BIN

/* x with its high word combined: the sign-bit operations below */
XD_HD double xhi_xor(double x, uint32_t m) {
  uint32_t lo, hi;
  xwords(x, lo, hi);
  return xjoin(lo, hi ^ m);
}
XD_HD uint32_t xhi(double x) {
  uint32_t lo, hi;
  xwords(x, lo, hi);
  return hi;
}
/* negation as a sign-bit flip: an FP64 negation that is not folded into its consumer is an FP64
 * instruction, and most consumers here are integer code (products, comparisons) */
template <bool MUL> XD_HD XD<MUL> operator-(const XD<MUL>& a) { return XD<MUL>(xhi_xor(a.v, 0x80000000u)); }

template <bool MUL> XD_HD bool operator<(const XD<MUL>& a, const XD<MUL>& b) { return xlt(a.v, b.v); }
template <bool MUL> XD_HD bool operator>(const XD<MUL>& a, const XD<MUL>& b) { return xlt(b.v, a.v); }
template <bool MUL> XD_HD bool operator<=(const XD<MUL>& a, const XD<MUL>& b) { return xle(a.v, b.v); }
template <bool MUL> XD_HD bool operator>=(const XD<MUL>& a, const XD<MUL>& b) { return xle(b.v, a.v); }
template <bool MUL> XD_HD bool operator==(const XD<MUL>& a, const XD<MUL>& b) { return xeq(a.v, b.v); }
template <bool MUL> XD_HD bool operator!=(const XD<MUL>& a, const XD<MUL>& b) { return !xeq(a.v, b.v); }
template <bool MUL> XD_HD bool operator<(const XD<MUL>& a, double c) { return xlt_c(a.v, c); }
template <bool MUL> XD_HD bool operator>(const XD<MUL>& a, double c) { return xgt_c(a.v, c); }
template <bool MUL> XD_HD bool operator<=(const XD<MUL>& a, double c) { return xle_c(a.v, c); }
template <bool MUL> XD_HD bool operator>=(const XD<MUL>& a, double c) { return xle(c, a.v); }
template <bool MUL> XD_HD bool operator==(const XD<MUL>& a, double c) { return xeq(a.v, c); }
template <bool MUL> XD_HD bool operator!=(const XD<MUL>& a, double c) {
  return xbits(c) == 0 ? !xzero(a.v) : !xeq(a.v, c);
}
template <bool MUL> XD_HD bool operator<(double c, const XD<MUL>& a) { return xgt_c(a.v, c); }
template <bool MUL> XD_HD bool operator>(double c, const XD<MUL>& a) { return xlt_c(a.v, c); }
template <bool MUL> XD_HD bool operator<=(double c, const XD<MUL>& a) { return xle(c, a.v); }
template <bool MUL> XD_HD bool operator>=(double c, const XD<MUL>& a) { return xle_c(a.v, c); }

template <bool MUL> XD_HD bool lt_nonneg(const XD<MUL>& a, const XD<MUL>& b) { return xlt_nonneg(a.v, b.v); }
template <bool MUL>
struct ConstOps<XD<MUL>> {
  static XD_HD double quot(double a, double d, double y) { return val(div_rn(XD<MUL>(a), d, y)); }
  static XD_HD double half(double x) { return val(halve(XD<MUL>(x))); }
  static XD_HD double dbl(double x) { return val(twice(XD<MUL>(x))); }
};

/* max(0, x) with dmax's results: x where 0 < x, else +0 (-0, negative and NaN x) */
template <bool MUL> XD_HD XD<MUL> dmax0(const XD<MUL>& x) { return xgt_c(x.v, 0.0) ? x : XD<MUL>(0.0); }

template <bool MUL> XD_HD XD<MUL> sqrt(const XD<MUL>& a) { return XD<MUL>(MUL ? em_sqrt(a.v) : ::sqrt(a.v)); }
struct MulInt {
  static XD_HD double mul(double a, double b) { return em_mul(a, b); }
};
XD_HD XD<false> rcbrt(const XD<false>& a) { return XD<false>(rcbrt(a.v)); }
XD_HD XD<true> rcbrt(const XD<true>& a) { return XD<true>(rcbrt_of<MulInt>(a.v)); }
template <bool MUL> XD_HD bool is_zero(const XD<MUL>& x) { return xzero(x.v); }
/* a b with a zero a on the fast path */
XD_HD XD<false> mulz(const XD<false>& a, const XD<false>& b) { return a * b; }
XD_HD XD<true> mulz(const XD<true>& a, const XD<true>& b) {
  uint32_t al, ah, bl, bh;
  xwords(a.v, al, ah);
  xwords(b.v, bl, bh);
  bool bad;
  double r = em_mul_fast(a.v, b.v, bad);
  const bool z = (((ah << 1) | al) == 0) & ((~bh & 0x7ff00000u) != 0);
  if (__builtin_expect(bad & !z, 0)) r = em_mul_rest(a.v, b.v);
  return XD<true>(z ? xjoin(0u, (ah ^ bh) & 0x80000000u) : r);
}
template <bool MUL> XD_HD XD<MUL> mirrored(const XD<MUL>& x) {
  uint32_t lo, hi;
  xwords(x.v, lo, hi);
  return XD<MUL>(xjoin(lo, ((hi << 1) | lo) == 0 ? 0u : hi ^ 0x80000000u));
}
/* 0 - x but for the sign of a zero, which the update adds to a depth */
template <bool MUL> XD_HD XD<MUL> zero_minus(const XD<MUL>& x) { return -x; }
/* a where b and c are finite (0 b and 0 c are zeros then) */
template <bool MUL> XD_HD XD<MUL> first_row(const XD<MUL>& a, const XD<MUL>& b, const XD<MUL>& c) {
  const bool fin = ((~xhi(b.v) & 0x7ff00000u) != 0) & ((~xhi(c.v) & 0x7ff00000u) != 0);
  return fin ? a : XD<MUL>(xdbl(0x7ff8000000000000ull));
}
template <bool MUL> XD_HD XD<MUL> fabs(const XD<MUL>& a) {
  uint32_t lo, hi;
  xwords(a.v, lo, hi);
  return XD<MUL>(xjoin(lo, hi & 0x7fffffffu));
}
template <bool MUL> XD_HD XD<MUL> sgnmul(const XD<MUL>& x, const XD<MUL>& y) {
  return XD<MUL>(xhi_xor(y.v, xhi(x.v) & 0x80000000u));
}

/* x * 2^K (K = -2, -1, 1) by a change of the exponent field, for a normal x whose result is
 * normal: the exact scaling, the bits of the FP64 product.  Zeros keep their bits; subnormal,
 * infinite and NaN operands and results out of the normal range take the FP64 product. */
template <int K>
XD_HD double xscale(double x) {
  uint32_t l, h;
  xwords(x, l, h);
  const uint32_t lo = (K < 0) ? (uint32_t)(1 - K) : 1u;          /* lowest exponent field handled */
  const uint32_t n = (K < 0) ? (uint32_t)(2046 + K) : (uint32_t)(2046 - K);  /* fields handled */
  const bool ok = h * 2u - (lo << 21) < (n << 21);
  if (__builtin_expect(!ok && ((h << 1) | l) != 0, 0)) return xmul_slow(x, (K == -2) ? 0.25 : ((K == -1) ? 0.5 : 2.0));
  return xjoin(l, ok ? h + ((uint32_t)K << 20) : h);
}
template <bool MUL> XD_HD XD<MUL> halve(const XD<MUL>& x) { return XD<MUL>(MUL ? xscale<-1>(x.v) : x.v * 0.5); }
template <bool MUL> XD_HD XD<MUL> quarter(const XD<MUL>& x) { return XD<MUL>(MUL ? xscale<-2>(x.v) : x.v * 0.25); }
template <bool MUL> XD_HD XD<MUL> twice(const XD<MUL>& x) { return XD<MUL>(MUL ? xscale<1>(x.v) : x.v * 2.0); }

/* RN(1/d) for the quotients of div_rn: not formed where the quotient is formed directly */
struct XNoRecip {};
XD_HD XD<false> recip(const XD<false>& d) { return XD<false>(1.0 / d.v); }
XD_HD XNoRecip recip(const XD<true>&) { return XNoRecip(); }

/* The quotient a / d that div_rn in cf_flux.h forms from y = RN(1/d) by Markstein's step: on the
 * integer path the division itself (the same bits), otherwise Markstein's step. */
template <bool MUL>
XD_HD XD<MUL> div_rn(const XD<MUL>& a, double d, double y) {
  if (MUL) return XD<MUL>(em_div_y(a.v, d, y));
  const double q = a.v * y;
  const double r = fma(-d, q, a.v);
  const double q1 = fma(r, y, q);
  return XD<MUL>(zero_u(xbits(a.v)) ? q : q1);
}
template <bool MUL>
XD_HD XD<MUL> div_rn(const XD<MUL>& a, const XD<MUL>& d, const XD<MUL>& y) {
  return div_rn(a, d.v, y.v);
}
XD_HD XD<true> div_rn(const XD<true>& a, const XD<true>& d, XNoRecip) { return XD<true>(em_div(a.v, d.v)); }

}  // namespace cf

#endif
