/*
 * dry_harness.cpp -- TEST INFRASTRUCTURE.  The dry-edge shortcut of the step (dry_edge_slots) against the
 * two-sided evaluation that it skips (edge_interior, the stages of the edge kernel), on the CPU.
 */
#include "../cuteflow_gb300/csrc/cf_flux.h"
#include "../cuteflow_gb300/csrc/cf_xd.h"

#include <cmath>

using namespace cf;

/* Over n edges between two elements of depth +0: random beds (signed zeros, ties, infinities, NaN), upwind
 * states (wet ones too, one or two of them), signs of g, nx, ny and len (zeros included), every scheme,
 * limiter, flux mode and arithmetic type.  The number of edges whose two slots differ in a bit; *taken: the
 * edges that the shortcut takes. */
extern "C" long long harness_dry_edges(long long n, unsigned long long seed, int iflux, long long* taken) {
  unsigned long long s = seed | 1;
  auto rnd = [&]() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; };
  auto unif = [&]() { return (double)(rnd() >> 11) * (1.0 / 9007199254740992.0); };
  auto sgn = [&](double x) { return (rnd() & 1) ? -x : x; };
  auto special = [&](double x) {
    const unsigned k = (unsigned)(rnd() % 16);
    return k == 0 ? 0.0 : k == 1 ? -0.0 : k == 2 ? (double)INFINITY : k == 3 ? -(double)INFINITY : k == 4 ? (double)NAN : x;
  };
  long long bad = 0, took = 0;
  for (long long i = 0; i < n; ++i) {
    MemberDev M;
    std::memset(&M, 0, sizeof(M));
    M.gp = (rnd() % 8 == 0) ? special(sgn(9.81)) : sgn(0.5 + 20.0 * unif());
    M.tolisec = (rnd() % 4 == 0) ? 0.0 : 1e-4 * unif();
    /* elements 0, 1: the edge's, dry, with any discharges; 2, 3 upwind of the first, 4, 5 of the second */
    double4 U[6];
    for (int k = 0; k < 6; ++k) {
      const double h = (k >= 2 && (rnd() & 1)) ? 2.0 * unif() : 0.0;
      U[k] = make_double4(h, sgn(unif()), sgn(unif()), h > 0.0 ? 1.0 / h : 0.0);
    }
    const int2 ab = make_int2(0, 1);
    const double d0 = 0.1 + unif();
    const double4 geo = make_double4((rnd() % 6 == 0) ? sgn(0.0) : (rnd() % 20 == 0 ? special(1.0) : sgn(unif())),
                                     (rnd() % 6 == 0) ? sgn(0.0) : (rnd() % 20 == 0 ? special(1.0) : sgn(unif())),
                                     (rnd() % 8 == 0) ? special(0.3) : 0.01 + 5.0 * unif(), d0);
    const double zl = (rnd() % 3 == 0) ? special(3.0 * unif()) : 3.0 * unif();
    const double zr = (rnd() % 3 == 0) ? zl : ((rnd() % 3 == 0) ? special(3.0 * unif()) : 3.0 * unif());
    const double4 ez = make_double4(zl, zr, 3.0 * unif(), 3.0 * unif());
    const int4 up = make_int4(2, 3, 4, 5);
    const double4 wt = make_double4((rnd() & 1) ? -1.0 : 0.1 + unif(), 0.1 + unif(), (rnd() & 1) ? -1.0 : 0.1 + unif(),
                                    0.1 + unif());
    auto dist = [&](double d1, double d2) { return d1 < 0.0 ? 0.1 + unif() : (d1 + d2) / 2.0; };
    const double da = dist(wt.x, wt.y), db = dist(wt.z, wt.w);
    const double4 dk = make_double4(da, db, 1.0 / da, 1.0 / db);
    const double4 inv = make_double4(1.0 / d0, 0.5 / da, 0.5 / db, 0.0);
    Slot want[2], got[2];
    std::memset(want, 0, sizeof(want));
    std::memset(got, 0, sizeof(got));
    StepArgs a;
    std::memset(&a, 0, sizeof(a));
    a.Uin = U;
    a.ecell = &ab;
    a.egeo = &geo;
    a.ez = &ez;
    a.eupw = &up;
    a.ewts = &wt;
    a.edk = &dk;
    a.einv = &inv;
    a.slots = want;
    a.ilimiteur = (int)(rnd() % 5);
    a.flux_mode = (int)(rnd() % 2);
    const double dt = 1e-3 + unif();
    const int xd = (int)(rnd() % 3);
    auto both = [&](auto flux) {
      constexpr int F = decltype(flux)::value;
      if (xd == 0) edge_interior<F>(a, M, 0, dt);
      else if (xd == 1) edge_interior<F, XD<false>>(a, M, 0, dt);
      else edge_interior<F, XD<true>>(a, M, 0, dt);
      return dry_edge_slots<F>(M.gp, a.flux_mode, geo, got, dt);
    };
    const bool t = iflux == 1   ? both(std::integral_constant<int, 1>())
                   : iflux == 2 ? both(std::integral_constant<int, 2>())
                   : iflux == 3 ? both(std::integral_constant<int, 3>())
                                : both(std::integral_constant<int, 4>());
    took += t;
    bad += t && std::memcmp(want, got, sizeof(want)) != 0;
  }
  *taken = took;
  return bad;
}
