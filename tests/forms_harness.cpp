/*
 * forms_harness.cpp -- TEST INFRASTRUCTURE.  The whole-edge form that the reverse sweep differentiates
 * (interior_edge) against the step's two-sided one (edge_interior), on the CPU.
 */
#include "../cuteflow_gb300/csrc/cf_flux.h"

#include <cmath>

using namespace cf;

/* Over n edges with axis-parallel normals: depths of two values or dry, normal velocities at and around
 * the celerity and twice it, flat or stepped beds, one upwind element a side.  The number whose ten values
 * differ; *standing: edges with a wave speed of exactly 0. */
template <int IFLUX>
static long long forms(long long n, unsigned long long seed, long long* standing) {
  unsigned long long s = seed | 1;
  auto rnd = [&]() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; };
  auto unif = [&]() { return (double)(rnd() >> 11) * (1.0 / 9007199254740992.0); };
  auto pick = [&](double a, double b, double c, double d) {
    const unsigned k = (unsigned)(rnd() % 4);
    return k == 0 ? a : k == 1 ? b : k == 2 ? c : d;
  };
  long long bad = 0;
  *standing = 0;
  for (long long i = 0; i < n; ++i) {
    MemberDev M;
    std::memset(&M, 0, sizeof(M));
    M.gp = pick(1.0, 4.0, 9.81, 10.0);
    M.tolisec = 1e-4;
    const double nx = pick(1.0, -1.0, 0.0, 0.0), ny = nx == 0.0 ? ((rnd() & 1) ? 1.0 : -1.0) : 0.0;
    double4 U[4];
    for (double4& u : U) {
      const double h = pick(1.0, 1.0, 0.25, rnd() % 3 ? 1.0 : 0.0), c = std::sqrt(M.gp * h);
      const double un = pick(c, -c, 2.0 * c, 0.0) * (rnd() % 4 ? 1.0 : unif()), ut = pick(c, 0.0, -c, 0.3);
      u = make_double4(h, h * (un * nx - ut * ny), h * (un * ny + ut * nx), h > 0.0 ? 1.0 / h : 0.0);
    }
    const int2 ab = make_int2(0, 1);
    const double d0 = 0.5 + unif(), da = 0.5 + unif(), db = 0.5 + unif();
    const double4 geo = make_double4(nx, ny, 0.5 + unif(), d0);
    const double zl = rnd() % 3 ? 0.0 : 0.1 * unif();
    const double4 ez = make_double4(zl, 0.0, zl, 0.0);
    const int4 up = make_int4(2, 2, 3, 3);
    const double4 wt = make_double4(-1.0, 0.0, -1.0, 0.0);
    const double4 dk = make_double4(da, db, 1.0 / da, 1.0 / db), inv = make_double4(1.0 / d0, 0.5 / da, 0.5 / db, 0.0);
    Slot got[2];
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
    a.slots = got;
    a.ilimiteur = (int)(rnd() % 5);
    a.flux_mode = (int)(rnd() % 2);
    const double dt = 0.01 + 0.1 * unif();
    edge_interior<IFLUX>(a, M, 0, dt);
    const EdgeGeo G = edge_geo(a, 0, IFLUX >= 3);
    double hl = 0.0, vl = 0.0, hr = 0.0, vr = 0.0, o[10];
    if (IFLUX == 3) {
      upwind_state(U, up.x, up.y, wt.x, wt.y, 1.0, G.ysum_a, nx, ny, M.tolisec, hl, vl);
      upwind_state(U, up.z, up.w, wt.z, wt.w, 1.0, G.ysum_b, nx, ny, M.tolisec, hr, vr);
    }
    interior_edge<IFLUX>(M, a.ilimiteur, a.flux_mode, G, dt, U[0].x, U[0].y, U[0].z, ez.x, U[0].w, U[1].x, U[1].y, U[1].z,
                         ez.y, U[1].w, hl, vl, ez.z, hr, vr, ez.w, o);
    const double g[10] = {got[0].f1, got[0].f2, got[0].f3, got[0].bx, got[0].by, got[1].f1, got[1].f2, got[1].f3,
                          got[1].bx, got[1].by};
    bool ok = true;
    for (int k = 0; k < 10; ++k) ok = ok && g[k] == o[k];
    bad += !ok;
    double h0, u0, v0, h1, u1, v1, sl, sr, set;
    to_frame(U[0].x, U[0].y, U[0].z, U[0].w, nx, ny, M.tolisec, h0, u0, v0);
    to_frame(U[1].x, U[1].y, U[1].z, U[1].w, nx, ny, M.tolisec, h1, u1, v1);
    if (zl == 0.0 && wave_speeds(M.gp, EPS_SECOND, h0, u0, h1, u1, sl, sr, set))
      *standing += sl == 0.0 || sr == 0.0 || set == 0.0;
  }
  return bad;
}

extern "C" long long harness_forms(int iflux, long long n, unsigned long long seed, long long* standing) {
  return iflux == 1 ? forms<1>(n, seed, standing) : iflux == 2 ? forms<2>(n, seed, standing) : forms<3>(n, seed, standing);
}
