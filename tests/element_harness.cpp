/*
 * element_harness.cpp -- TEST INFRASTRUCTURE.  The transposed element stage of the reverse sweep
 * (adj_element in cf_dual.h) against the element stage differentiated in nine Dual lanes, on the CPU.
 */
#include "../cuteflow_gb300/csrc/cf_dual.h"

#include <cmath>

using namespace cf;

/* The largest difference relative to the element's largest contribution, over n random elements of one
 * friction option: depths around the dry threshold and up, velocities at rest, around the floor tol and
 * up, clamped and free updates, a zero Manning n. */
extern "C" double harness_adj_element(long long n, unsigned long long seed, int friction, int fricimplic) {
  unsigned long long s = seed | 1;
  auto rnd = [&]() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; };
  auto unif = [&]() { return (double)(rnd() >> 11) * (1.0 / 9007199254740992.0); };
  auto sym = [&]() { return 2.0 * unif() - 1.0; };
  typedef Dual<9> D;
  double worst = 0.0;
  for (long long i = 0; i < n; ++i) {
    MemberDev M;
    std::memset(&M, 0, sizeof(M));
    M.gp = 9.81; M.tolisec = 1e-4; M.tol = (double)1e-6f; M.friction = friction; M.fricimplic = fricimplic;
    const double h = rnd() % 5 == 0 ? 2e-4 * unif() : 0.01 + 3.0 * unif();
    const double vel = rnd() % 4 == 0 ? 0.0 : (rnd() % 4 == 0 ? 3e-6 : 2.0);
    const double4 U = make_double4(h, h * vel * sym(), h * vel * sym(), h > 0.0 ? 1.0 / h : 0.0);
    const double area = 0.5 + 3.0 * unif();
    const double4 st = make_double4(area, rnd() % 16 == 0 ? 0.0 : 0.01 + 0.05 * unif(), 0.0, 1.0 / area);
    Slot q;
    q.f1 = sym() * (rnd() % 3 == 0 ? 10.0 : 0.5); q.f2 = sym(); q.f3 = sym(); q.bx = sym(); q.by = sym(); q.q = 0.0;
    const double4 L = make_double4(sym(), sym(), sym(), 0.0);
    const double dt = 0.2 * unif();
    double4 own;
    Slot w;
    double nb;
    adj_element(M, U, st, q, L, dt, own, w, nb);
    D H, HU, HV;
    bool nf;
    element_core(M, area, st.w, D::var(st.y, 8), D::var(U.x, 0), D::var(U.y, 1), D::var(U.z, 2), D::var(q.f1, 3),
                 D::var(q.f2, 4), D::var(q.f3, 5), D::var(q.bx, 6), D::var(q.by, 7), dt, H, HU, HV, nf, U.w);
    const double got[9] = {own.x, own.y, own.z, w.f1, w.f2, w.f3, w.bx, w.by, nb};
    double err = 0.0, top = 1e-30;
    for (int k = 0; k < 9; ++k) {
      const double want = L.x * H.d[k] + L.y * HU.d[k] + L.z * HV.d[k];
      err = std::fmax(err, std::fabs(got[k] - want));
      top = std::fmax(top, std::fabs(want));
      if (!(got[k] == got[k])) return INFINITY;
    }
    worst = std::fmax(worst, err / top);
  }
  return worst;
}

/* adj_edge_hllc against the edge differentiated in six Dual lanes, on edges with a side at the dry
 * threshold (masked, with a raw depth that reconstructs to the threshold).  Relative to the largest sum
 * of the magnitudes of a component's terms: a component itself may cancel to any degree (a bed source
 * along the edge). */
extern "C" double harness_adj_nearly_dry(long long n, unsigned long long seed) {
  unsigned long long s = seed | 1;
  auto rnd = [&]() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; };
  auto unif = [&]() { return (double)(rnd() >> 11) * (1.0 / 9007199254740992.0); };
  auto sym = [&]() { return 2.0 * unif() - 1.0; };
  typedef Dual<6> D;
  double worst = 0.0;
  for (long long i = 0; i < n; ++i) {
    MemberDev M;
    std::memset(&M, 0, sizeof(M));
    M.gp = 9.81; M.tolisec = 1e-3;
    const double phi = 6.283 * unif();
    EdgeGeo G = EdgeGeo();
    G.nx = std::cos(phi); G.ny = std::sin(phi); G.len = 0.5 + unif();
    const double zl = rnd() & 1 ? 0.0 : 0.1 * unif(), zr = rnd() % 3 ? zl : 0.1 * unif();
    auto depth = [&](int k) { return k == 0 ? M.tolisec : (k == 1 ? 0.5 * M.tolisec : 0.002 + 2.0 * unif()); };
    const int k = (int)(rnd() % 2);
    double hl = depth(k ? 0 : (int)(rnd() % 3)), hr = depth(k ? (int)(rnd() % 3) : 0);
    const double4 UA = make_double4(hl, hl * sym(), hl * sym(), 1.0 / hl), UB = make_double4(hr, hr * sym(), hr * sym(), 1.0 / hr);
    double w[10], la[3], lb[3];
    for (double& x : w) x = sym();
    if (!adj_edge_hllc(M, G, UA, UB, zl, zr, w, la, lb)) return INFINITY;
    D o[10];
    interior_edge<1>(M, 1, 0, G, 0.01, D::var(UA.x, 0), D::var(UA.y, 1), D::var(UA.z, 2), zl, UA.w, D::var(UB.x, 3),
                     D::var(UB.y, 4), D::var(UB.z, 5), zr, UB.w, D(0.0), D(0.0), 0.0, D(0.0), D(0.0), 0.0, o);
    double err = 0.0, top = 1e-30;
    for (int j = 0; j < 6; ++j) {
      double want = 0.0, terms = 0.0;
      for (int q = 0; q < 10; ++q) {
        want += w[q] * o[q].d[j];
        terms += std::fabs(w[q] * o[q].d[j]);
      }
      const double got = j < 3 ? la[j] : lb[j - 3];
      if (!(got == got)) return INFINITY;
      err = std::fmax(err, std::fabs(got - want));
      top = std::fmax(top, terms);
    }
    worst = std::fmax(worst, err / top);
  }
  return worst;
}

/* element_update_pair (the two lanes of the element kernel) against element_update_full on n random
 * elements of every friction option and arithmetic type; the number of different results (zeros of
 * either sign are equal). */
extern "C" long long harness_element_pair(long long n, unsigned long long seed) {
  unsigned long long s = seed | 1;
  auto rnd = [&]() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; };
  auto unif = [&]() { return (double)(rnd() >> 11) * (1.0 / 9007199254740992.0); };
  auto sym = [&]() { return rnd() % 12 == 0 ? 0.0 : 2.0 * unif() - 1.0; };
  auto same = [](double a, double b) { return a == b || (a != a && b != b); };
  long long bad = 0;
  for (long long i = 0; i < n; ++i) {
    MemberDev M;
    std::memset(&M, 0, sizeof(M));
    M.gp = 9.81; M.tolisec = rnd() % 4 ? 1e-4 : 0.0; M.tol = (double)1e-6f;
    M.friction = (int)(rnd() % 4 != 0); M.fricimplic = (int)(rnd() % 3);
    const double h = rnd() % 5 == 0 ? (rnd() % 2 ? 2e-4 * unif() : 0.0) : 0.01 + 3.0 * unif();
    const double vel = rnd() % 4 == 0 ? 0.0 : (rnd() % 4 == 0 ? 3e-6 : 2.0);
    const double4 U = make_double4(h, h * vel * sym(), h * vel * sym(), h > 0.0 ? 1.0 / h : 0.0);
    const double area = 0.5 + 3.0 * unif();
    const double4 st = make_double4(area, rnd() % 16 == 0 ? 0.0 : 0.01 + 0.05 * unif(), 0.0, 1.0 / area);
    Slot c[3];
    for (int k = 0; k < 3; ++k) {
      double* f = &c[k].f1;
      for (int j = 0; j < 6; ++j) f[j] = sym();
      if (rnd() % 50 == 0) f[rnd() % 5] = rnd() % 2 ? INFINITY : NAN;
    }
    const double dt = 0.3 * unif();
    const int xd = (int)(rnd() % 3);
    bool n0 = false, n1 = false;
    double4 a, b;
    if (xd == 0) {
      a = element_update_full<double>(M, U, st, c[0], c[1], c[2], dt, n0);
      b = element_update_pair<double>(M, U, st, c[0], c[1], c[2], dt, n1);
    } else if (xd == 1) {
      a = element_update_full<XD<false>>(M, U, st, c[0], c[1], c[2], dt, n0);
      b = element_update_pair<XD<false>>(M, U, st, c[0], c[1], c[2], dt, n1);
    } else {
      a = element_update_full<XD<true>>(M, U, st, c[0], c[1], c[2], dt, n0);
      b = element_update_pair<XD<true>>(M, U, st, c[0], c[1], c[2], dt, n1);
    }
    if (!(n0 == n1 && same(a.x, b.x) && same(a.y, b.y) && same(a.z, b.z) && same(a.w, b.w))) ++bad;
  }
  return bad;
}
