/*
 * cf_cell_kernel.cuh -- the element update on one thread or two lanes, for the element kernel of the
 * step (cf_kernels.cu) and its replay (cf_adjoint.cu).
 *
 * An element's update is a chain of dependent quotients, products and roots.  One thread takes ~2,900
 * instructions for it, which is the least work; two neighbouring lanes, one for each component of the
 * momentum (ElemSide in cf_flux.h), take ~2,260 each, with the depth's part on both.  So small meshes,
 * whose elements leave the GPU partly idle, go by two lanes and large ones by one thread (two_lanes: the
 * line is at 38,912 elements on 152 SMs): us per step by two lanes / by one, when the line was drawn: 1.4k triangles 21.6 / 24.0, 6k 27.8 / 30.3, 25k 33.3 /
 * 34.7, 51k (gradient) 96.8 / 96.6, dam break 80k 49.8 / 44.7, 134k 70.6 / 64.1, WAF 1M 274 / 248.
 */
#ifndef CF_CELL_KERNEL_CUH
#define CF_CELL_KERNEL_CUH

#include <cuda_runtime.h>

#include "cf_flux.h"
#include "cf_xd.h"

namespace cf {
namespace {

__device__ __forceinline__ Slot load_slot(const Slot* p) {
  const double2* q = reinterpret_cast<const double2*>(p);
  const double2 a = q[0], b = q[1], c = q[2];
  Slot s;
  s.f1 = a.x; s.f2 = a.y; s.f3 = b.x; s.bx = b.y; s.by = c.x; s.q = c.y;
  return s;
}
/* an element's sums for the adjoint's record (the sums element_update forms: same expressions) */
__device__ __forceinline__ void store_sums(Slot* p, const Slot& s0, const Slot& s1, const Slot& s2) {
  store_slot(p, s0.f1 + s1.f1 + s2.f1, s0.f2 + s1.f2 + s2.f2, s0.f3 + s1.f3 + s2.f3, s0.bx + s1.bx + s2.bx,
             s0.by + s1.by + s2.by, 0.0);
}
__device__ __forceinline__ double4 cell_thread(const StepArgs& a, const MemberDev& M, const double4& U, const double4& st,
                                               const Slot& s0, const Slot& s1, const Slot& s2, double dt,
                                               bool& nonfinite) {
  /* bit 4 of xd_mul_mask: the element's arithmetic on the integer pipes (cf_xd.h) */
  if (a.xd_cmp && (a.xd_mul_mask & XD_CELLS)) return element_update<XD<true>>(M, U, st, s0, s1, s2, dt, nonfinite);
  return element_update(M, U, st, s0, s1, s2, dt, nonfinite);
}

/* The parts of an element's three slots (sl) that component comp needs, each summed in the reference's
 * edge order; zero: every one of them is +-0. */
struct CompSums {
  double rc1, rcq, sb;
  bool zero;
};
__device__ __forceinline__ CompSums comp_sums(const Slot* slots, const int4& sl, int comp) {
  const double* p[3] = {&slots[sl.x].f1, &slots[sl.y].f1, &slots[sl.z].f1};
  double f[3], q[3], b[3];
  uint64_t z = 0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    f[k] = p[k][0];
    q[k] = p[k][1 + comp];
    b[k] = p[k][3 + comp];
    z |= dbits_hd(f[k]) | dbits_hd(q[k]) | dbits_hd(b[k]);
  }
  CompSums s;
  s.zero = zero_u(z);
  s.rc1 = f[0] + f[1] + f[2];
  s.rcq = q[0] + q[1] + q[2];
  s.sb = b[0] + b[1] + b[2];
  return s;
}

__device__ __forceinline__ void store_comp_sums(Slot* p, const CompSums& s, int comp) {
  double* q = &p->f1;   /* the layout of a slot: f1 f2 | f3 bx | by 0 */
  if (comp == 0) {
    *reinterpret_cast<double2*>(q) = make_double2(s.rc1, s.rcq);
    q[3] = s.sb;
  } else {
    q[2] = s.rcq;
    *reinterpret_cast<double2*>(q + 4) = make_double2(s.sb, 0.0);
  }
}

/* The new state of an element, on both its lanes; mask: the lanes at work */
template <class T>
__device__ __forceinline__ double4 elem_lanes(const MemberDev& M, int comp, const double4& U, const double4& st,
                                              const CompSums& s, double dt, unsigned mask, bool& nonfinite) {
  ElemSide<T> e;
  auto exchange = [&](int n) {
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (k < n) e.y[k] = T(__shfl_xor_sync(mask, val(e.x[k]), 1));
  };
  e.velocity(M, comp, U, s.rc1, s.rcq, s.sb);
  exchange(2);
  e.friction(M, U, st, dt);
  exchange(3);
  nonfinite = !e.update(M, dt);
  const double h = val(e.h), q = val(e.qn), o = __shfl_xor_sync(mask, q, 1);
  /* the new state carries RN(1/h) for the next step's quotients by h */
  return make_double4(h, comp ? o : q, comp ? q : o, h > 0.0 ? val(T(1.0) / e.h) : 0.0);
}

/* The update of one element by its two lanes from its slots, or its dry shortcut; every lane of the
 * warp comes here (run: the lane's element is to be updated from its slots). */
__device__ __forceinline__ double4 cell_lanes(const StepArgs& a, const MemberDev& M, int comp, bool run, const double4& U,
                                              const double4& st, const CompSums& s, double dt, bool& nonfinite) {
  double4 V = make_double4(0.0, 0.0, 0.0, 0.0);
  nonfinite = false;
  const int zero = __shfl_xor_sync(0xffffffffu, (int)s.zero, 1) & (int)s.zero;
  if (run && zero && dry_element_state(M, U, st, dt)) run = false;   /* no water reaches it this step (dry_element) */
  const unsigned mask = __ballot_sync(0xffffffffu, run);
  if (run) {
    if (a.xd_cmp && (a.xd_mul_mask & XD_CELLS)) V = elem_lanes<XD<true>>(M, comp, U, st, s, dt, mask, nonfinite);
    else V = elem_lanes<double>(M, comp, U, st, s, dt, mask, nonfinite);
  }
  return V;
}

}  // namespace
}  // namespace cf

#endif
