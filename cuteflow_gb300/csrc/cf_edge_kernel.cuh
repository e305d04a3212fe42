/*
 * cf_edge_kernel.cuh -- the edge kernel of the step (included by one small translation unit per
 * scheme, cf_edges_<IFLUX>.cu, so that the launch shapes of the four schemes compile in parallel).
 *
 * k_edges<IFLUX, BE, EPT>: blocks of BE threads, two neighbouring lanes per edge, one for each of its
 * sides (EdgeSide in cf_flux.h: what the sides share goes through shuffles), each lane evaluating EPT
 * sides (i, i + BE, ... of its block's BE * EPT consecutive ones).  Edges keep their layout of tiles of
 * TILE_E = 128 edges, each owned by one member, whatever the shape: a lane looks up its edge's member,
 * and the integer-pipe warp mask bit w applies to the edges (e mod 128) / 32 = w of a tile (of a list: by
 * their position in it).  Every
 * shape evaluates the same edges with the same arithmetic, so results do not depend on it (the
 * autotuner chooses one; cf_ctx.h has the one a context starts with).
 *
 * What bounds it: a wet WAF side is ~4,000 instructions of which 55 are FP64 ones (76 cycles each on
 * their pipe): issue slots 58 %, FP64 pipe 65 %, the two integer pipes 56 and 41 % busy, waits on
 * fixed latencies and on instruction fetch between them (WAF 201k triangles, fully wet: 185 us
 * per step with one thread per edge for both sides, 153 with two lanes, 149 with the limiter's shared
 * branches and overlapping launches, 150 with the signs of zero wave speeds kept).
 *
 * Register budget: every IFLUX 1-3 shape keeps 1024 threads per SM (at most 64 registers); 768, 1280
 * and 1536 threads measured the same within 3 % or slower (WAF 201k: 168 us per step at 1024; 172, 175,
 * 181).  MUSCL-Hancock keeps 512 threads per SM (128 registers); 640 and 768 measured the same.
 */
#ifndef CF_EDGE_KERNEL_CUH
#define CF_EDGE_KERNEL_CUH

#include <cuda_runtime.h>

#include "cf_flux.h"
#include "cf_launch.cuh"
#include "cf_xd.h"

namespace cf {
namespace {

/* Start of member M's step (by the thread of its first edge, or by k_begin_step): the dt sanity
 * test of cfl_condition.cuf:129-132 (a failing dt ends the run with the current state), the next
 * time, and the start value of the next dt minimum (cflcond sets dt_d = 1e6 and the block
 * reduction pads a partial last block with 1e5, cfl_condition.cuf:21,86). */
__device__ __forceinline__ void step_start(const MemberDev& M, MemberState* S, int p) {
  const double dt = S->dt[p];
  const double t = S->t[p];
  if (S->nstep > 0 && (dt > 9999.0 || dt < DT_LOW)) {   /* the initial dt is not tested (:113-116) */
    atomicOr(&S->status, CF_STATUS_DT_RANGE);
  } else if (S->nstep > 0 && !((S->tc + dt) - S->ts + 2.0 * TOL_LOOP < TOL_LOOP)) {
    /* the time loop's test (finite_volumes_method.cuf:123) on tc = tc + dt (:232); tc keeps
     * its value, so that a later cf_run adds this dt once and tests again */
    atomicOr(&S->status, CF_STATUS_END);
  } else if (S->nstep == 0 && !(S->tc - S->ts + 2.0 * TOL_LOOP < TOL_LOOP)) {
    atomicOr(&S->status, CF_STATUS_END);
  } else {
    if (S->nstep > 0) S->tc = S->tc + dt;
    S->t[1 - p] = t + dt;
    S->dt[1 - p] = M.dt_reset;
    S->nstep += 1;
  }
}

/* The gauge elevations of a state, by one block */
__device__ __forceinline__ void record_gauges(const StepRec& r, const double4* U) {
  pdl_begin();
  for (int g = threadIdx.x; g < r.ng; g += blockDim.x) {
    const int c = __ldg(r.gcell + g);
    r.eta[g] = U[c].x + __ldg(r.zcell + c);
  }
}

/* One side of an edge on this lane, the other one on the neighbouring lane (lane ^ 1); mask holds the
 * lanes whose edges are being evaluated. */
template <int IFLUX, class T_>
struct LanePair {
  using T = T_;
  using Side = EdgeSide<IFLUX, T>;
  Side s;
  T out[5];
  unsigned mask;
  template <class F>
  __device__ __forceinline__ void each(F&& f) { f(s, out); }
  __device__ __forceinline__ void exchange(int n) {
#pragma unroll
    for (int k = 0; k < 6; ++k)
      if (k < n) s.y[k] = T(__shfl_xor_sync(mask, val(s.x[k]), 1));
  }
};

/* This lane's side of the interior edge e (element state U), by every lane of mask at once */
template <int IFLUX, class T>
__device__ __forceinline__ void edge_side(const StepArgs& a, const MemberDev& M, unsigned mask, int e, int side,
                                          const double4& geo, const double4& U, double dt) {
  LanePair<IFLUX, T> p;
  p.mask = mask;
  side_load(a, M, e, side, geo, U, dt, p.s);
  double4 dk = make_double4(0.0, 0.0, 0.0, 0.0);
  if (IFLUX == 4) dk = ld4(a.edk + e);
  side_stages<IFLUX>(p, a.ilimiteur, dk.x, dk.z, dk.y, dk.w);
  if (a.flux_mode == 1) {   /* side B: side A's flux, negated */
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const T f = T(__shfl_xor_sync(mask, val(p.out[k]), 1));
      if (side) p.out[k] = -f;
    }
  }
  store_side(a.slots + 2 * (size_t)e + side, p.out, geo.z);
}

/* What every path of an edge reads of the mesh's tables: loaded before the kernel waits for the one
 * before it. */
struct EdgeHead {
  int2 ab;
  double4 geo;
  __device__ __forceinline__ void load(const StepArgs& a, int e, bool live) {
    ab = make_int2(0, -3);
    geo = make_double4(0.0, 0.0, 0.0, 0.0);
    if (live) {
      ab = ldro(a.ecell + e);
      const double2* q = reinterpret_cast<const double2*>(a.egeo + e);
      const double2 u = ldro(q), v = ldro(q + 1);
      geo = make_double4(u.x, u.y, v.x, v.y);
    }
  }
};

/* Edge e of a step, at position pos of the kernel's order, on the lanes of its two sides, in the
 * context's arithmetic type.  Every lane of the warp comes here; live: the lane's edge is one to evaluate.
 * The shuffles name every lane whose edge is evaluated, so the 16 edges of a warp have to be of one member
 * and of one arithmetic type: int_products goes by the position, which a warp's edges share up to the last
 * four bits, and not by the edge's number (those of a list are of any tile). */
template <int IFLUX>
__device__ __forceinline__ void edge_lanes(const StepArgs& a, const MemberDev& M, const EdgeHead& E, int e, int pos,
                                           int side, bool live, double dt, double t, const double* surf) {
  const int2 ab = E.ab;
  const double4 geo = E.geo;
  double4 U = make_double4(0.0, 0.0, 0.0, 0.0);
  if (live) U = ld4(a.Uin + ((side && ab.y >= 0) ? ab.y : ab.x));   /* {h, hu, hv, RN(1/h)} */
  const double hp = __shfl_xor_sync(0xffffffffu, U.x, 1);
  bool run = live && ab.y >= 0;
  if (run && (dbits_hd(U.x) | dbits_hd(hp)) == 0 && dry_edge_ok<IFLUX>(M.gp, geo, dt)) {
    /* an edge between two dry elements (most of a flood plain that the water has not reached) needs
     * neither its beds nor its upwind states */
    dry_slot<IFLUX>(M.gp, a.flux_mode, geo, side, a.slots + 2 * (size_t)e + side);
    run = false;
  }
  const unsigned mask = __ballot_sync(0xffffffffu, run);
  if (run) {
    if (a.xd_cmp) {
      /* the same arithmetic with exact integer comparisons and, in the warps of xd_mul_mask, exact
       * integer products, quotients and roots: the FP64 pipe and the integer pipes share the work */
      if (int_products(a.xd_mul_mask, pos)) edge_side<IFLUX, XD<true>>(a, M, mask, e, side, geo, U, dt);
      else edge_side<IFLUX, XD<false>>(a, M, mask, e, side, geo, U, dt);
    } else {
      edge_side<IFLUX, double>(a, M, mask, e, side, geo, U, dt);
    }
  } else if (live && ab.y < 0 && side == 0) {
    boundary_slot<IFLUX>(a, M, e, ab, geo, U, t, surf);
  }
}

template <int IFLUX, int BE, int EPT, bool REC>
__device__ __forceinline__ void edges_block(const StepArgs& a, const StepRec* r) {
  const int p = a.parity;
  const int nside = 2 * a.n_etiles * TILE_E;
#pragma unroll 1
  for (int j = 0; j < EPT; ++j) {
    const int i = (blockIdx.x * EPT + j) * BE + threadIdx.x;
    if (i >= nside) return;
    const int e = i >> 1;
    const int m = __ldg(a.etile_mem + e / TILE_E);
    const MemberDev& M = a.mdev[m];
    MemberState* S = a.mst + m;
    EdgeHead E;
    E.load(a, e, e < M.edge_end);
    if (j == 0) pdl_begin();
    /* one answer for the warp, whose lanes shuffle below: the member's first lane, in another warp, may be
     * setting the status, and an earlier side may have split this one */
    if (__any_sync(0xffffffffu, S->status != 0)) continue;
    const double dt = S->dt[p];
    const double t = S->t[p];
    if (i == 2 * M.edge_begin) {
      if (REC) {
        r->dt[m] = dt;
        r->t[m] = t;
      }
      step_start(M, S, p);
    }
    edge_lanes<IFLUX>(a, M, E, e, e, i & 1, e < M.edge_end, dt, t, S->surf);
  }
}

template <int IFLUX, int BE, int EPT>
__global__ void __launch_bounds__(BE, ((IFLUX == 4) ? 512 : 1024) / BE) k_edges(StepArgs a) {
  edges_block<IFLUX, BE, EPT, false>(a, nullptr);
}

/* The adjoint's forward: a step that also records what the reverse sweep and the objective need of it,
 * the gauges by one block more.  (By a kernel after every step: ~2 us a step; gradient over 51k triangles
 * 4.08 -> 4.00 ms, batched descent iteration 2.74 -> 2.69 ms.) */
template <int IFLUX, int BE, int EPT>
__global__ void __launch_bounds__(BE, 1024 / BE) k_edges_rec(StepArgs a, StepRec r) {
  if (r.eta && blockIdx.x == gridDim.x - 1) return record_gauges(r, a.Uin);
  edges_block<IFLUX, BE, EPT, true>(a, &r);
}

/* The edges of a list (a part's phase of its step; a part is a context of one member): TILE_E lanes per
 * block; the step's start is made by k_begin_step before the first phase. */
template <int IFLUX>
__global__ void __launch_bounds__(TILE_E, (IFLUX == 4) ? 4 : 8) k_edges_list(StepArgs a, const int32_t* list, int n) {
  const int i = (blockIdx.x * TILE_E + threadIdx.x) >> 1;
  const MemberDev& M = a.mdev[0];
  MemberState* S = a.mst;
  if (__any_sync(0xffffffffu, S->status != 0)) return;
  const int e = i < n ? list[i] : 0;
  EdgeHead E;
  E.load(a, e, i < n && e < M.edge_end);
  edge_lanes<IFLUX>(a, M, E, e, i, threadIdx.x & 1, i < n && e < M.edge_end, S->dt[a.parity], S->t[a.parity], S->surf);
}

template <int IFLUX, int BE, int EPT>
int launch_edges_shape(const StepArgs& a, cudaStream_t st, const StepRec* rec) {
  const int nside = 2 * a.n_etiles * TILE_E;
  const int nb = (nside + BE * EPT - 1) / (BE * EPT);
  if (!rec) {
    launch_pdl(k_edges<IFLUX, BE, EPT>, nb, BE, st, a);
  } else {
    if constexpr (IFLUX <= 3) launch_pdl(k_edges_rec<IFLUX, BE, EPT>, nb + (rec->eta ? 1 : 0), BE, st, a, *rec);
    else return CF_ENOTSUP;
  }
  return cudaGetLastError() == cudaSuccess ? CF_OK : CF_ECUDA;
}

}  // namespace

template <int IFLUX>
int launch_edges_list_iflux(const StepArgs& a, const int32_t* list, int32_t n, cudaStream_t st) {
  if (n <= 0) return CF_OK;
  k_edges_list<IFLUX><<<(2 * n + TILE_E - 1) / TILE_E, TILE_E, 0, st>>>(a, list, n);
  return cudaGetLastError() == cudaSuccess ? CF_OK : CF_ECUDA;
}

/* The shapes a context can choose (cf_set_launch_shape): BE in {64, 128, 256}, EPT in {1, 2}. */
template <int IFLUX>
int launch_edges_iflux(const StepArgs& a, cudaStream_t st, const StepRec* rec) {
  const int key = a.eblock * 10 + a.ept;
  switch (key) {
    case 641: return launch_edges_shape<IFLUX, 64, 1>(a, st, rec);
    case 642: return launch_edges_shape<IFLUX, 64, 2>(a, st, rec);
    case 1281: return launch_edges_shape<IFLUX, 128, 1>(a, st, rec);
    case 1282: return launch_edges_shape<IFLUX, 128, 2>(a, st, rec);
    case 2561: return launch_edges_shape<IFLUX, 256, 1>(a, st, rec);
    case 2562: return launch_edges_shape<IFLUX, 256, 2>(a, st, rec);
    default: return CF_EINVAL;
  }
}

}  // namespace cf

#endif
