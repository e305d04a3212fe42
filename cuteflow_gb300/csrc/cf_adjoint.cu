/*
 * cf_adjoint.cu -- sm_103a kernels of the discrete adjoint of the step (dt of every step frozen).
 *
 * The step maps U^n to U^{n+1} in two stages: every edge computes the slot values of its two
 * sides (flux * len and bed source) from the states of its elements (and, second order, of
 * their upwind elements); every element then combines its state, the sums of its three slots
 * and its Manning n.  The adjoint runs the stages backwards:
 *
 *   k_adj_cells  : per element, lambda^{n+1} gathered (its own part of the previous reverse
 *                  step, the contributions of its three edge slots and of the edges it is
 *                  an upwind element of, the objective's weights on its gauges; fixed order,
 *                  no atomics), then the transposed local Jacobian of the element stage
 *                  applied to it: its own part of lambda^n, the adjoint of its flux and bed
 *                  sums (cadj) and dJ/dn += .. ,
 *   k_adj_edges  : per edge, the transposed Jacobian of the edge stage applied to the cadj of
 *                  its two elements: one contribution per side (and per upwind element).
 * The flux and bed sums at U^n come from the replay of the checkpoint segment (k_rep_cells
 * stores them), so a reverse step recomputes no edge fluxes.
 *
 * The local Jacobians come from the step's own arithmetic (cf_flux.h) instantiated on
 * Dual<D> numbers, whose value lane repeats the forward's IEEE operations, so every branch
 * (wet/dry masks, hydrostatic reconstruction, wave regions, limiter cases, friction
 * floors, the wet/dry clamp of the update) is the one the forward took.  For an edge the D
 * derivative lanes run in chunks over its 6 (first order) or 10 (WAF: + the upwind
 * reconstructions) inputs; D trades registers for repeated value lanes.  The element stage
 * is transposed by hand (adj_element), and so is the first-order HLLC edge of flux_mode 0 (AdjSide, two
 * lanes per edge).
 *
 * Replay kernels (k_rep_edges, k_rep_cells) advance a state with a recorded dt / time
 * sequence; they run the step's own edge_lanes / element_update, so a replayed trajectory is
 * bit-identical to the recorded one.
 */
#include <cuda_runtime.h>

#include <algorithm>

#include "cf_cell_kernel.cuh"
#include "cf_dual.h"
#include "cf_edge_kernel.cuh"
#include "cf_xd.h"

namespace cf {
namespace {

/* Dual<D> for input k of the lane chunk starting at base */
template <int D>
__device__ __forceinline__ Dual<D> seed(double v, int k, int base) {
  Dual<D> r(v);
#pragma unroll
  for (int i = 0; i < D; ++i) r.d[i] = (k - base == i) ? 1.0 : 0.0;
  return r;
}

/* ---- replay of the forward -------------------------------------------------------------- */

/* The recorded dt and start time of step n of member m: histories are [N][members]. */
__device__ __forceinline__ size_t hidx(int n, int m, int nm) { return (size_t)n * nm + m; }

/* The replays keep the forward kernels' occupancy, 1024 threads per SM (64 registers), where the latency
 * of the integer-pipe chains is hidden by more warps. */
template <int IFLUX>
__global__ void __launch_bounds__(2 * TILE_E, 4) k_rep_edges(StepArgs a, StepRec r, const double* dt_hist, const double* t_hist, int n) {
  const int tile = blockIdx.x;
  if (tile == a.n_etiles) return record_gauges(r, a.Uin);
  const int m = __ldg(a.etile_mem + tile);
  const MemberDev& M = a.mdev[m];
  const int e = tile * TILE_E + (threadIdx.x >> 1);
  EdgeHead E;
  E.load(a, e, e < M.edge_end);
  pdl_begin();
  const size_t h = hidx(n, m, a.nmembers);
  edge_lanes<IFLUX>(a, M, E, e, e, threadIdx.x & 1, e < M.edge_end, dt_hist[h], t_hist[h], nullptr);
}

template <int LANES>
__global__ void __launch_bounds__(128, 8) k_rep_cells(StepArgs a, const double* dt_hist, int n, uint32_t* flag,
                                                      Slot* sums_out) {
  const int c = (blockIdx.x * 128 + threadIdx.x) / LANES, comp = threadIdx.x % LANES;
  const int m = __ldg(a.ctile_mem + c / TILE_C);
  const MemberDev& M = a.mdev[m];
  const bool active = c < M.cell_end;
  pdl_begin();
  const double dt = dt_hist[hidx(n, m, a.nmembers)];
  double4 U = make_double4(0.0, 0.0, 0.0, 0.0), st = U, V = U;
  Slot s0, s1, s2;
  CompSums sums = {0.0, 0.0, 0.0, false};
  bool nonfinite = false;
  if (active) {
    U = ld4(a.Uin + c);
    st = ld4(a.cstat + c);
    const int4 sl = __ldg(a.cslot + c);
    if (LANES == 2) {
      sums = comp_sums(a.slots, sl, comp);
    } else {
      s0 = load_slot(a.slots + sl.x);
      s1 = load_slot(a.slots + sl.y);
      s2 = load_slot(a.slots + sl.z);
    }
  }
  if (LANES == 2) V = cell_lanes(a, M, comp, active, U, st, sums, dt, nonfinite);
  else if (active) V = cell_thread(a, M, U, st, s0, s1, s2, dt, nonfinite);
  if (nonfinite) atomicOr(flag, CF_STATUS_NONFINITE);
  if (!active) return;
  if (a.Uout) {
    double2* o = reinterpret_cast<double2*>(a.Uout + c);
    if (LANES == 2) {
      o[comp] = comp ? make_double2(V.z, V.w) : make_double2(V.x, V.y);
    } else {
      o[0] = make_double2(V.x, V.y);
      o[1] = make_double2(V.z, V.w);
    }
  }
  if (sums_out) {
    if (LANES == 2) store_comp_sums(sums_out + c, sums, comp);
    else store_sums(sums_out + c, s0, s1, s2);
  }
}

/* The gauge elevations of the last state (a step's edge launch records those of the state before it). */
__global__ void k_record(StepRec r, const double4* U) { record_gauges(r, U); }

/* ---- adjoint of the element stage --------------------------------------------------------- */

/* lambda^{n+1} of element c: its own part plus the contributions the edge adjoint of step n+1
 * left in its three slots and in the upwind entries it belongs to, plus the objective's
 * weights of the gauges it carries; fixed order. */
__device__ __forceinline__ double4 gather_lambda(const AdjArgs& A, int c, const int4& sl, int2 gauges, const double* gw) {
  double4 L = ld4(A.lam_own + c);
  const double4 e0 = ld4(A.eadj + sl.x), e1 = ld4(A.eadj + sl.y), e2 = ld4(A.eadj + sl.z);
  L.x = L.x + e0.x + e1.x + e2.x;
  L.y = L.y + e0.y + e1.y + e2.y;
  L.z = L.z + e0.z + e1.z + e2.z;
  if (A.uoff) {
    for (int j = __ldg(A.uoff + c), j1 = __ldg(A.uoff + c + 1); j < j1; ++j) {
      const double4 u = ld4(A.uadj + __ldg(A.uidx + j));
      L.x += u.x;
      L.y += u.y;
      L.z += u.z;
    }
  }
  if (gw)
    for (int j = gauges.x; j < gauges.y; ++j) L.x += gw[__ldg(A.gidx + j)];
  return L;
}

/* The transposed element stage (adj_element) of every element, with lambda gathered first.  Its values
 * and lone products run on the integer pipes, its sums and multiply-adds on the FP64 pipe: ~40 FP64
 * instructions per element, 243 while the friction ran on four dual lanes (51k triangles, with the
 * reverse edge then at one thread per edge: backward and forward of 50 steps 5.9 -> 4.8 ms).  Five, six and
 * eight blocks per SM measure the same within 3 %. */
constexpr int ADJ_CELLS_BLOCK = 128;
__global__ void __launch_bounds__(ADJ_CELLS_BLOCK, 6) k_adj_cells(AdjArgs A) {
  const StepArgs& a = A.s;
  const int c = blockIdx.x * ADJ_CELLS_BLOCK + threadIdx.x;
  const int mem = __ldg(a.ctile_mem + c / TILE_C);
  const MemberDev& M = a.mdev[mem];
  const bool active = c < M.cell_end;
  int4 sl = make_int4(0, 0, 0, 0);
  int2 gauges = make_int2(0, 0);
  if (active) {   /* the tables before the wait (here and below; 10k triangles 28.5 -> 27.9 us per reverse step) */
    sl = __ldg(a.cslot + c);
    if (A.gw) gauges = make_int2(__ldg(A.goff + c), __ldg(A.goff + c + 1));
  }
  pdl_begin();
  if (!active) return;
  const double dt = A.dt_hist[hidx(A.n, mem, a.nmembers)];
  const double4 U = ld4(a.Uin + c), st = ld4(a.cstat + c);
  const Slot sums = load_slot(A.sums + c);
  const double4 L = A.gather ? gather_lambda(A, c, sl, gauges, A.gw) : ld4(A.lam_init + c);
  double4 own;
  Slot w;
  double nb;
  adj_element(M, U, st, sums, L, dt, own, w, nb);
  A.lam_own[c] = own;
  store_slot(A.cadj + c, w.f1, w.f2, w.f3, w.bx, w.by, w.q);
  A.gman[c] += nb;
}

/* ---- adjoint of the edge stage ---------------------------------------------------------- */

/* lambda contributions of one upwind pair (U_i1, U_i2 -> the side's (h, v) reconstruction)
 * given the adjoints wh, wv of that reconstruction. */
__device__ __forceinline__ void upwind_chain(const double4* U, int i1, int i2, double d1, double d2, double ysum,
                                             double nx, double ny, double tolisec, double wh, double wv, double4* o1,
                                             double4* o2) {
  const double4 A1 = ld4(U + i1);
  const double4 A2 = (d1 < 0.0) ? make_double4(0.0, 0.0, 0.0, 0.0) : ld4(U + i2);
  Dual<6> hu_, vu_;
  upwind_mix(Dual<6>::var(A1.x, 0), Dual<6>::var(A1.y, 1), Dual<6>::var(A1.z, 2), A1.w, Dual<6>::var(A2.x, 3),
             Dual<6>::var(A2.y, 4), Dual<6>::var(A2.z, 5), A2.w, d1, d2, ysum, nx, ny, tolisec, hu_, vu_);
  *o1 = make_double4(wh * hu_.d[0] + wv * vu_.d[0], wh * hu_.d[1] + wv * vu_.d[1], wh * hu_.d[2] + wv * vu_.d[2], 0.0);
  *o2 = make_double4(wh * hu_.d[3] + wv * vu_.d[3], wh * hu_.d[4] + wv * vu_.d[4], wh * hu_.d[5] + wv * vu_.d[5], 0.0);
}

/* The transposed edge stage of boundary edge e (side A only): its flux differentiated in three
 * Dual lanes, contracted with the side's slot adjoint. */
template <int IFLUX>
__device__ __forceinline__ void adj_boundary_edge(const AdjArgs& A, const MemberDev& M, int e, int2 ab, double t) {
  const StepArgs& a = A.s;
  const double4 UA = ld4(a.Uin + ab.x);
  const double4 ez = ld4(a.ez + e);
  const Slot wa = A.cadj[ab.x];
  const double4 geo = ld4(a.egeo + e);
  const int id = ldro(a.ebid + e);
  Dual<3> f1, f2, f3, q;
  boundary_flux(IFLUX, M, ab.y, id, t, geo.x, geo.y, Dual<3>::var(UA.x, 0), Dual<3>::var(UA.y, 1),
                Dual<3>::var(UA.z, 2), UA.w, ez.x, f1, f2, f3, q);
  const double len = geo.z;
  double o[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) o[i] = (wa.f1 * f1.d[i] + wa.f2 * f2.d[i] + wa.f3 * f3.d[i]) * len;
  A.eadj[2 * (size_t)e] = make_double4(o[0], o[1], o[2], 0.0);
}

/* The transposed edge stage of interior edge e: the edge's slot values differentiated in Dual<D>
 * chunks over its 6 (first order) or 10 (WAF: + the upwind reconstructions) inputs, contracted
 * with the slot adjoints of its two elements. */
template <int IFLUX, int D>
__device__ __forceinline__ void adj_interior_edge(const AdjArgs& A, const MemberDev& M, int e, int2 ab, double dt) {
  const StepArgs& a = A.s;
  const double4 UA = ld4(a.Uin + ab.x);
  const double4 ez = ld4(a.ez + e);
  const Slot wa = A.cadj[ab.x];
  const double4 UB = ld4(a.Uin + ab.y);
  const Slot wb = A.cadj[ab.y];
  const EdgeGeo G = edge_geo(a, e, IFLUX >= 3);
  double hl_upw = 0.0, vl_upw = 0.0, hr_upw = 0.0, vr_upw = 0.0;
  int4 up = make_int4(0, 0, 0, 0);
  double4 dw = make_double4(0.0, 0.0, 0.0, 0.0);
  if (IFLUX >= 3) {
    up = ldro(a.eupw + e);
    dw = ld4(a.ewts + e);
    upwind_state(a.Uin, up.x, up.y, dw.x, dw.y, dw.x + dw.y, G.ysum_a, G.nx, G.ny, M.tolisec, hl_upw, vl_upw);
    upwind_state(a.Uin, up.z, up.w, dw.z, dw.w, dw.z + dw.w, G.ysum_b, G.nx, G.ny, M.tolisec, hr_upw, vr_upw);
  }
  constexpr int NDIR = (IFLUX >= 3) ? 10 : 6;
  const double w[10] = {wa.f1, wa.f2, wa.f3, wa.bx, wa.by, wb.f1, wb.f2, wb.f3, wb.bx, wb.by};
  double acc[NDIR];
#pragma unroll
  for (int base = 0; base < NDIR; base += D) {
    Dual<D> o[10];
    interior_edge<IFLUX>(M, a.ilimiteur, a.flux_mode, G, dt, seed<D>(UA.x, 0, base), seed<D>(UA.y, 1, base),
                         seed<D>(UA.z, 2, base), ez.x, UA.w, seed<D>(UB.x, 3, base), seed<D>(UB.y, 4, base),
                         seed<D>(UB.z, 5, base), ez.y, UB.w, seed<D>(hl_upw, 6, base), seed<D>(vl_upw, 7, base), ez.z,
                         seed<D>(hr_upw, 8, base), seed<D>(vr_upw, 9, base), ez.w, o, A.freeze_r != 0);
#pragma unroll
    for (int i = 0; i < D; ++i) {
      if (base + i < NDIR) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < 10; ++k) s = fma(w[k], o[k].d[i], s);
        acc[base + i] = s;
      }
    }
  }
  A.eadj[2 * (size_t)e] = make_double4(acc[0], acc[1], acc[2], 0.0);
  A.eadj[2 * (size_t)e + 1] = make_double4(acc[3], acc[4], acc[5], 0.0);
  if constexpr (IFLUX >= 3) {
    double4 c0, c1, c2, c3;
    upwind_chain(a.Uin, up.x, up.y, dw.x, dw.y, G.ysum_a, G.nx, G.ny, M.tolisec, acc[6], acc[7], &c0, &c1);
    upwind_chain(a.Uin, up.z, up.w, dw.z, dw.w, G.ysum_b, G.nx, G.ny, M.tolisec, acc[8], acc[9], &c2, &c3);
    double4* u = A.uadj + 4 * (size_t)e;
    u[0] = c0;
    u[1] = c1;
    u[2] = c2;
    u[3] = c3;
  }
}

template <int IFLUX, int D>
__global__ void __launch_bounds__(TILE_E) k_adj_edges(AdjArgs A) {
  const StepArgs& a = A.s;
  const int tile = blockIdx.x;
  const int m = __ldg(a.etile_mem + tile);
  const MemberDev& M = a.mdev[m];
  const int e = tile * TILE_E + threadIdx.x;
  pdl_begin();
  if (e >= M.edge_end) return;
  const size_t h = hidx(A.n, m, a.nmembers);
  const double dt = A.dt_hist[h], t = A.t_hist[h];
  const int2 ab = ldro(a.ecell + e);
  if (ab.y < 0) adj_boundary_edge<IFLUX>(A, M, e, ab, t);
  else adj_interior_edge<IFLUX, D>(A, M, e, ab, dt);
}

/* One side of a reverse HLLC edge on this lane, the other one on lane ^ 1; mask: the lanes at work */
struct AdjLanePair {
  AdjSide s;
  double lam[3];
  unsigned mask;
  template <class F>
  __device__ __forceinline__ void each(F&& f) { f(s, lam); }
  __device__ __forceinline__ void exchange(int n) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < n) s.y[k] = XD<true>(__shfl_xor_sync(mask, val(s.x[k]), 1));
  }
  __device__ __forceinline__ void finish() {
    if (__any_sync(mask, s.odd)) {
      const bool odd = s.odd | __shfl_xor_sync(mask, (int)s.odd, 1);
      double o[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, q[6], one[3];
      if (odd) s.one_side(o);
#pragma unroll
      for (int k = 0; k < 6; ++k) q[k] = __shfl_xor_sync(mask, o[k], 1);
      s.join(o, q, one);
      s.reverse3(odd ? one : nullptr, lam);
    } else {
      s.reverse3(nullptr, lam);
    }
  }
};

/* First-order HLLC (flux_mode 0): the closed-form reverse edge (AdjSide), two lanes per edge as in the
 * edge kernel: ~3,000 instructions a lane, 59 of them FP64 ones.  Us per reverse step, 22k / 51k
 * triangles: 25 / 33 (one thread per edge: 39, latency-bound / 38; on four dual lanes 339 at 200k).
 * BLOCKS per SM: 3 (80 registers; 16 and 20 warps per SM measured the same), or 4 (64 registers, some
 * spilled) where that makes all edges resident at once and 3 would leave a second, nearly empty wave: us
 * per reverse step with 3 / 4 at 39.4k triangles 42.2 / 39.7, 42k 43.9 / 42.0, 48k 46.2 / 42.9, 51.6k 46.8 /
 * 43.1; on either side of that, 38.6k 34.5 / 35.5 and 52.4k 47.0 / 49.4.  Where 4 saves the third wave it does
 * not pay: 79k 61.9 / 61.6, 90k 65.5 / 64.8, 96k 67.5 / 69.2, 103k 70.0 / 71.5; at 200k 138.3 / 140.5. */
template <int BLOCKS>
__global__ void __launch_bounds__(2 * TILE_E, BLOCKS) k_adj_edges_hllc(AdjArgs A) {
  const StepArgs& a = A.s;
  const int tile = blockIdx.x;
  const int m = __ldg(a.etile_mem + tile);
  const MemberDev& M = a.mdev[m];
  const int e = tile * TILE_E + (threadIdx.x >> 1), side = threadIdx.x & 1;
  const bool live = e < M.edge_end;
  EdgeHead E;
  E.load(a, e, live);
  double2 z = make_double2(0.0, 0.0);
  if (live) z = ldro(reinterpret_cast<const double2*>(a.ez + e));
  pdl_begin();
  const int2 ab = E.ab;
  const bool run = live && ab.y >= 0;
  const unsigned mask = __ballot_sync(0xffffffffu, run);
  if (run) {
    const int c = side ? ab.y : ab.x;
    const double4 geo = E.geo, U = ld4(a.Uin + c);
    const Slot wc = load_slot(A.cadj + c);
    const double w[5] = {wc.f1, wc.f2, wc.f3, wc.bx, wc.by};
    AdjLanePair p;
    p.mask = mask;
    p.s.begin(M, side, geo, U, side ? z.y : z.x, side ? z.x : z.y, w);
    adj_stages(p);
    A.eadj[2 * (size_t)e + side] = make_double4(p.lam[0], p.lam[1], p.lam[2], 0.0);
  } else if (live && side == 0) {
    adj_boundary_edge<1>(A, M, e, ab, A.t_hist[hidx(A.n, m, a.nmembers)]);
  }
}

/* ---- lambda^0 -------------------------------------------------------------------------- */

__global__ void __launch_bounds__(TILE_C) k_adj_final(AdjArgs A) {
  const int tile = blockIdx.x;
  const MemberDev& M = A.s.mdev[__ldg(A.s.ctile_mem + tile)];
  const int c = tile * TILE_C + threadIdx.x;
  if (c >= M.cell_end) return;
  A.lam_own[c] = gather_lambda(A, c, __ldg(A.s.cslot + c), make_int2(0, 0), nullptr);
}

/* lambda.h += the objective's weights of the gauges an element carries (the final state's
 * gauge terms) */
__global__ void k_add_gauges(double4* lam, const int32_t* goff, const int32_t* gidx, const double* gw, int n) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  for (int j = goff[c]; j < goff[c + 1]; ++j) lam[c].x += gw[gidx[j]];
}

__global__ void k_gather_scalar(const double* x, const int32_t* iperm, double* out, int n) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o < n) out[o] = x[iperm[o]];
}

__global__ void k_set_manning(double4* cstat, const int32_t* perm, const double* nref, int n) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < n) cstat[c].y = nref[perm[c]];
}

/* ---- Manning zones (calibration parameters) ------------------------------------------------ */

/* dJ/d(zone value) = the sum of dJ/dn over the zone's elements, in the fixed order of the
 * zone's element list (one block per zone: strided partial sums, then a tree). */
__global__ void __launch_bounds__(256) k_zone_sum(const double* gman, const int32_t* zoff, const int32_t* zidx,
                                                  double* gz) {
  __shared__ double s[256];
  const int z = blockIdx.x;
  double v = 0.0;
  for (int j = zoff[z] + threadIdx.x; j < zoff[z + 1]; j += 256) v += gman[zidx[j]];
  s[threadIdx.x] = v;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) gz[z] = s[0];
}

/* projected gradient step on the zone values: v = min(hi, max(lo, v - lr g)) */
__global__ void k_zone_step(double* v, const double* g, int nz, double lr, double lo, double hi) {
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  if (z < nz) v[z] = fmin(hi, fmax(lo, v[z] - lr * g[z]));
}

/* the Manning n of every element of a zone (elements without a zone keep theirs) */
__global__ void k_zone_apply(double4* cstat, const int32_t* zone_of, const double* v, int n) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < n && zone_of[c] >= 0) cstat[c].y = v[zone_of[c]];
}

int chk(cudaError_t e) { return e == cudaSuccess ? CF_OK : CF_ECUDA; }

}  // namespace

int launch_replay_step(const StepArgs& a, const double* dt_hist, const double* t_hist, int n, uint32_t* flag,
                       Slot* sums, stream_t s, const StepRec& rec) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(s);
  const int nb = a.n_etiles + (rec.eta ? 1 : 0);
  switch (a.iflux) {
    case 1: launch_pdl(k_rep_edges<1>, nb, 2 * TILE_E, st, a, rec, dt_hist, t_hist, n); break;
    case 2: launch_pdl(k_rep_edges<2>, nb, 2 * TILE_E, st, a, rec, dt_hist, t_hist, n); break;
    case 3: launch_pdl(k_rep_edges<3>, nb, 2 * TILE_E, st, a, rec, dt_hist, t_hist, n); break;
    default: return CF_ENOTSUP;
  }
  const int nc = a.n_ctiles * TILE_C;
  if (two_lanes(a)) launch_pdl(k_rep_cells<2>, 2 * nc / 128, 128, st, a, dt_hist, n, flag, sums);
  else launch_pdl(k_rep_cells<1>, nc / 128, 128, st, a, dt_hist, n, flag, sums);
  return chk(cudaGetLastError());
}

int launch_record(const StepRec& r, const double4* U, stream_t s) {
  launch_pdl(k_record, 1, 256, reinterpret_cast<cudaStream_t>(s), r, U);
  return chk(cudaGetLastError());
}

static void adj_edges_hllc(const AdjArgs& A, cudaStream_t st) {
  const int n = A.s.n_etiles;
  if (adj_hllc_blocks(n, A.s.sms) == 4) launch_pdl(k_adj_edges_hllc<4>, n, 2 * TILE_E, st, A);
  else launch_pdl(k_adj_edges_hllc<3>, n, 2 * TILE_E, st, A);
}

int launch_adjoint_step(const AdjArgs& A, stream_t s) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(s);
  const StepArgs& a = A.s;
  launch_pdl(k_adj_cells, a.n_ctiles * (TILE_C / ADJ_CELLS_BLOCK), ADJ_CELLS_BLOCK, st, A);
  switch (a.iflux) {
    case 1:
      if (a.flux_mode == 0) adj_edges_hllc(A, st);
      else launch_pdl(k_adj_edges<1, 6>, a.n_etiles, TILE_E, st, A);
      break;
    case 2: launch_pdl(k_adj_edges<2, 3>, a.n_etiles, TILE_E, st, A); break;
    case 3: launch_pdl(k_adj_edges<3, 2>, a.n_etiles, TILE_E, st, A); break;
    default: return CF_ENOTSUP;
  }
  return chk(cudaGetLastError());
}

int launch_adjoint_final(const AdjArgs& A, stream_t s) {
  k_adj_final<<<A.s.n_ctiles, TILE_C, 0, reinterpret_cast<cudaStream_t>(s)>>>(A);
  return chk(cudaGetLastError());
}

int launch_add_gauges(double4* lam, const int32_t* goff, const int32_t* gidx, const double* gw, int32_t n, stream_t s) {
  if (n <= 0) return CF_OK;
  k_add_gauges<<<(n + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(s)>>>(lam, goff, gidx, gw, n);
  return chk(cudaGetLastError());
}

int launch_gather_scalar(const double* x, const int32_t* iperm, double* out, int32_t n, stream_t s) {
  if (n <= 0) return CF_OK;
  k_gather_scalar<<<(n + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(s)>>>(x, iperm, out, n);
  return chk(cudaGetLastError());
}

int launch_set_manning(double4* cstat, const int32_t* perm, const double* nref, int32_t n, stream_t s) {
  if (n <= 0) return CF_OK;
  k_set_manning<<<(n + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(s)>>>(cstat, perm, nref, n);
  return chk(cudaGetLastError());
}

int launch_zone_sum(const double* gman, const int32_t* zoff, const int32_t* zidx, double* gz, int32_t nz, stream_t s) {
  if (nz <= 0) return CF_OK;
  k_zone_sum<<<nz, 256, 0, reinterpret_cast<cudaStream_t>(s)>>>(gman, zoff, zidx, gz);
  return chk(cudaGetLastError());
}

int launch_zone_step(double* v, const double* g, int32_t nz, double lr, double lo, double hi, stream_t s) {
  if (nz <= 0) return CF_OK;
  k_zone_step<<<(nz + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(s)>>>(v, g, nz, lr, lo, hi);
  return chk(cudaGetLastError());
}

int launch_zone_apply(double4* cstat, const int32_t* zone_of, const double* v, int32_t n, stream_t s) {
  if (n <= 0) return CF_OK;
  k_zone_apply<<<(n + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(s)>>>(cstat, zone_of, v, n);
  return chk(cudaGetLastError());
}

}  // namespace cf
