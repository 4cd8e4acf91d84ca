// The LagrangeLeapFrog step as four sm_103a kernels. k_force and k_kinematics
// run three threads per element, one per coordinate, on 64-bit fixed-point
// numbers (lulesh_fixed.cuh; elements these do not take in FP64), k_node and
// k_material one thread per node or element in FP64:
//   k_force      calcVolumeForceForElems: stress integration + FB hourglass,
//                one 8-corner force triple per element corner
//                (src/domain.jl:963-1762)
//   k_node       deterministic corner-force gather in nodeElemCornerList
//                order + acceleration, symmetry BCs, velocity and position
//                (src/domain.jl:1112-1127, 1676-1693, 1781-1838)
//   k_kinematics calcKinematicsForElems + calcLagrangeElements +
//                calcMonotonicQGradientsForElems (src/domain.jl:2099-2320)
//   k_material   calcMonotonicQRegionForElems + qstop check +
//                applyMaterialPropertiesForElems/evalEOSForElems +
//                updateVolumesForElems + Courant/hydro dt minima
//                (src/domain.jl:2322-3064)
// plus timeIncrement! (src/domain.jl:920-961) for the device-resident run loop,
// in blocks of k_force or as k_time_increment.
#include "lulesh_courant.cuh"
#include "lulesh_device.cuh"
#include "lulesh_element_fp64.cuh"
#include "lulesh_fixed_force.cuh"
#include "lulesh_fixed_kin.cuh"
#include "lulesh_kernels.h"
#include "lulesh_launch.cuh"

namespace lulesh {

// Each kernel stops at once when an earlier kernel of the step (or of the
// device run loop) recorded an error or finished the run, as the reference
// stops at its first raised error.
__device__ __forceinline__ bool step_off(const DevState* st) {
  const uint2 f = __ldcv(reinterpret_cast<const uint2*>(&st->status));
  return (f.x | f.y) != 0u;
}

// timeIncrement! of one problem in the device run loop.
__device__ void advance_time(DevState* st, const Params& prm) {
  if (st->done) return;
  if (st->status) { st->done = 1; return; }
  // fold the previous step's minima (src/domain.jl:3012-3014, 3050-3052)
  if (dt_registers(st->acc_courant)) st->dtcourant = __longlong_as_double((long long)st->acc_courant);
  if (dt_registers(st->acc_hydro)) st->dthydro = __longlong_as_double((long long)st->acc_hydro);
  st->acc_courant = kInfBits;
  st->acc_hydro = kInfBits;
  // examples/benchmark.jl:82-98: while time < stoptime ... break if cycle >= num_iters
  if (!(st->time < prm.stoptime) || (!st->first && st->cycle >= st->num_iters)) { st->done = 1; return; }
  st->first = 0;
  double time = st->time, dt = st->deltatime;
  long long cycle = st->cycle;
  time_increment(time, dt, cycle, st->dtcourant, st->dthydro, prm);
  st->time = time;
  st->deltatime = dt;
  st->cycle = cycle;
}

// blocks of k_force that run the time steps of n problems
__host__ __device__ constexpr int time_blocks(int n) { return (n + 3 * kFixedElems - 1) / (3 * kFixedElems); }

// ---------------------------------------------------------------------------
// k_force
// ---------------------------------------------------------------------------
// The taped volume derivatives, scaled modes and mode sums of an element.
template <bool ON>
struct ForceTape {
  static constexpr bool on = ON;
  double* p;  // d.tapeGeo at this element
  int E;
  bool live;
  __device__ void put(int slot, double v) const { if (live) p[row(slot, E, 0)] = v; }
  __device__ void derivative(int k, int n, double v) const { put(8 * k + n, v); }
  __device__ void mode(int k, int m, double v) const { put(24 + 4 * k + m, v); }
  __device__ void sum(int k, int m, double v) const { put(36 + 4 * k + m, v); }
};

// The FP64 form, for the elements of a block that the fixed-point form does not
// take (`mine`); every thread of the block calls it. Out of line: its registers
// are not the kernel's.
template <int MODE, bool TAPE>
__device__ __noinline__ void force_fallback(const DevDomain& d, DevState* st, unsigned* status, fx::Num* column, int e,
                                            bool mine, double hgcoef) {
  const int E = d.E;
  const int lane = threadIdx.x % kFixedElems, k = threadIdx.x / kFixedElems;
  const double* const X = k == 0 ? d.x : k == 1 ? d.y : d.z;
  const double* const U = k == 0 ? d.xd : k == 1 ? d.yd : d.zd;
  double x[8], v[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int nd = LULESH_IDX(LDG(&d.nodelist[c * E + e]), d.N, st);
    x[c] = X[nd];
    v[c] = U[nd];
  }
  ForceScalars c;
  c.v = d.v[e];
  const double rc = inv_cbrt(LDG(&d.volo[e]) * c.v);
  c.vi12 = (rc * rc) * (rc * (1.0 / 12.0));
  c.coef = ((-hgcoef * 0.01) * d.ss[e]) * LDG(&d.elemMass[e]) * rc;
  c.s8 = ((-d.p[e]) - d.q[e]) * 0.125;
  c.hourglass = gt_zero(hgcoef);
  double* const out = (k == 0 ? d.fcx : k == 1 ? d.fcy : d.fcz) + e;
  force_fp64<MODE>(k, RealSlots{reinterpret_cast<double*>(column) + lane, kFixedElems}, x, v, c, mine, status,
                   [&](int n, double f) { out[n * E] = f; }, ForceTape<TAPE>{TAPE ? d.tapeGeo + e : nullptr, E, true});
}

// Three threads per element, one per coordinate and each in a warp of its own:
// a block is 32 elements (lulesh_fixed_force.cuh). Bound by the integer pipes
// (multiply-adds, shifts and logic issue every other cycle and share them: ALU 52 %
// and FMA-heavy 40 % of the cycles, FP64 28 %): 0.92 ms per cycle at 150^3, where
// FP64 took 1.98 ms with the geometry stored by k_kinematics (0.87 ms of that
// kernel). Eight blocks per SM, 80 registers: seven 0.94 ms, six (96 registers)
// 1.02; below 45^3 alike.
//
// TIME: the cycle's timeIncrement! runs here too, by blocks of its own after
// the elements'; the forces need neither dt nor time. The element blocks may
// see the problem's done flag of before or after: a cycle it ends leaves
// nothing but the corner forces, which nobody reads. An error they find waits in
// force_status until k_node knows whether the cycle takes place. A launch less
// per cycle: 25.8 -> 22.7 us at 8^3, 40.2 -> 35.3 at 30^3, 2139 -> 2137 at 150^3,
// with the flags read in one load (one by one, past the first-level cache,
// k_node's third flag cost 12 us at 150^3).
template <int MODE, bool ENS, bool TAPE, bool TIME>
__global__ void __launch_bounds__(3 * kFixedElems, 8)
    k_force(const __grid_constant__ DevDomain d, const __grid_constant__ Params prm) {
  __shared__ fx::Num column[fx::FS_COUNT * kFixedElems];
  const int E = d.E;
  const int lane = threadIdx.x % kFixedElems, k = threadIdx.x / kFixedElems;
  if (TIME) {
    const int block = blockIdx.x - (E + kFixedElems - 1) / kFixedElems;
    if (block >= 0) {
      const int problem = block * (3 * kFixedElems) + threadIdx.x;
      wait_for_last_kernel();
      if (problem < d.ninst) advance_time(d.st + problem, prm);
      return;
    }
  }
  // threads past the end repeat the last element and store nothing
  const int slot = blockIdx.x * kFixedElems + lane;
  const int e = slot < E ? slot : E - 1;
  const int inst = ENS ? LULESH_IDX(LDG(&d.elemInst[e]), d.ninst, d.st) : 0;
  DevState* const st = d.st + inst;
  int nd[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) nd[c] = LULESH_IDX(LDG(&d.nodelist[c * E + e]), d.N, st);
  wait_for_last_kernel();
  const bool live = slot < E && !step_off(st);
  if (!__syncthreads_or(live)) return;
  const double hgcoef = ENS ? LDG(&d.instHg[inst]) : prm.hgcoef;
  const fx::Slots sh{column + lane, kFixedElems};
  fx::ForceLane r;
  const ForceTape<TAPE> tape{TAPE ? d.tapeGeo + e : nullptr, E, live};
  {
    const double* const X = k == 0 ? d.x : k == 1 ? d.y : d.z;
    const double* const U = k == 0 ? d.xd : k == 1 ? d.yd : d.zd;
    double v[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      r.x[c] = X[nd[c]];
      v[c] = U[nd[c]];
    }
    if (k == 0) {
      // determ^(-1/3) serves the coefficient (src/domain.jl:1605), its cube
      // the modes' 1/(12 determ); a volume that is not positive takes neither
      const double vol = d.v[e];
      const double rc = inv_cbrt(LDG(&d.volo[e]) * vol);
      const double coef = gt_zero(hgcoef) ? ((-hgcoef * 0.01) * d.ss[e]) * LDG(&d.elemMass[e]) * rc : 0.0;
      fx::force_scales(sh, gt_zero(vol) ? (rc * rc) * (rc * (1.0 / 12.0)) : 0.0, coef);
    } else if (k == 1) {
      fx::force_stress(sh, ((-d.p[e]) - d.q[e]) * 0.125);
    }
    fx::force_load(k, sh, v, r);
  }
  long long hm[4];
  __syncthreads();
  fx::force_diagonals(k, sh, r, hm, fx::wide());
  __syncthreads();
  fx::force_products<MODE>(k, sh, r, hm, tape, fx::wide());
  __syncthreads();
  fx::force_base(k, sh, r);
  const int others = __syncthreads_or(live && !r.ok);
  if (live && r.ok) {
    double* const out = (k == 0 ? d.fcx : k == 1 ? d.fcy : d.fcz) + e;
    fx::force_corners(k, sh, r, [&](int n, double f) { out[n * E] = f; }, tape);
  }
  if (others) {
    __syncthreads();
    force_fallback<MODE, TAPE>(d, st, TIME ? &st->force_status : &st->status, column, e, live && !r.ok, hgcoef);
  }
}

// ---------------------------------------------------------------------------
// k_node
// ---------------------------------------------------------------------------
template <bool AUX, bool ENS>
__global__ void __launch_bounds__(kMaxNodeBlock) k_node(DevDomain d, Params prm) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.N) return;
  DevState* const st = d.st + (ENS ? LULESH_IDX(LDG(&d.nodeInst[i]), d.ninst, d.st) : 0);
  const int s = LDG(&d.nodeElemStart[i]);
  int t = LDG(&d.nodeElemStart[i + 1]);
  const double im = LDG(&d.inv_nodalMass[i]);
  const int first = s < t ? LDG(&d.cornerList[LULESH_IDX(s, d.nCornerList, st)]) : 0;
  wait_for_last_kernel();
  const uint4 flags = __ldcv(reinterpret_cast<const uint4*>(&st->status));  // status, done, force_status
  const double dt = st->deltatime;
  if (flags.x | flags.y) return;
  // what a k_force that ran beside the time step found
  if (flags.z) {
    atomicOr(&st->status, flags.z);
    return;
  }
#ifdef LULESH_CHECK
  // the node's corner range must lie within the corner list; an empty one reads nothing
  if (s < 0 || t < s || t > d.nCornerList) { atomicOr(&st->status, ST_INDEX); t = s; }
#endif
  double fx = 0.0, fy = 0.0, fz = 0.0;
  if (s < t) {
    const int c0 = LULESH_IDX(first, d.nCornerSlot, st);
    fx = d.fcx[c0]; fy = d.fcy[c0]; fz = d.fcz[c0];
    for (int j = s + 1; j < t; ++j) {
      const int c = LULESH_IDX(LDG(&d.cornerList[j]), d.nCornerSlot, st);
      fx += d.fcx[c]; fy += d.fcy[c]; fz += d.fcz[c];
    }
  }
  double ax = fx * im, ay = fy * im, az = fz * im;
  const unsigned bc = d.nodeBC[i];
  if (bc & 1u) ax = 0.0;
  if (bc & 2u) ay = 0.0;
  if (bc & 4u) az = 0.0;
  double xd = fma(ax, dt, d.xd[i]);
  double yd = fma(ay, dt, d.yd[i]);
  double zd = fma(az, dt, d.zd[i]);
  if (abs_lt(xd, prm.u_cut)) xd = 0.0;
  if (abs_lt(yd, prm.u_cut)) yd = 0.0;
  if (abs_lt(zd, prm.u_cut)) zd = 0.0;
  d.xd[i] = xd; d.yd[i] = yd; d.zd[i] = zd;
  d.x[i] = fma(xd, dt, d.x[i]);
  d.y[i] = fma(yd, dt, d.y[i]);
  d.z[i] = fma(zd, dt, d.z[i]);
  if (AUX) {
    d.fx[i] = fx; d.fy[i] = fy; d.fz[i] = fz;
    d.xdd[i] = ax; d.ydd[i] = ay; d.zdd[i] = az;
  }
}

// ---------------------------------------------------------------------------
// k_kinematics
// ---------------------------------------------------------------------------
// The quotients of the elements marked `mine` from the sums that `get` gives,
// divided among the three threads: coordinate 1 the divergence and 1/(64
// volume), both from one division, coordinate 0 the volume's change and the
// characteristic length, coordinate k direction k of the monotonic-Q gradients.
// Every thread of the block calls it. Returns the largest face's place (taped
// runs).
template <bool AUX, bool TAPE, class Sums>
__device__ __forceinline__ int kin_quotients(const DevDomain& d, DevState* st, const fx::Slots& sh, int k, int e,
                                             bool mine, const Sums& get) {
  const int E = d.E;
  const double volume = get.volume12() * (1.0 / 12.0);
  const double vnew = volume * LDG(&d.inv_volo[e]);
  const double volq = LDG(&d.volo[e]) * vnew;
  double rcl = 0.0;
  auto tape = [&](int slot, double v) { d.tapeKin[row(slot, E, e)] = v; };
  if (mine) {
    if (k == 1) {
      const double q64 = fma(64.0, volq, 64.0 * 1.e-36);
      double inv, norm64;
      recip2(get.jacobian(), q64, inv, norm64);
      const double vdov = get.rate() * inv;
      d.vdov[e] = vdov;
      sh.put(fx::KS_MID, __double_as_longlong(norm64));
      if (AUX) {
        sh.put(fx::KS_MID + 1, __double_as_longlong(inv));
        sh.put(fx::KS_MID + 2, __double_as_longlong(vdov));
      }
      if (TAPE) {
        tape(27, inv);
        tape(40, norm64);
      }
    } else if (k == 0) {
      // 4*volume/sqrt(max area) with area = 4*|face vector|^2
      // (src/domain.jl:1874-1930)
      int place;
      rcl = rsqrt(get.face(place));
      if (le_zero(vnew)) atomicOr(&st->status, ST_KINEMATICS);
      d.vnew[e] = vnew;
      d.delv[e] = vnew - d.v[e];
      d.arealg[e] = (2.0 * volume) * rcl;
      if (TAPE) sh.put(fx::KS_MID + 1, place);
    }
  }
  __syncthreads();
  if (!mine) return 0;
  // src/domain.jl:2175-2320; with the reference's dxi = W_xi/4 etc.: delx =
  // 16*vol/sqrt(|A|^2 + 256*ptiny) and delv = norm/64 * (A . W(v)) for the cross
  // product A of two Walsh vectors
  double* const delx = k == 0 ? d.delx_xi : k == 1 ? d.delx_eta : d.delx_zeta;
  double* const delv = k == 0 ? d.delv_xi : k == 1 ? d.delv_eta : d.delv_zeta;
  const double norm64 = __longlong_as_double(sh.get(fx::KS_MID));
  const double rs = rsqrt(get.area(k));
  delx[e] = (16.0 * volq) * rs;
  delv[e] = norm64 * get.flow(k);
  if (AUX) {
    double* const dd = k == 0 ? d.dxx : k == 1 ? d.dyy : d.dzz;
    const double inv = __longlong_as_double(sh.get(fx::KS_MID + 1));
    const double vdov = __longlong_as_double(sh.get(fx::KS_MID + 2));
    dd[e] = get.own_rate(k) * inv - vdov / 3.0;
  }
  if (!TAPE) return 0;
  const int place = (int)sh.get(fx::KS_MID + 1);
  tape(37 + k, rs);
  if (k == 0) {
    tape(44, rcl);
    d.tapeFlags[e] = (unsigned long long)place << TF_FACE_SHIFT;
  }
  return place;
}

// Coordinate k's taped components; t gives them as doubles. The 12 diagonals
// in the order d61 d70 d63 d20 d50 d64 d31 d72 d43 d57 d14 d25 (force-order
// index, sign), the largest face's vector in the reference's face order, the
// last two faces with reversed diagonals.
template <class Taped>
__device__ __forceinline__ void kin_tape(const DevDomain& d, int k, int e, int place, const Taped& t) {
  const int E = d.E;
  auto put = [&](int slot, double v) { d.tapeKin[row(slot, E, e)] = v; };
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    put(3 * k + a, t.w(a));
    put(9 + 3 * k + a, t.vw(a));
    put(18 + 3 * a + k, t.C(a));
    put(28 + 3 * a + k, t.A(a));
    put(81 + 3 * a + k, t.gU(a));
  }
  constexpr int gi[12] = {4, 9, 7, 0, 2, 10, 1, 6, 8, 11, 3, 5};
#pragma unroll
  for (int q = 0; q < 12; ++q) put(45 + 3 * q + k, q == 1 || q == 2 ? -t.g(gi[q]) : t.g(gi[q]));
  const double c = place == 0 ? t.n(0) : place == 1 ? t.n(5) : place == 2 ? t.n(1) : place == 3 ? t.n(2)
                                    : place == 4 ? -t.n(3) : -t.n(4);
  put(41 + k, c);
}

// The next cycle's face normals, for its hourglass transpose.
template <class Taped>
__device__ __forceinline__ void kin_tape_next(const DevDomain& d, int k, int e, const Taped& t) {
#pragma unroll
  for (int f = 0; f < 5; ++f) d.tapeGeoNext[row(48 + 6 * k + f, d.E, e)] = t.n(f);
}

struct FixedSums {
  const fx::Slots& sh;
  const fx::KinLane& r;
  __device__ double volume12() const { return fx::kin_volume12(sh, r); }
  __device__ double face(int& place) const { return fx::kin_largest_face(sh, r, place); }
  // (from 2^-54 up the guard is below half a unit)
  __device__ double area(int k) const {
    const double a = fx::kin_area(sh, r, k);
    return fx::hi_word(a) < (1023 - 54) << 20 ? a + 256.e-36 : a;
  }
  __device__ double flow(int k) const { return fx::kin_flow(sh, r, k); }
  __device__ double rate() const { return fx::kin_rate(sh, r); }
  __device__ double jacobian() const { return fx::kin_jacobian(sh, r); }
  __device__ double own_rate(int k) const { return fx::kin_own_rate(sh, r, k); }
};
struct FixedTaped {
  const fx::KinLane& r;
  __device__ double w(int a) const { return fx::to_double(r.w[a], 2 - r.s); }
  __device__ double vw(int a) const { return fx::to_double(r.vw[a], 2 - r.sv); }
  __device__ double C(int a) const { return fx::to_double(r.C[a], 66 - (r.all - r.s)); }
  __device__ double A(int a) const { return fx::to_double(r.A[a], 68 - r.up[a] - (r.all - r.s)); }
  __device__ double gU(int a) const { return fx::to_double(r.gU[a], 64 - (r.all - r.s)); }
  __device__ double g(int q) const { return fx::to_double(r.g[q], -r.s); }
  __device__ double n(int f) const { return fx::to_double(r.n[f], 64 - (r.all - r.s)); }
};
struct RealSums {
  const KinSums& s;
  __device__ double volume12() const { return s.volume12; }
  __device__ double face(int& place) const { place = s.place; return s.face; }
  __device__ double area(int) const { return s.area; }
  __device__ double flow(int) const { return s.flow; }
  __device__ double rate() const { return s.rate; }
  __device__ double jacobian() const { return s.jacobian; }
  __device__ double own_rate(int) const { return s.own_rate; }
};
struct RealTaped {
  const KinTaped& t;
  __device__ double w(int a) const { return t.w[a]; }
  __device__ double vw(int a) const { return t.vw[a]; }
  __device__ double C(int a) const { return t.C[a]; }
  __device__ double A(int a) const { return t.A[a]; }
  __device__ double gU(int a) const { return t.gU[a]; }
  __device__ double g(int q) const { return t.g[q]; }
  __device__ double n(int f) const { return t.n[f]; }
};

// The FP64 form, for the elements of a block that the fixed-point form does not
// take (`mine`); every thread of the block calls it. `geometry`: the next
// cycle's normals are its too (they depend on the positions alone, and the
// fixed-point form takes those of an element whose velocities it refuses).
template <bool AUX, bool TAPE>
__device__ __noinline__ void kin_fallback(const DevDomain& d, DevState* st, fx::Num* column, int e, bool mine,
                                          bool geometry, double dt) {
  const int E = d.E;
  const int lane = threadIdx.x % kFixedElems, k = threadIdx.x / kFixedElems;
  const double* const X = k == 0 ? d.x : k == 1 ? d.y : d.z;
  const double* const U = k == 0 ? d.xd : k == 1 ? d.yd : d.zd;
  double x[8], v[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int nd = LULESH_IDX(LDG(&d.nodelist[c * E + e]), d.N, st);
    x[c] = X[nd];
    v[c] = U[nd];
  }
  KinSums sums;
  KinTaped t;
  kin_fp64(k, RealSlots{reinterpret_cast<double*>(column) + lane, kFixedElems}, x, v, dt, sums, t);
  const int place = kin_quotients<AUX, TAPE>(d, st, fx::Slots{column + lane, kFixedElems}, k, e, mine, RealSums{sums});
  if (TAPE && mine) {
    kin_tape(d, k, e, place, RealTaped{t});
    if (d.tapeGeoNext && geometry) kin_tape_next(d, k, e, RealTaped{t});
  }
}

// Three threads per element as in k_force (lulesh_fixed_kin.cuh). Bound by the
// integer pipes (ALU 60 %, FMA-heavy 34 %) and FP64 (59 %): 0.65 ms per cycle at
// 150^3 (FP64: 1.93 ms without the force geometry), of which the scales by
// coordinate and the terms' exponents are 0.09. Seven blocks per SM, 80 registers:
// eight 0.66 ms, six (96) 0.79.
template <bool AUX, bool ENS, bool TAPE>
__global__ void __launch_bounds__(3 * kFixedElems, 7)
    k_kinematics(const __grid_constant__ DevDomain d, const __grid_constant__ Params prm) {
  __shared__ fx::Num column[fx::KS_COUNT * kFixedElems];
  const int E = d.E;
  const int lane = threadIdx.x % kFixedElems, k = threadIdx.x / kFixedElems;
  // threads past the end repeat the last element and store nothing
  const int slot = blockIdx.x * kFixedElems + lane;
  const int e = slot < E ? slot : E - 1;
  DevState* const st = d.st + (ENS ? LULESH_IDX(LDG(&d.elemInst[e]), d.ninst, d.st) : 0);
  int nd[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) nd[c] = LULESH_IDX(LDG(&d.nodelist[c * E + e]), d.N, st);
  wait_for_last_kernel();
  const bool live = slot < E && !step_off(st);
  if (!__syncthreads_or(live)) return;
  const double dt = st->deltatime;
  const fx::Slots sh{column + lane, kFixedElems};
  fx::KinLane r;
  {
    const double* const X = k == 0 ? d.x : k == 1 ? d.y : d.z;
    const double* const U = k == 0 ? d.xd : k == 1 ? d.yd : d.zd;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      r.x[c] = X[nd[c]];
      r.v[c] = U[nd[c]];
    }
  }
  fx::kin_extents(k, sh, r);
  __syncthreads();
  fx::kin_edges(k, sh, 0.5 * dt, r, fx::wide());
  __syncthreads();
  fx::kin_products(k, sh, r);
  __syncthreads();
  fx::kin_terms(k, sh, r);
  __syncthreads();
  fx::kin_accept(sh, r);
  const int others = __syncthreads_or(live && !r.ok);
  const int place = kin_quotients<AUX, TAPE>(d, st, sh, k, e, live && r.ok, FixedSums{sh, r});
  if (TAPE && live) {
    if (r.ok) kin_tape(d, k, e, place, FixedTaped{r});
    if (d.tapeGeoNext && r.ok_x) kin_tape_next(d, k, e, FixedTaped{r});
  }
  if (others) {
    __syncthreads();
    kin_fallback<AUX, TAPE>(d, st, column, e, live && !r.ok, !r.ok_x, dt);
  }
}

// At the start of a taped segment: the first cycle's face diagonals and
// normals on their tapes, by the phases of k_kinematics, which writes later
// cycles' (so a segment's first cycle has the bits it has in mid-segment).
__global__ void __launch_bounds__(3 * kFixedElems) k_tape_geometry(const __grid_constant__ DevDomain d) {
  __shared__ fx::Num column[fx::KS_COUNT * kFixedElems];
  const int E = d.E;
  const int lane = threadIdx.x % kFixedElems, k = threadIdx.x / kFixedElems;
  const int slot = blockIdx.x * kFixedElems + lane;
  const int e = slot < E ? slot : E - 1;
  const fx::Slots sh{column + lane, kFixedElems};
  fx::KinLane r;
  const double* const X = k == 0 ? d.x : k == 1 ? d.y : d.z;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    r.x[c] = LDG(&X[LULESH_IDX(LDG(&d.nodelist[c * E + e]), d.N, d.st)]);
    r.v[c] = 0.0;
  }
  fx::kin_extents(k, sh, r);
  __syncthreads();
  fx::kin_edges(k, sh, 0.0, r, fx::wide());
  __syncthreads();
  fx::kin_products(k, sh, r);
  __syncthreads();
  const bool taken = fx::kin_positions_taken(sh, r);
  const bool live = slot < E;
  double g[12], n[5];
#pragma unroll
  for (int q = 0; q < 12; ++q) g[q] = fx::to_double(r.g[q], -r.s);
#pragma unroll
  for (int f = 0; f < 5; ++f) n[f] = fx::to_double(r.n[f], 64 - (r.all - r.s));
  if (__syncthreads_or(live && !taken)) {
    KinSums sums;
    KinTaped t;
    double v[8] = {};
    kin_fp64(k, RealSlots{reinterpret_cast<double*>(column) + lane, kFixedElems}, r.x, v, 0.0, sums, t);
    if (!taken) {
#pragma unroll
      for (int q = 0; q < 12; ++q) g[q] = t.g[q];
#pragma unroll
      for (int f = 0; f < 5; ++f) n[f] = t.n[f];
    }
  }
  if (!live) return;
  if (d.tapeGeoNext)
#pragma unroll
    for (int f = 0; f < 5; ++f) d.tapeGeoNext[row(48 + 6 * k + f, E, e)] = n[f];
  if (d.tapeDiag)
#pragma unroll
    for (int q = 0; q < 12; ++q) d.tapeDiag[row(3 * q + k, E, e)] = g[q];
}

// ---------------------------------------------------------------------------
// k_material
// ---------------------------------------------------------------------------

// One limiter direction, src/domain.jl:2330-2376, in units of 2 (delv + ptiny):
// hn = 1 / (2 (delv + ptiny)), dm and dp the neighbours' values, mult2 twice
// the limiter's multiplier. The comparisons are made before the quotient, with
// its sign moved to dm and dp, so one product forms the result instead of two
// and a half. `src` reports which value it is (PHI_*), for the adjoint's tape.
__device__ __forceinline__ double monoq_phi(double hn, double dm, double dp, const Params& prm, int& src) {
  const long long sign = __double_as_longlong(hn) & (long long)0x8000000000000000ull;
  dm = __longlong_as_double(__double_as_longlong(dm) ^ sign);
  dp = __longlong_as_double(__double_as_longlong(dp) ^ sign);
  double f = dm + dp;
  src = PHI_MEAN;
  dm *= prm.monoq_mult2;
  dp *= prm.monoq_mult2;
  // the comparisons on the integer keys (fkey), with IEEE's outcomes
  long long kf = fkey(f);
  const long long km = fkey(dm), kp = fkey(dp);
  if (km < kf) { f = dm; kf = km; src = PHI_M; }
  if (kp < kf) { f = dp; src = PHI_P; }
  double phi = f * fabs(hn);
  long long kphi = fkey(phi);
  if (kphi < 0) { phi = 0.0; kphi = 0; src = PHI_ZERO; }
  if (kphi > prm.k_max_slope) { phi = prm.monoq_max_slope; src = PHI_MAX; }
  return phi;
}

// Element whose value one face of the limiter reads (the four BC cases); -1
// for the value 0.
__device__ __forceinline__ int monoq_neighbour(unsigned mask, unsigned bits, unsigned symm, unsigned freeb,
                                               unsigned comm, int idx, int self, int E, bool& bad) {
  const unsigned c = mask & bits;
  if (c == 0u || c == comm) {
    if (idx < 0 || idx >= E) { bad = true; return -1; }
    return idx;
  }
  if (c == symm) return self;
  if (c != freeb) bad = true;
  return -1;
}

// The time constraints of a set of elements: the least Courant candidate (bits
// of a non-negative double) and the largest |vdov| (likewise). The hydro
// constraint dvovmax / (|vdov| + 1e-20) (src/domain.jl:3022-3054) falls with
// |vdov|, and its rounding with it, so the set's least is that of its largest
// |vdov|: one division for the set.
struct Limits {
  unsigned long long courant, rate;
};
__device__ __forceinline__ void merge(Limits& a, unsigned long long courant, unsigned long long rate) {
  a.courant = courant < a.courant ? courant : a.courant;
  a.rate = rate > a.rate ? rate : a.rate;
}
__device__ __forceinline__ void warp_merge(Limits& a) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long c = __shfl_xor_sync(0xffffffffu, a.courant, o);
    const unsigned long long r = __shfl_xor_sync(0xffffffffu, a.rate, o);
    merge(a, c, r);
  }
}
__device__ __forceinline__ double hydro_limit(double rate, const Params& prm) {
  return prm.dvovmax / (rate + 1.e-20);
}
__device__ __forceinline__ void register_limits(const Limits& a, DevState* st, const Params& prm) {
  if (a.courant != kInfBits) atomicMin(&st->acc_courant, a.courant);
  if (a.rate != 0ull) {
    const double h = hydro_limit(__longlong_as_double((long long)a.rate), prm);
    atomicMin(&st->acc_hydro, (unsigned long long)__double_as_longlong(h));
  }
}

// Every thread of the block must call this.
__device__ __forceinline__ void block_limits(Limits a, DevState* st, const Params& prm) {
  __shared__ Limits part[32];
  warp_merge(a);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) part[w] = a;
  __syncthreads();
  if (w == 0) {
    const int nw = blockDim.x >> 5;
    a.courant = l < nw ? part[l].courant : kInfBits;
    a.rate = l < nw ? part[l].rate : 0ull;
    warp_merge(a);
    if (l == 0) register_limits(a, st, prm);
  }
}

// Per-instance limits of an ensemble: a warp whose elements all belong to one
// instance reduces first; a warp straddling two instances (or the ragged
// tail) falls back to one atomic per thread. Every lane must call this.
__device__ __forceinline__ void warp_limits_by_instance(Limits a, int inst, DevState* st, const Params& prm) {
  const unsigned full = 0xffffffffu;
  const int inst0 = __shfl_sync(full, inst, 0);
  if (__all_sync(full, inst == inst0)) {
    warp_merge(a);
    if ((threadIdx.x & 31) == 0) register_limits(a, st + inst0, prm);
  } else {
    register_limits(a, st + inst, prm);
  }
}

// An empty register move the compiler cannot see through: a value passed
// through it must be recomputed from it.
__device__ __forceinline__ void opaque(double& x) { asm volatile("" : "+d"(x)); }

// Bound by FP64 issue (pipe 82 % busy): 0.48 ms per cycle at 150^3 in mid-blast
// (0.71 ms with the limiter and the time constraints formed for every element);
// over a run's first 200 cycles 0.36 ms, 0.75 before.
//
// REGION: threads take elements in region order (d.regOrder) so that a warp
// runs one region's rep count; each element's EOS is evaluated that many times.
template <int MODE, bool AUX, bool ENS, bool TAPE, bool REGION>
__global__ void __launch_bounds__(kMaxElemBlock) k_material(DevDomain d, Params prm) {
  const int E = d.E;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = REGION ? (t < E ? LULESH_IDX(LDG(&d.regOrder[t]), E, d.st) : E) : t;
  // every thread of the block takes part in the dt reduction
  Limits limits = {kInfBits, 0ull};
  const int inst = (ENS && i < E) ? LULESH_IDX(LDG(&d.elemInst[i]), d.ninst, d.st) : 0;
  DevState* const st = d.st + inst;
  // the limiter's neighbours
  bool bad = false;
  int xim = -1, xip = -1, etm = -1, etp = -1, ztm = -1, ztp = -1;
  if (i < E) {
    const unsigned mask = LDG(&d.elemBC[i]);
    // xi-plus: the reference indexes delv_xi[lxip[i]] without +1 (:2349)
    const int ixp = (MODE & 4) ? LDG(&d.lxip[i]) : LDG(&d.lxip[i]) - 1;
    const int Eg = d.Eg;  // neighbour reads may reach the ghost slots of a block-partitioned mesh
    xim = monoq_neighbour(mask, XI_M, XI_M_SYMM, XI_M_FREE, XI_M_COMM, LDG(&d.lxim[i]), i, Eg, bad);
    xip = monoq_neighbour(mask, XI_P, XI_P_SYMM, XI_P_FREE, XI_P_COMM, ixp, i, Eg, bad);
    etm = monoq_neighbour(mask, ETA_M, ETA_M_SYMM, ETA_M_FREE, ETA_M_COMM, LDG(&d.letam[i]), i, Eg, bad);
    etp = monoq_neighbour(mask, ETA_P, ETA_P_SYMM, ETA_P_FREE, ETA_P_COMM, LDG(&d.letap[i]), i, Eg, bad);
    ztm = monoq_neighbour(mask, ZETA_M, ZETA_M_SYMM, ZETA_M_FREE, ZETA_M_COMM, LDG(&d.lzetam[i]), i, Eg, bad);
    ztp = monoq_neighbour(mask, ZETA_P, ZETA_P_SYMM, ZETA_P_FREE, ZETA_P_COMM, LDG(&d.lzetap[i]), i, Eg, bad);
  }
  wait_for_last_kernel();
  const bool live = (i < E) && !step_off(st);
  if (live) {
    unsigned int err = 0u;
    unsigned long long fl = 0ull;  // branch record (TAPE only)
    // ---- calcMonotonicQRegionForElems, src/domain.jl:2322-2513 ----
    const double vdov = d.vdov[i];
    // an expanding element has no viscosity (qlin = qquad = 0), nor has one
    // whose velocity gradients are zero: its limiter is only checked, not formed
    const bool expanding = gt_zero(vdov);
    const double dvxi = d.delv_xi[i], dveta = d.delv_eta[i], dvzeta = d.delv_zeta[i];
    const bool still = is_zero(dvxi) && is_zero(dveta) && is_zero(dvzeta);
    int src0 = PHI_MEAN, src1 = PHI_MEAN, src2 = PHI_MEAN;
    if (bad) err |= ST_BAD_BC;
    // d.tapeMat slot q of this element (TAPE only)
    auto tm = [&](int q, double v) { if (TAPE) d.tapeMat[row(q, E, i)] = v; };
    double phixi = 0.0, phieta = 0.0, phizeta = 0.0;
    if (TAPE || !(expanding || still)) {
      auto at = [](const double* dv, int j) { return j < 0 ? 0.0 : dv[j]; };
      const double xm = at(d.delv_xi, xim), xp = at(d.delv_xi, xip), em = at(d.delv_eta, etm),
                   ep = at(d.delv_eta, etp), zm = at(d.delv_zeta, ztm), zp = at(d.delv_zeta, ztp);
      // the three 1/(2 (delv + ptiny)) from one division
      double hx, hy, hz;
      recip3(fma(2.0, dvxi, 2.e-36), fma(2.0, dveta, 2.e-36), fma(2.0, dvzeta, 2.e-36), hx, hy, hz);
      phixi = monoq_phi(hx, xm, xp, prm, src0);
      phieta = monoq_phi(hy, em, ep, prm, src1);
      phizeta = monoq_phi(hz, zm, zp, prm, src2);
      if (TAPE) {
        // limiter terms per direction: norm, dm/norm, dp/norm
        fl |= (unsigned long long)(src0 | (src1 << 3) | (src2 << 6));
        const double nx = 2.0 * hx, ny = 2.0 * hy, nz = 2.0 * hz;
        tm(0, nx); tm(1, ny); tm(2, nz);
        tm(3, xm * nx); tm(4, em * ny); tm(5, zm * nz);
        tm(6, xp * nx); tm(7, ep * ny); tm(8, zp * nz);
      }
    }

    const double vnew = d.vnew[i];
    const double delvc_in = d.delv[i];

    // ---- applyMaterialPropertiesForElems' clamp, src/domain.jl:2860-2910 ----
    // (the threshold tests of this kernel compare integer keys, fkey)
    double vnewc_in = vnew;
    long long kvn = fkey(vnew);
    bool clamped = false;
    if (prm.has_eosvmin && kvn < prm.k_eosvmin) {
      vnewc_in = prm.eosvmin; kvn = prm.k_eosvmin; clamped = true;
      if (TAPE) fl |= TF_VNEW_MIN;
    }
    if (prm.has_eosvmax && kvn > prm.k_eosvmax) {
      vnewc_in = prm.eosvmax; clamped = true;
      if (TAPE) fl |= TF_VNEW_MAX;
    }
    // 1/vnewc and 1/vchalf (vchalf = vnewc - delvc/2 > 0) from one division
    double inv_vnewc_in, inv_vchalf_in;
    recip2(vnewc_in, fma(delvc_in, -0.5, vnewc_in), inv_vnewc_in, inv_vchalf_in);
    const double inv_vnew = clamped ? 1.0 / vnew : inv_vnewc_in;
    double qlin, qquad;
    const bool inviscid = expanding || (still && !TAPE);
    if (inviscid) {
      qlin = 0.0;
      qquad = 0.0;
      if (TAPE) {
        fl |= TF_QZERO;
#pragma unroll
        for (int q = 9; q < 14; ++q) tm(q, 0.0);
      }
    } else {
      double dxxi = dvxi * d.delx_xi[i];
      double dxeta = dveta * d.delx_eta[i];
      double dxzeta = dvzeta * d.delx_zeta[i];
      if (gt_zero(dxxi)) { dxxi = 0.0; if (TAPE) fl |= TF_DXCLAMP0; }
      if (gt_zero(dxeta)) { dxeta = 0.0; if (TAPE) fl |= TF_DXCLAMP0 << 1; }
      if (gt_zero(dxzeta)) { dxzeta = 0.0; if (TAPE) fl |= TF_DXCLAMP0 << 2; }
      // rho = elemMass / (volo vnew), from the reciprocals of volo and vnew
      const double rho = (LDG(&d.elemMass[i]) * LDG(&d.inv_volo[i])) * inv_vnew;
      const double s1sum = fma(dxxi, 1.0 - phixi, fma(dxeta, 1.0 - phieta, dxzeta * (1.0 - phizeta)));
      const double s2sum = fma(dxxi * dxxi, fma(-phixi, phixi, 1.0),
                               fma(dxeta * dxeta, fma(-phieta, phieta, 1.0), (dxzeta * dxzeta) * fma(-phizeta, phizeta, 1.0)));
      qlin = (-prm.qlc_monoq * rho) * s1sum;
      qquad = (prm.qqc_monoq * rho) * s2sum;
      tm(9, rho); tm(10, qlin); tm(11, qquad); tm(12, s1sum); tm(13, s2sum);
    }
    if (AUX) { d.ql[i] = qlin; d.qq[i] = qquad; }

    // ---- qstop check on the old q, src/domain.jl:2567-2582 ----
    const double q_old_in = d.q[i];
    if (fkey(q_old_in) > prm.k_qstop) err |= ST_QSTOP;

    // ---- applyMaterialPropertiesForElems' volume check ----
    {
      double vc = d.v[i];
      long long kvc = fkey(vc);
      if (prm.has_eosvmin && kvc < prm.k_eosvmin) { vc = prm.eosvmin; kvc = prm.k_eosvmin; }
      if (prm.has_eosvmax && kvc > prm.k_eosvmax) vc = prm.eosvmax;
      if (le_zero(vc)) err |= ST_MATERIAL;
    }

    // ---- evalEOSForElems + calcEnergyForElems + calcSoundSpeedForElems,
    //      src/domain.jl:2617-2857, per element ----
    // The region cost model (LULESH 2.0's rep loop in EvalEOSForElems, which
    // the reference computes in regReps but never applies) evaluates the
    // energy update `reps` times with identical inputs; the inputs pass
    // through an opaque register move each time so no evaluation is folded
    // away, and the last one is kept. Results do not depend on reps.
    const int reps = REGION ? LDG(&d.posReps[t]) : 1;
    const double e_old_in = d.e[i];
    const double p_old_in = d.p[i];
    const double c1s = 2.0 / 3.0;
    // (the reference density is 1 unless the caller sets it)
    auto over_rho0 = [&](double x) { return prm.inv_refdens == 1.0 ? x : x * prm.inv_refdens; };
    double e_out = 0.0, p_out = 0.0, vv_out = 0.0;
    bool compress_out = false;
    // TINY-guarded sound-speed square root (src/domain.jl:2655-2659, 2738-2742)
    auto tiny_sqrt = [&](double ssc, unsigned long long bit) -> double {
      // ssc <= 0.111111e-36 (a positive threshold: the signed bit patterns order)
      if (__double_as_longlong(ssc) <= 0x3842E7910CC4BCABll) { if (TAPE) fl |= bit; return 0.333333e-18; }
      return ssc * rsqrt(ssc);
    };
    // Without viscosity q is s 0 + 0 for the sound speed s of (e, p, v): zero, and s
    // not formed, where s is certainly finite (all three below 2^300). The EOS is
    // FP64-bound, and most of a blast's elements are at rest: 2139 -> 2098 us per
    // cycle at 150^3, 23.3 -> 20.8 ms at 256^3 with region repetitions.
    auto no_viscosity = [&](double e, double p, double v) {
      const unsigned top = fx::umax(fx::umax((unsigned)__double2hiint(e) & 0x7fffffffu, (unsigned)__double2hiint(p) & 0x7fffffffu),
                                    (unsigned)__double2hiint(v) & 0x7fffffffu);
      return !TAPE && inviscid && top < (1023u + 300u) << 20 && prm.inv_refdens == 1.0;
    };
#pragma unroll 1
    for (int rep = 0; rep < reps; ++rep) {
    double delvc = delvc_in, e_old = e_old_in, p_old = p_old_in, q_old = q_old_in, vnewc = vnewc_in;
    if (REGION) { opaque(delvc); opaque(e_old); opaque(p_old); opaque(q_old); opaque(vnewc); }
    const double vchalf = fma(delvc, -0.5, vnewc);
    // the rep passes form the reciprocals anew from their opaque inputs
    double inv_vnewc = inv_vnewc_in, inv_vchalf = inv_vchalf_in;
    if (REGION) recip2(vnewc, vchalf, inv_vnewc, inv_vchalf);
    // compression = 1/vnewc - 1 and compHalfStep = 1/vchalf - 1 enter only as
    // bvc = c1s (1 + compression) and bvc_half = c1s (1 + compHalfStep):
    // bv and bvh are those factors over c1s for the branch taken
    const long long kv = fkey(vnewc);
    const bool at_vmin = prm.has_eosvmin && kv <= prm.k_eosvmin;  // eosvmin != 0 && vnewc <= eosvmin
    const bool vmax_hit = kv >= prm.k_eosvmax;                     // vnewc >= eosvmax
    const bool at_vmax = prm.has_eosvmax && vmax_hit;
    double bv = inv_vnewc, bvh = inv_vchalf;
    if (at_vmin) { bvh = bv; if (TAPE) fl |= TF_HALF_EQ_COMP; }
    if (at_vmax) {
      p_old = 0.0; bv = 1.0; bvh = 1.0;
      if (TAPE) fl |= TF_VMAX_HIT;
    }
    // calcPressureForElems (src/domain.jl:2585-2614) for one element; the
    // cut / pmin outcomes go to the tape bits given
    auto pressure = [&](double enew, double bvc, unsigned long long cut_bit, unsigned long long min_bit) -> double {
      double pn = bvc * enew;
      if (abs_lt(pn, prm.p_cut)) { pn = 0.0; if (TAPE) fl |= cut_bit; }
      if (vmax_hit) pn = 0.0;
      if (fkey(pn) < prm.k_pmin) { pn = prm.pmin; if (TAPE) fl |= min_bit; }
      return pn;
    };
    const double pq_old = p_old + q_old;
    // 0.5 delvc and pHalfStep + q_new serve both energy updates (the negated
    // and scaled forms are exact, so the values are those of separate products)
    const double hdv = 0.5 * delvc;
    double e_new = fma(-hdv, pq_old, e_old);
    if (fkey(e_new) < prm.k_emin) { e_new = prm.emin; if (TAPE) fl |= TF_E1_MIN; }
    const double bvc_half = c1s * bvh;
    const double pHalfStep = pressure(e_new, bvc_half, TF_PH_CUT, TF_PH_MIN);
    // vhalf = 1 / (1 + compHalfStep): vchalf, vnewc or 1 by the branch taken
    const double vhalf = at_vmax ? 1.0 : at_vmin ? vnewc : vchalf;
    const bool compress = !gt_zero(delvc);   // delvc <= 0 (non-NaN)
    if (TAPE && compress) fl |= TF_COMPRESS;
    tm(14, bv); tm(15, bvh); tm(16, e_new); tm(17, pHalfStep); tm(18, vhalf);
    double q_new = 0.0;
    if (compress && !no_viscosity(e_new, pHalfStep, vhalf)) {
      // vhalf^2 bvc_half = c1s vhalf, 1 + compHalfStep being 1/vhalf in each branch
      const double ssc = over_rho0(fma(c1s, e_new, (c1s * vhalf) * pHalfStep));
      const double s1 = tiny_sqrt(ssc, TF_S1_TINY);
      q_new = fma(s1, qlin, qquad);
      tm(19, s1); tm(28, ssc);
    } else {
      tm(19, 0.0); tm(28, 0.0);
    }
    tm(20, q_new);
    const double sh = pHalfStep + q_new;
    e_new = fma(hdv, fma(3.0, pq_old, -4.0 * sh), e_new);
    if (abs_lt(e_new, prm.e_cut)) { e_new = 0.0; if (TAPE) fl |= TF_E2_CUT; }
    if (fkey(e_new) < prm.k_emin) { e_new = prm.emin; if (TAPE) fl |= TF_E2_MIN; }
    const double bvc = c1s * bv;
    double p_new = pressure(e_new, bvc, TF_PN1_CUT, TF_PN1_MIN);
    // vnewc^2 bvc = c1s vnewc, bvc being c1s/vnewc, except where vnewc >= eosvmax
    double vv_bvc = c1s * vnewc;
    if (at_vmax) vv_bvc *= vnewc;
    tm(21, e_new); tm(22, p_new);
    double q_tilde = 0.0;
    if (compress && !no_viscosity(e_new, p_new, vv_bvc)) {
      const double ssc = over_rho0(fma(c1s, e_new, vv_bvc * p_new));
      const double s2 = tiny_sqrt(ssc, TF_S2_TINY);
      q_tilde = fma(s2, qlin, qquad);
      tm(23, s2); tm(29, ssc);
    } else {
      tm(23, 0.0); tm(29, 0.0);
    }
    tm(24, q_tilde);
    e_new = fma(-(fma(7.0, pq_old, -8.0 * sh) + (p_new + q_tilde)), delvc * (1.0 / 6.0), e_new);
    if (abs_lt(e_new, prm.e_cut)) { e_new = 0.0; if (TAPE) fl |= TF_E3_CUT; }
    if (fkey(e_new) < prm.k_emin) { e_new = prm.emin; if (TAPE) fl |= TF_E3_MIN; }
    p_new = pressure(e_new, bvc, TF_PN2_CUT, TF_PN2_MIN);
    e_out = e_new; p_out = p_new; vv_out = vv_bvc; compress_out = compress;
    }  // rep loop
    const double e_new = e_out, p_new = p_out, vv_bvc = vv_out;
    const bool compress = compress_out;
    double q_new = 0.0;
    // the last q evaluation and the sound speed share one expression
    const double ssc3 = over_rho0(fma(c1s, e_new, vv_bvc * p_new));
    const double ss_new = tiny_sqrt(ssc3, TF_SS_TINY);
    tm(25, e_new); tm(26, p_new); tm(27, ss_new); tm(30, ssc3);
    if (compress) {
      q_new = fma(ss_new, qlin, qquad);
      if (abs_lt(q_new, prm.q_cut)) { q_new = 0.0; if (TAPE) fl |= TF_Q_CUT; }
    }
    d.p[i] = p_new;
    d.e[i] = e_new;
    d.q[i] = q_new;
    d.ss[i] = ss_new;

    // ---- updateVolumesForElems, src/domain.jl:2912-2930 ----
    double tmpV = vnew;
    if (abs_lt(tmpV - 1.0, prm.v_cut)) { tmpV = 1.0; if (TAPE) fl |= TF_V_SNAP; }
    d.v[i] = tmpV;
    if (le_zero(tmpV)) err |= ST_UPDATE;

    // ---- Courant and hydro constraints, src/domain.jl:2964-3054 ----
    // A candidate that is certainly above the least so far is not formed (what it
    // compares with only falls).
    double dtc = __longlong_as_double((long long)kInfBits), dth = dtc;
    if (!is_zero(vdov)) {
      const double arealg = d.arealg[i];
      const unsigned long long rate = (unsigned long long)__double_as_longlong(vdov) & 0x7FFFFFFFFFFFFFFFull;
      if (rate <= kInfBits) limits.rate = rate;  // (a NaN constrains nothing)
      bool skip = false;
      if (!TAPE) {
        const double least = __longlong_as_double((long long)*(volatile unsigned long long*)&st->acc_courant);
        skip = courant_above(arealg, ss_new, vdov, least, prm.qqc8);
      }
      if (!skip) {
        double dtf = ss_new * ss_new;
        if (lt_zero(vdov)) dtf = fma(prm.qqc2x64 * (arealg * arealg), vdov * vdov, dtf);
        dtc = arealg * rsqrt(dtf);
        limits.courant = (unsigned long long)__double_as_longlong(dtc);
      }
      if (TAPE) dth = hydro_limit(fabs(vdov), prm);
    }
    if (TAPE) {
      d.tapeFlags[i] |= fl;  // k_kinematics stored the face bits of this cycle
      d.tapeDtc[i] = dtc;
      d.tapeDth[i] = dth;
    }
    if (err) atomicOr(&st->status, err);
  }
  if (ENS) warp_limits_by_instance(limits, inst, d.st, prm);
  else block_limits(limits, d.st, prm);
}

// ---------------------------------------------------------------------------
// Halo copies of a block-partitioned mesh (the single-GPU form of commSBN and
// commMonoQ, src/comm.jl:776, 1127): each ghost slot takes the value of the
// corner force or element its owning block computed.
// ---------------------------------------------------------------------------
__global__ void k_halo_corners(DevDomain d) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const int base = 8 * d.E;
  if (g >= d.nCornerSlot - base) return;
  wait_for_last_kernel();
  if (step_off(d.st)) return;
  const int s = LULESH_IDX(LDG(&d.haloCornerSrc[g]), base, d.st);
  d.fcx[base + g] = d.fcx[s];
  d.fcy[base + g] = d.fcy[s];
  d.fcz[base + g] = d.fcz[s];
}

__global__ void k_halo_delv(DevDomain d) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= d.Eg - d.E) return;
  wait_for_last_kernel();
  if (step_off(d.st)) return;
  const int s = LULESH_IDX(LDG(&d.haloDelvSrc[g]), d.E, d.st);
  d.delv_xi[d.E + g] = d.delv_xi[s];
  d.delv_eta[d.E + g] = d.delv_eta[s];
  d.delv_zeta[d.E + g] = d.delv_zeta[s];
}

// ---------------------------------------------------------------------------
// k_time_increment (device run loop): one thread per problem
// ---------------------------------------------------------------------------
__global__ void k_time_increment(DevState* st, int n, Params prm) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  wait_for_last_kernel();
  if (k < n) advance_time(st + k, prm);
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
void launch_tape_geometry(const DevDomain& d, cudaStream_t s) {
  k_tape_geometry<<<(d.E + kFixedElems - 1) / kFixedElems, 3 * kFixedElems, 0, s>>>(d);
}

void launch_force(const DevDomain& d, const Params& prm, cudaStream_t s, bool time) {
  const int bs = 3 * kFixedElems;
  const int grid = (d.E + kFixedElems - 1) / kFixedElems;
  const int with = grid + time_blocks(d.ninst);
#define LULESH_FORCE(M)                                                            \
  (time ? (d.elemInst ? launch(k_force<M, true, false, true>, with, bs, s, d, prm)  \
                      : launch(k_force<M, false, false, true>, with, bs, s, d, prm)) \
   : d.elemInst ? launch(k_force<M, true, false, false>, grid, bs, s, d, prm)       \
   : d.tapeGeo  ? launch(k_force<M, false, true, false>, grid, bs, s, d, prm)       \
                : launch(k_force<M, false, false, false>, grid, bs, s, d, prm))
  switch (d.mode & 3) {
    case 0: LULESH_FORCE(0); break;
    case 1: LULESH_FORCE(1); break;
    case 2: LULESH_FORCE(2); break;
    default: LULESH_FORCE(3); break;
  }
#undef LULESH_FORCE
}

void launch_node(const DevDomain& d, const Params& prm, bool aux, const Tuning& t, cudaStream_t s) {
  if (d.haloCornerSrc) {
    const int n = d.nCornerSlot - 8 * d.E;
    launch(k_halo_corners, (n + 255) / 256, 256, s, d);
  }
  const int bs = threads_per_block(d.N, t.node, kNodeBlock);
  const int grid = (d.N + bs - 1) / bs;
  if (d.nodeInst) launch(k_node<false, true>, grid, bs, s, d, prm);
  else if (aux) launch(k_node<true, false>, grid, bs, s, d, prm);
  else launch(k_node<false, false>, grid, bs, s, d, prm);
}

void launch_kinematics(const DevDomain& d, const Params& prm, bool aux, cudaStream_t s) {
  const int bs = 3 * kFixedElems;
  const int grid = (d.E + kFixedElems - 1) / kFixedElems;
  if (d.elemInst) launch(k_kinematics<false, true, false>, grid, bs, s, d, prm);
  else if (d.tapeFlags) launch(k_kinematics<false, false, true>, grid, bs, s, d, prm);
  else if (aux) launch(k_kinematics<true, false, false>, grid, bs, s, d, prm);
  else launch(k_kinematics<false, false, false>, grid, bs, s, d, prm);
}

void launch_material(const DevDomain& d, const Params& prm, bool aux, const Tuning& t, cudaStream_t s) {
  if (d.haloDelvSrc) {
    const int n = d.Eg - d.E;
    launch(k_halo_delv, (n + 255) / 256, 256, s, d);
  }
  const int bs = threads_per_block(d.E, t.mat, kMatBlock);
  const int grid = (d.E + bs - 1) / bs;
  const bool fix = (d.mode & 4) != 0;
  const bool region = d.regOrder != nullptr;
#define LULESH_MAT(M, AUX, ENS, TAPE, REGION) launch(k_material<M, AUX, ENS, TAPE, REGION>, grid, bs, s, d, prm)
  if (d.elemInst) {
    if (fix) LULESH_MAT(4, false, true, false, false);
    else LULESH_MAT(0, false, true, false, false);
  } else if (d.tapeFlags) {
    if (fix) LULESH_MAT(4, false, false, true, false);
    else LULESH_MAT(0, false, false, true, false);
  } else if (region) {
    if (fix) { if (aux) LULESH_MAT(4, true, false, false, true); else LULESH_MAT(4, false, false, false, true); }
    else { if (aux) LULESH_MAT(0, true, false, false, true); else LULESH_MAT(0, false, false, false, true); }
  } else if (fix) {
    if (aux) LULESH_MAT(4, true, false, false, false);
    else LULESH_MAT(4, false, false, false, false);
  } else {
    if (aux) LULESH_MAT(0, true, false, false, false);
    else LULESH_MAT(0, false, false, false, false);
  }
#undef LULESH_MAT
}

// One problem's step state to and from the device by kernels of the cycle's
// chain: a copy of 96 bytes goes through the copy engine, which waits for the
// kernel before it to flush and holds up the one after it.
__global__ void k_put_state(DevState* st, DevState value) {
  wait_for_last_kernel();
  if (threadIdx.x == 0) *st = value;
}
__global__ void k_get_state(const DevState* st, DevState* host) {
  wait_for_last_kernel();
  if (threadIdx.x == 0) *host = *st;
}
void launch_put_state(DevState* st, const DevState& value, cudaStream_t s) { launch(k_put_state, 1, 32, s, st, value); }
void launch_get_state(const DevState* st, DevState* pinned, cudaStream_t s) {
  launch(k_get_state, 1, 32, s, st, pinned);
}

void launch_time_increment(DevState* st, int n, const Params& prm, cudaStream_t s) {
  launch(k_time_increment, (n + 127) / 128, 128, s, st, n, prm);
}

}  // namespace lulesh
