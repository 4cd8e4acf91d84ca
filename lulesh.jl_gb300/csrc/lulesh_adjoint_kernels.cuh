// Reverse-mode adjoint kernels of the LagrangeLeapFrog step.
//
// Each kernel is the hand-written transpose (vector-Jacobian product) of one
// forward kernel of lulesh_kernels.cu, in the same formulation (Walsh
// coefficients, face-diagonal cross products, edge sums). Forward values are
// recomputed from the cycle's tape (start state, end positions/velocities,
// accelerations, kinematics outputs); every branch (cut-offs, clamps, limiter
// cases, the characteristic-length face, velocity snaps) is read from the
// tape the taping forward kernels wrote, so the derivative is that of the
// branches actually taken. Node sums are transposed into per-corner buffers
// and gathered back in nodeElemCornerList order; neighbour reads of the Q
// limiter are transposed into per-face slots and gathered through an inverse
// neighbour list: no atomics, so gradients are bitwise reproducible.
#pragma once

#include <climits>

#include "lulesh_device.cuh"
#include "lulesh_fixed_force.cuh"
#include "lulesh_kernels.h"
#include "lulesh_launch.cuh"

namespace lulesh {

constexpr int kAdjBlock = 128;

// Scalars of one recorded cycle: timeIncrement!'s inputs and output, and the
// elements that attained the Courant and hydro minima (INT_MAX: none).
struct CycleRec {
  double time_prev, dt_prev, dtc_in, dth_in, dt;
  long long cycle_prev;
  int active_c, active_h, argmin_c, argmin_h;
};

// Adjoints of the Domain scalars carried from cycle to cycle.
struct AdjScal {
  double Ltime, Ldt, Ldtc, Ldth;
};

// The 11 state fields (x y z xd yd zd e p q v ss) of one stored state.
struct StateSet {
  double* f[11];
};

struct AdjDev {
  int E, N;
  // constants of the problem
  const int* nodelist;        // [8][E]
  const int* nodeElemStart;   // N+1
  const int* cornerList;      // 8E, values c*E + e
  const unsigned char* nodeBC;
  const double *inv_nodalMass, *volo, *inv_volo, *elemMass;
  const unsigned* elemBC;
  const int *lxim, *lxip, *letam, *letap, *lzetam, *lzetap;
  const int *nbStart, *nbList;  // inverse neighbour lists (entries slot*E + j)
  // cycle start state S0 and end positions/velocities S1
  const double *x0, *y0, *z0, *xd0, *yd0, *zd0, *e0, *p0, *q0, *v0, *ss0;
  const double *x1, *y1, *z1, *xd1, *yd1, *zd1, *p1, *q1;
  // tape of the cycle
  const double *ax, *ay, *az;                 // accelerations (N)
  const double *vnew, *delv, *arealg, *vdov;  // kinematics outputs (E)
  const double *dvl[3], *dxl[3];              // delv_{xi,eta,zeta}, delx_{xi,eta,zeta}
  const unsigned long long* flags;
  const double* geo;                          // [66][E] force-kernel tape (dv, hms, S, N)
  const double* diag0;                        // [36][E] face diagonals at the run's start (first cycle)
  const double* kin;                          // [90][E] kinematics-kernel tape
  const double* mat;                          // [31][E] material-kernel tape
  // adjoints of the state (in place: S1 on entry, S0 on exit)
  double *lx, *ly, *lz, *lxd, *lyd, *lzd;     // N
  double *le, *lp, *lq, *lss, *lv;            // E
  // adjoints of intermediate quantities
  double *lfx, *lfy, *lfz;                    // N
  double *lvnew, *ldelv, *larealg, *lvdov;    // E
  double *ldv[3], *ldx[3];                    // E
  double* lnb;                                // [6][E]: limiter neighbour slots
  double *cX, *cV;                            // [3][8][E] kinematics corner buffers
  double *fX, *fV;                            // [3][8][E] force corner buffers: the first cycle's position
                                              // transpose; each cycle's hourglass velocity corners
  double *part_dt, *part_dtn, *part_hg;       // per-block partial sums (kinematics, node; hourglass over the cycles)
  double *sLdv, *sLhm;                        // [3][8][E], [3][4][E]: hourglass -> geometry
  double* sLU;                                // [5][3][E]: the stress force's face terms (hourglass -> geometry)
};

// Deterministic block sum (fixed tree order); thread 0 writes the block's sum.
__device__ __forceinline__ void block_sum_to(double v, double* out) {
  __shared__ double sh[kAdjBlock];
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int s = kAdjBlock / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[blockIdx.x] = sh[0];
}

struct V3 {
  double x, y, z;
};
__device__ __forceinline__ V3 v3(double x, double y, double z) { return V3{x, y, z}; }
__device__ __forceinline__ V3 vcross(const V3& a, const V3& b) {
  V3 c;
  cross(a.x, a.y, a.z, b.x, b.y, b.z, c.x, c.y, c.z);
  return c;
}
__device__ __forceinline__ void vadd(V3& y, const V3& x) { y.x += x.x; y.y += x.y; y.z += x.z; }

// Resolved limiter neighbour: the element whose delv is read (self for a
// symmetry face or the reference's self-reading xi-plus index), -1 for a free
// face.
__device__ __forceinline__ int limiter_index(unsigned mask, unsigned bits, unsigned symm, unsigned freeb,
                                             unsigned comm, int idx, int self, int E) {
  const unsigned c = mask & bits;
  if (c == 0u || c == comm) return (idx >= 0 && idx < E) ? idx : -1;
  if (c == symm) return self;
  return -1;
}

// ---------------------------------------------------------------------------
// ka_material: transpose of k_material (Q limiter, EOS, volume update,
// Courant and hydro candidates).
// ---------------------------------------------------------------------------
template <int MODE>
__global__ void __launch_bounds__(kAdjBlock, 4) ka_material(AdjDev a, Params prm, double irho0, const CycleRec* rec,
                                                          const AdjScal* sc) {
  const int E = a.E;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= E) return;
  wait_for_last_kernel();
  // the cycle's Courant/hydro minima pass their adjoint to the element that
  // attained them
  const int argmin_c = rec->argmin_c, argmin_h = rec->argmin_h;
  const double lam_c = rec->active_c ? sc->Ldtc : 0.0, lam_h = rec->active_h ? sc->Ldth : 0.0;
  const unsigned long long fl = a.flags[i];
  const unsigned mask = a.elemBC[i];
  // neighbour resolution exactly as the forward kernel
  int im[3], ip[3];
  im[0] = limiter_index(mask, XI_M, XI_M_SYMM, XI_M_FREE, XI_M_COMM, a.lxim[i], i, E);
  ip[0] = limiter_index(mask, XI_P, XI_P_SYMM, XI_P_FREE, XI_P_COMM, (MODE & 4) ? a.lxip[i] : a.lxip[i] - 1, i, E);
  im[1] = limiter_index(mask, ETA_M, ETA_M_SYMM, ETA_M_FREE, ETA_M_COMM, a.letam[i], i, E);
  ip[1] = limiter_index(mask, ETA_P, ETA_P_SYMM, ETA_P_FREE, ETA_P_COMM, a.letap[i], i, E);
  im[2] = limiter_index(mask, ZETA_M, ZETA_M_SYMM, ZETA_M_FREE, ZETA_M_COMM, a.lzetam[i], i, E);
  ip[2] = limiter_index(mask, ZETA_P, ZETA_P_SYMM, ZETA_P_FREE, ZETA_P_COMM, a.lzetap[i], i, E);

  // forward values from the material kernel's tape (slots: see tapeMat)
  auto tm = [&](int q) { return a.mat[row(q, E, i)]; };
  double self[3], norm[3], tdm[3], tdp[3], phi[3], delx[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    self[d] = a.dvl[d][i];
    norm[d] = tm(d);
    tdm[d] = tm(3 + d);  // minus neighbour's delv * norm
    tdp[d] = tm(6 + d);  // plus neighbour's delv * norm
    const int src = (int)((fl >> (3 * d)) & 7ull);
    phi[d] = src == PHI_MEAN ? 0.5 * (tdm[d] + tdp[d])
           : src == PHI_M ? tdm[d] * prm.monoq_limiter_mult
           : src == PHI_P ? tdp[d] * prm.monoq_limiter_mult
           : src == PHI_ZERO ? 0.0 : prm.monoq_max_slope;
    delx[d] = a.dxl[d][i];
  }
  const double vdov = a.vdov[i], vnew = a.vnew[i];
  const double delvc = a.delv[i], arealg = a.arealg[i];
  const bool vmin_c = (fl & TF_VNEW_MIN) != 0, vmax_c = (fl & TF_VNEW_MAX) != 0;
  const double vnewc = vmin_c ? prm.eosvmin : vmax_c ? prm.eosvmax : vnew;
  const bool vmax_hit = (fl & TF_VMAX_HIT) != 0, half_eq = (fl & TF_HALF_EQ_COMP) != 0;
  // bv = 1 + compression and bvh = 1 + compHalfStep as the forward formed
  // them: 1/vnewc and 1/vchalf on the branches where they are reciprocals
  const double bv = tm(14), bvh = tm(15);
  const double inv_vnewc = vmax_hit ? 1.0 / vnewc : bv;
  const double inv_vnew = (vnewc == vnew) ? inv_vnewc : 1.0 / vnew;
  const double inv_vchalf = (vmax_hit || half_eq) ? 0.0 : bvh;
  const bool qzero = (fl & TF_QZERO) != 0;
  double dx[3] = {0.0, 0.0, 0.0};
  const double rho = tm(9), qlin = tm(10), qquad = tm(11), s1sum = tm(12), s2sum = tm(13);
  if (!qzero) {
#pragma unroll
    for (int d = 0; d < 3; ++d) dx[d] = (fl & (TF_DXCLAMP0 << d)) ? 0.0 : self[d] * delx[d];
  }
  const double p_old = vmax_hit ? 0.0 : a.p0[i], q_old = a.q0[i];
  const double c1s = 2.0 / 3.0;  // irho0 = 1 / refdens
  const double pq = p_old + q_old;
  const bool e1min = (fl & TF_E1_MIN) != 0;
  const double e1 = tm(16), pH = tm(17), vhalf = tm(18);
  const double bvc_h = c1s * bvh;
  const bool pH_on = !vmax_hit && !(fl & (TF_PH_CUT | TF_PH_MIN));
  const bool comp = (fl & TF_COMPRESS) != 0;
  const bool s1t = (fl & TF_S1_TINY) != 0, s2t = (fl & TF_S2_TINY) != 0, sst = (fl & TF_SS_TINY) != 0;
  // each square root s = sqrt(c) comes with h = 0.5 / s = 0.5 rsqrt(c)
  const double s1 = tm(19), qn1 = tm(20);
  const double h1 = (comp && !s1t) ? 0.5 * rsqrt(tm(28)) : 0.0;
  const bool e2fix = (fl & (TF_E2_CUT | TF_E2_MIN)) != 0;
  const double k2 = fma(3.0, pq, -4.0 * (pH + qn1));
  const double e2 = tm(21), pn1 = tm(22);
  const double bvc = c1s * bv;
  const bool pn1_on = !vmax_hit && !(fl & (TF_PN1_CUT | TF_PN1_MIN));
  const double vv_bvc = (vnewc * vnewc) * bvc;
  const double s2 = tm(23), qt = tm(24);
  const double h2 = (comp && !s2t) ? 0.5 * rsqrt(tm(29)) : 0.0;
  const double k3 = fma(7.0, pq, -8.0 * (pH + qn1)) + (pn1 + qt);
  const bool e3fix = (fl & (TF_E3_CUT | TF_E3_MIN)) != 0;
  const double e3 = tm(25), pn2 = tm(26), ss = tm(27);
  const bool pn2_on = !vmax_hit && !(fl & (TF_PN2_CUT | TF_PN2_MIN));
  const double hs = sst ? 0.0 : 0.5 * rsqrt(tm(30));

  // ---------------- reverse ----------------
  double Le3 = a.le[i], Lpn2 = a.lp[i], Lq = a.lq[i], Lss = a.lss[i], Lv1 = a.lv[i];
  double Lvnew = 0.0, Larealg = 0.0, Lvdov = 0.0, Ldelvc = 0.0;
  // Courant and hydro candidates (only the arg-min element carries a seed)
  if (i == argmin_c && vdov != 0.0) {
    const double qqc2 = (64.0 * prm.qqc) * prm.qqc;
    double dtf = ss * ss;
    if (vdov < 0.0) dtf = fma(qqc2 * (arealg * arealg), vdov * vdov, dtf);
    const double rs = rsqrt(dtf);
    Larealg += lam_c * rs;
    const double Ldtf = lam_c * arealg * (-0.5) * rs * rs * rs;
    Lss += 2.0 * ss * Ldtf;
    if (vdov < 0.0) {
      Larealg += Ldtf * 2.0 * qqc2 * arealg * vdov * vdov;
      Lvdov += Ldtf * 2.0 * qqc2 * arealg * arealg * vdov;
    }
  }
  if (i == argmin_h && vdov != 0.0) {
    const double den = fabs(vdov) + 1.e-20;
    Lvdov += lam_h * (-prm.dvovmax / (den * den)) * (vdov < 0.0 ? -1.0 : 1.0);
  }
  if (!(fl & TF_V_SNAP)) Lvnew += Lv1;
  double Lqlin = 0.0, Lqquad = 0.0;
  // final q = ss*qlin + qquad
  if (comp && !(fl & TF_Q_CUT)) { Lss += Lq * qlin; Lqlin += Lq * ss; Lqquad += Lq; }
  double Lvv = 0.0, Lbvc = 0.0, Le2 = 0.0, Lpn1 = 0.0, Lpq = 0.0, LpH = 0.0, Lqn1 = 0.0, Lqt = 0.0;
  // ss = sqrt(ssc3)
  if (!sst) {
    const double Lssc = Lss * hs * irho0;
    Le3 += Lssc * c1s;
    Lvv += Lssc * pn2;
    Lpn2 += Lssc * vv_bvc;
  }
  if (pn2_on) { Lbvc += Lpn2 * e3; Le3 += Lpn2 * bvc; }
  if (!e3fix) {
    Le2 += Le3;
    const double Lk = -Le3 * delvc * (1.0 / 6.0);
    Ldelvc += -Le3 * k3 * (1.0 / 6.0);
    Lpq += 7.0 * Lk; LpH += -8.0 * Lk; Lqn1 += -8.0 * Lk; Lpn1 += Lk; Lqt += Lk;
  }
  if (comp) {
    Lqlin += Lqt * s2; Lqquad += Lqt;
    if (!s2t) {
      const double Lssc = Lqt * qlin * h2 * irho0;
      Le2 += Lssc * c1s;
      Lvv += Lssc * pn1;
      Lpn1 += Lssc * vv_bvc;
    }
  }
  double Lvnewc = 2.0 * vnewc * bvc * Lvv;
  Lbvc += Lvv * (vnewc * vnewc);
  if (pn1_on) { Lbvc += Lpn1 * e2; Le2 += Lpn1 * bvc; }
  double Le1 = 0.0;
  if (!e2fix) {
    Le1 += Le2;
    Ldelvc += Le2 * 0.5 * k2;
    Lpq += Le2 * 1.5 * delvc;
    LpH += -2.0 * delvc * Le2;
    Lqn1 += -2.0 * delvc * Le2;
  }
  double Lchs = 0.0, Lbvch = 0.0;
  if (comp) {
    Lqlin += Lqn1 * s1; Lqquad += Lqn1;
    if (!s1t) {
      const double Lssc = Lqn1 * qlin * h1 * irho0;
      Le1 += Lssc * c1s;
      const double Lvhalf = Lssc * 2.0 * vhalf * bvc_h * pH;
      Lbvch += Lssc * (vhalf * vhalf) * pH;
      LpH += Lssc * (vhalf * vhalf) * bvc_h;
      Lchs += -Lvhalf * vhalf * vhalf;
    }
  }
  if (pH_on) { Lbvch += LpH * e1; Le1 += LpH * bvc_h; }
  Lchs += Lbvch * c1s;
  double Le_old = 0.0;
  if (!e1min) {
    Le_old += Le1;
    Ldelvc += -0.5 * pq * Le1;
    Lpq += -0.5 * delvc * Le1;
  }
  double Lcomp = Lbvc * c1s;
  const double Lp_old = vmax_hit ? 0.0 : Lpq;
  const double Lq_old = Lpq;
  if (!vmax_hit) {
    if (half_eq) Lcomp += Lchs;
    else {
      const double Lvch = -Lchs * (inv_vchalf * inv_vchalf);
      Lvnewc += Lvch;
      Ldelvc += -0.5 * Lvch;
    }
    Lvnewc += -Lcomp * (inv_vnewc * inv_vnewc);
  }
  if (!vmin_c && !vmax_c) Lvnew += Lvnewc;
  // qlin / qquad
  double Lself[3] = {0.0, 0.0, 0.0}, Ldx[3] = {0.0, 0.0, 0.0};
  double Lphi[3] = {0.0, 0.0, 0.0};
  if (!qzero) {
    const double Lrho = Lqlin * (-prm.qlc_monoq) * s1sum + Lqquad * prm.qqc_monoq * s2sum;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double Ldxd = Lqlin * (-prm.qlc_monoq * rho) * (1.0 - phi[d]) +
                          Lqquad * (prm.qqc_monoq * rho) * 2.0 * dx[d] * fma(-phi[d], phi[d], 1.0);
      Lphi[d] = Lqlin * (prm.qlc_monoq * rho) * dx[d] + Lqquad * (-prm.qqc_monoq * rho) * dx[d] * dx[d] * 2.0 * phi[d];
      if (!(fl & (TF_DXCLAMP0 << d))) { Lself[d] += Ldxd * delx[d]; Ldx[d] += Ldxd * self[d]; }
    }
    Lvnew += -Lrho * rho * inv_vnew;
  }
  // limiter
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int src = (int)((fl >> (3 * d)) & 7ull);
    double Ldm = 0.0, Ldp = 0.0;
    if (qzero) {  // the limiter was not used
      a.lnb[row(2 * d, E, i)] = 0.0;
      a.lnb[row(2 * d + 1, E, i)] = 0.0;
      a.ldv[d][i] = 0.0;
      a.ldx[d][i] = 0.0;
      continue;
    }
    if (src == PHI_MEAN) { Ldm = 0.5 * Lphi[d]; Ldp = 0.5 * Lphi[d]; }
    else if (src == PHI_M) Ldm = prm.monoq_limiter_mult * Lphi[d];
    else if (src == PHI_P) Ldp = prm.monoq_limiter_mult * Lphi[d];
    const double Lm = Ldm * norm[d], Lp = Ldp * norm[d];
    // norm = 1/(self + ptiny): d(mv norm)/dself = -(mv norm) norm
    Lself[d] += -fma(Ldm, tdm[d], Ldp * tdp[d]) * norm[d];
    double sm = 0.0, sp = 0.0;
    if (im[d] == i) Lself[d] += Lm; else if (im[d] >= 0) sm = Lm;
    if (ip[d] == i) Lself[d] += Lp; else if (ip[d] >= 0) sp = Lp;
    a.lnb[row(2 * d, E, i)] = sm;
    a.lnb[row(2 * d + 1, E, i)] = sp;
    a.ldv[d][i] = Lself[d];
    a.ldx[d][i] = Ldx[d];
  }
  a.lvdov[i] = Lvdov;
  a.lvnew[i] = Lvnew;
  a.ldelv[i] = Ldelvc;
  a.larealg[i] = Larealg;
  // adjoints of the cycle's start state from the material update
  a.le[i] = Le_old;
  a.lp[i] = Lp_old;
  a.lq[i] = Lq_old;
  a.lss[i] = 0.0;
  a.lv[i] = 0.0;
}

// Transpose of walsh1: adds dL/dv of the 8 corner values for the adjoints
// Lw of the three coefficients (through the body diagonals, 14 adds).
template <class T>
__device__ __forceinline__ void walsh1_t(const T Lw[3], T L[8]) {
  const T p = Lw[0] + Lw[2], q = Lw[2] - Lw[0];
  const T La = p + Lw[1], Lb = p - Lw[1], Lc = q + Lw[1], Ld = q - Lw[1];
  L[6] += La; L[0] -= La;
  L[5] += Lb; L[3] -= Lb;
  L[7] += Lc; L[1] -= Lc;
  L[4] += Ld; L[2] -= Ld;
}

// Transpose of the hourglass mode transform: out[n] = sum_m gamma[n][m] t[m]
// (12 adds).
template <class T>
__device__ __forceinline__ void walsh_modes_t(const T t[4], T out[8]) {
  const T cm = t[2] - t[3], cp = t[2] + t[3];
  const T s = t[0] + t[1], d = t[0] - t[1];
  out[0] = s + cm; out[1] = d - cm; out[2] = cm - s; out[3] = -d - cm;
  out[4] = cp - s; out[5] = -d - cp; out[6] = s + cp; out[7] = d - cp;
}

// A coefficient's mantissa in the unit 2^u of a sum, its own unit being 2^e.
__device__ __forceinline__ fx::i64 in_unit(const fx::Float& f, int e, int u) { return f.m >> fx::imin(u - e, 63); }
// The unit 2^k of a cross product's component whose two products have scales of
// their own (2^-61 of their bounds): how far each is shifted to it.
struct Unit {
  int k, dp, dn;
  __device__ __forceinline__ Unit() {}
  // edge and vector scales of the positive and of the negative product
  __device__ __forceinline__ Unit(int ep, int vp, int en, int vn) {
    const int p = 61 - (ep + vp), n = 61 - (en + vn);
    k = fx::imax(p, n);
    dp = fx::imin(k - p, 63);
    dn = fx::imin(k - n, 63);
  }
};
// Whether a sum is in range: coefficients at most 2^400 (so not infinities or
// NaN, top their largest exponent), and a unit whose values are doubles or none.
__device__ __forceinline__ bool good_sum(int top, int u) { return top <= 340 && (u < -2000 || u >= -950); }

// ---------------------------------------------------------------------------
// ka_kinematics: transpose of k_kinematics (volume, characteristic length,
// velocity-gradient trace, monotonic-Q gradients), into the corner buffers.
// The cycle's end positions are the next cycle's start positions, so the
// position transpose of the next cycle's k_force (what force_geo_t does for
// the first cycle) joins it here, from what that cycle's ka_hourglass left:
// its modes' transpose starts the position corners, its volume-derivative
// Hessian-vector product merges with this cycle's volume gradient, and its
// stress terms add to the same face-diagonal adjoints, scattered once.
// ---------------------------------------------------------------------------
//
// Three threads per element, one per coordinate and each in a warp of its own,
// as in the forward kernels: a thread forms its component of every product,
// and what a cross product needs of the other components is in shared memory.
//
// The crosses onto the edges and the face diagonals, all of an edge, a diagonal
// (or a sum of two) and an adjoint vector, and the sums onto the position corners
// run on the integer pipes. Edges and diagonals are scaled by their coordinate's
// extent, adjoint vectors by their coordinate's largest; what else joins the corners (edges, modes, V x W)
// enters as mantissas in the largest term's unit. Elements of sizes or adjoints
// out of range take the crosses in doubles, the positions' part from the tape.
// Bound by FP64 issue (350 slots per element, the pipe 69 % busy; ALU 32 %,
// multiply-adds 15 %). At 48^3 173 us with the crosses and corner sums on the FP64
// pipe (87 % busy), 116 us so; a gradient of 40 cycles at 48^3 21.7 -> 20.0 ms, of
// 24 cycles at 15^3 2.81 -> 2.73. Six blocks per SM (96 registers; 148 slots are
// the most six can have) against five and seven: 20.04, 20.37, 20.18 ms. The
// volume's scalars in one thread instead of all three (a barrier more) and the
// velocity corners on the integer pipes: 101 us, 19.52 -> 18.91 ms, 2.65 -> 2.61;
// the edges' crosses there too: 95 us, 18.61 -> 18.29, 2.60 -> 2.60; a scale for each
// coordinate's adjoint vectors, 96 us.
enum : int {
  // per coordinate: mean edges, half-step edges, 12 diagonals, U vectors (limbs),
  // the differences of dL/ddv along V and -W, the faces' terms (by the face's
  // first diagonal), Lv12 U + dU; then the adjoints of the edges' cross products
  // and of the cofactors (doubles, then limbs)
  KA_W = 0, KA_F = 3, KA_D = 6, KA_U = 18, KA_DV = 21, KA_DW = 24, KA_LN = 27, KA_A = 33,
  KA_LA = 36, KA_LC = 39, KA_COMP = 42,
  // per direction d: 2 Ls2, Ldv norm64, its part of Lvol; 3 k + d: dot terms; per
  // coordinate sg and the largest scales its adjoint vectors take
  KA_DIR = 3 * KA_COMP, KA_DOT = KA_DIR + 9, KA_EXP = KA_DOT + 9, KA_COUNT = KA_EXP + 3
};

template <int MODE>
__global__ void __launch_bounds__(3 * kFixedElems, 6) ka_kinematics(AdjDev a, const CycleRec* rec) {
  __shared__ double column[KA_COUNT * kFixedElems];
  const int E = a.E;
  const int lane = threadIdx.x % kFixedElems, k = threadIdx.x / kFixedElems;
  const int slot = blockIdx.x * kFixedElems + lane;
  const bool live = slot < E;
  const int e = live ? slot : E - 1;  // threads past the end repeat the last element and store nothing
  wait_for_last_kernel();
  const double dt = rec->dt;
  auto sh = [&](int i) -> double& { return column[i * kFixedElems + lane]; };
  auto num = [&](int i) -> fx::Num& { return reinterpret_cast<fx::Num*>(column)[i * kFixedElems + lane]; };
  const int own = KA_COMP * k, c1 = KA_COMP * (k == 2 ? 0 : k + 1), c2 = KA_COMP * (k == 0 ? 2 : k - 1);
  // forward values from the kinematics kernel's tape (slots: see tapeKin)
  auto tk = [&](int q) { return a.kin[row(q, E, e)]; };

  const double vnew = a.vnew[e], volo = a.volo[e], inv_volo = a.inv_volo[e];
  const double vol = volo * vnew, norm64 = tk(40);  // norm64 = 1/(64 vol + 64 ptiny)
  const double inv = tk(27), lvdov = a.lvdov[e];
  const double Ls = lvdov * inv, Ldet = -lvdov * a.vdov[e] * inv;
  const double ldelv = a.ldelv[e], Lar = a.larealg[e], lvnew_in = a.lvnew[e];
  if (live && k == 0) a.lv[e] -= ldelv;  // delv = vnew - v
  double A[3], VW[3], C[3], U[3], dU[3], F1;
  unsigned top = 0;  // high word of the largest adjoint vector component
  bool ok;           // extent in range
  int sg;            // its scale
  {
    // direction k: limiter reads of this element's delv by its neighbours
    // (inverse neighbour list, fixed order) join its own delv adjoint
    double Ldv = a.ldv[k][e];
    for (int j = a.nbStart[e]; j < a.nbStart[e + 1]; ++j) {
      const int ent = a.nbList[j];
      if (((ent / E) >> 1) == k) Ldv += a.lnb[ent];
    }
    const double rs = tk(37 + k);  // 1/sqrt(|A|^2 + 256 ptiny)
    const double t = a.ldx[k][e] * 16.0 * rs;
    sh(KA_DIR + k) = -(t * vol) * (rs * rs);  // 2 Ls2, Ls2 = Ldx 16 vol (-1/2) rs^3
    sh(KA_DIR + 3 + k) = Ldv * norm64;
    sh(KA_DIR + 6 + k) = t;
    const double dt2 = -0.5 * dt;
    double W[3], F[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double w = tk(3 * k + d);
      VW[d] = tk(9 + 3 * k + d);
      A[d] = tk(28 + 3 * d + k);
      C[d] = tk(18 + 3 * d + k);
      W[d] = w;
      F[d] = fma(dt2, VW[d], w);
      top = fx::umax(top, fx::umax((unsigned)fx::hi_word(W[d]) & 0x7fffffffu, (unsigned)fx::hi_word(F[d]) & 0x7fffffffu));
      sh(KA_DOT + 3 * k + d) = A[d] * VW[d];
    }
    F1 = F[1];
    // the 12 diagonals of the new positions: d61 d70 d63 d20 d50 d64 d31 d72
    // d43 d57 d14 d25
    double g[12];
#pragma unroll
    for (int q = 0; q < 12; ++q) {
      g[q] = tk(45 + 3 * q + k);
      top = fx::umax(top, (unsigned)fx::hi_word(g[q]) & 0x7fffffffu);
    }
    const int eg = fx::exponent_field(top);
    top = 0;
    ok = eg >= fx::wide().least_extent && eg <= 1023 + 40;
    sg = 1081 - eg;  // below 2^59
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      num(own + KA_W + d) = fx::limbs(fx::to_fixed(W[d], 6 - eg));
      num(own + KA_F + d) = fx::limbs(fx::to_fixed(F[d], 6 - eg));
    }
    fx::i64 x[12];
#pragma unroll
    for (int q = 0; q < 12; ++q) {
      x[q] = fx::to_fixed(g[q], 6 - eg);
      num(own + KA_D + q) = fx::limbs(x[q]);
    }
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      U[t] = g[6 + 2 * t] + g[7 + 2 * t];
      num(own + KA_U + t) = fx::limbs(fx::add(x[6 + 2 * t], x[7 + 2 * t]));
    }
    // The next cycle's force kernel used the gradient of 12*volume (its
    // voluDer, dv): G = dL/ddv (zero before the first transposed cycle; the
    // faithful slots 1 and 3 swapped back) makes its transpose the
    // Hessian-vector product of the same triple products along G; dU, dV, dW
    // are the differences of G along U, V, W.
    double G[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int src = (MODE & 2) ? c : c == 1 ? 3 : c == 3 ? 1 : c;
      G[c] = a.sLdv[row(k * 8 + src, E, e)];
    }
    dU[0] = (G[3] - G[1]) + (G[7] - G[2]);
    dU[1] = (G[4] - G[3]) + (G[5] - G[7]);
    dU[2] = (G[1] - G[4]) + (G[2] - G[5]);
    auto put = [&](int i, double y) {
      top = fx::umax(top, (unsigned)fx::hi_word(y) & 0x7fffffffu);
      sh(own + i) = y;
    };
    put(KA_DV, G[6] - G[3]);
    put(KA_DV + 1, G[6] - G[4]);
    put(KA_DV + 2, G[6] - G[1]);
    put(KA_DW, G[0] - G[2]);
    put(KA_DW + 1, G[0] - G[7]);
    put(KA_DW + 2, G[0] - G[5]);
    // The next cycle's stress force: face f's normal d1 x d2 with LN = s8 LU_f
    // gives d1 the adjoint d2 x LN and d2 the adjoint LN x d1; s8 from this
    // cycle's end state. Faces (d20, d31) (d50, d14) (d61, d25) (d72, d36) (d43,
    // d07) with d36 = -d63, d07 = -d70, the adjoint pairs of the last two turned.
    const double s8 = ((-a.p1[e]) - a.q1[e]) * 0.125;
    constexpr int at[5] = {3, 4, 0, 2, 1};
#pragma unroll
    for (int f = 0; f < 5; ++f) put(KA_LN + at[f], s8 * a.sLU[row(3 * f + k, E, e)]);
    sh(own + KA_LN + 5) = 0.0;  // the face (d64, d57), of the characteristic length alone
  }
  __syncthreads();
  // ---- the edges' adjoints; in thread 0 the scalars of the volume ----
  double LVW[3], LA[3], LC[3];
  {
    unsigned ta = 0, tc = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double ldn = sh(KA_DIR + 3 + d);
      LA[d] = fma(A[d], sh(KA_DIR + d), ldn * VW[d]);
      LVW[d] = fma(ldn, A[d], Ls * C[d]);
      // velocity-gradient trace: cofactor columns C and 1/det
      LC[d] = d == 1 ? fma(Ldet, F1, Ls * VW[1]) : Ls * VW[d];
      ta = fx::umax(ta, (unsigned)fx::hi_word(LA[d]) & 0x7fffffffu);
      tc = fx::umax(tc, (unsigned)fx::hi_word(LC[d]) & 0x7fffffffu);
    }
    // the scale of below 2^59, plus 512; 0: out of range
    auto limit = [&](unsigned t) {
      const int x = fx::exponent_field(t);
      return ok && (t == 0 || (x >= fx::kMinSpeed && x <= fx::kMaxSpeed)) ? 1081 - fx::imax(x, fx::kMinSpeed) + 512 : 0;
    };
    num(KA_EXP + k).lo = (sg & 0xff) | limit(ta) << 8 | limit(tc) << 20;
  }
  if (k == 0) {
    double Lvol = 0.0, Lnorm64 = 0.0;  // the latter times norm64
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      Lvol += sh(KA_DIR + 6 + d);
      Lnorm64 = fma(sh(KA_DIR + 3 + d), (sh(KA_DOT + d) + sh(KA_DOT + 3 + d)) + sh(KA_DOT + 6 + d), Lnorm64);
    }
    Lvol = fma(Lnorm64, -64.0 * norm64, Lvol);
    const double Lvnew = fma(Lvol, volo, lvnew_in + ldelv);
    // characteristic length from the face the tape recorded
    const double rsc = tk(44);  // 1/|fa x fb|
    sh(KA_DOT) = fma(Lar * 2.0, rsc, Lvnew * inv_volo) * (1.0 / 12.0);
    // 2 Lcl, Lcl = Lar 2 volume (-1/2) rsc^3
    sh(KA_DOT + 1) = -2.0 * (Lar * vol) * (rsc * rsc * rsc);
  }
  __syncthreads();
  const double Lv12 = sh(KA_DOT);
  {
    // the characteristic length joins the terms of its face: in the kinematics
    // face order (d20, d31) (d64, d57) (d50, d14) (d61, d25) (d72, d63) (d43, d70)
    const double lf = tk(41 + k) * sh(KA_DOT + 1);
    const int f = (int)((a.flags[e] >> TF_FACE_SHIFT) & 7ull);
    const int at = KA_LN + ((0x120453 >> (4 * f)) & 15);
    const double ln = sh(own + at) + (f < 4 ? lf : -lf);
    sh(own + at) = ln;
    top = fx::umax(top, (unsigned)fx::hi_word(ln) & 0x7fffffffu);
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      const double y = fma(Lv12, U[t], dU[t]);
      sh(own + KA_A + t) = y;
      top = fx::umax(top, (unsigned)fx::hi_word(y) & 0x7fffffffu);
    }
    int ea = fx::exponent_field(top);
    ok = ok && (top == 0 || (ea >= fx::kMinSpeed && ea <= fx::kMaxSpeed));
    num(KA_EXP + k).hi = ok ? 1081 - fx::imax(ea, fx::kMinSpeed) : fx::kNoExponent;  // below 2^59
  }
  // The edges' adjoints in their units. Each coordinate's adjoint vectors have a
  // scale of their own: what a component's two coordinates hold may be far below
  // what the third does.
  const int k1 = k == 2 ? 0 : k + 1, k2 = k == 0 ? 2 : k - 1;
  bool ok_edges;
  Unit unit_A, unit_C;
  {
    const int x0 = num(KA_EXP).lo, x1 = num(KA_EXP + 1).lo, x2 = num(KA_EXP + 2).lo;
    const int here = num(KA_EXP + k).lo, xp = num(KA_EXP + k1).lo, xq = num(KA_EXP + k2).lo;
    auto scale = [](int x, int shift) { return ((x >> shift) & 0xfff) - 512; };
    auto all = [&](int shift) { return (x0 >> shift & 0xfff) != 0 && (x1 >> shift & 0xfff) != 0 && (x2 >> shift & 0xfff) != 0; };
    ok_edges = all(8) && all(20);
    unit_A = Unit(xp & 0xff, scale(xq, 8), xq & 0xff, scale(xp, 8));
    unit_C = Unit(xp & 0xff, scale(xq, 20), xq & 0xff, scale(xp, 20));
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (ok_edges) {
        num(own + KA_LA + d) = fx::limbs(fx::to_fixed0(LA[d], scale(here, 8) - 1075));
        num(own + KA_LC + d) = fx::limbs(fx::to_fixed0(LC[d], scale(here, 20) - 1075));
      } else {
        sh(own + KA_LA + d) = LA[d];
        sh(own + KA_LC + d) = LC[d];
      }
    }
  }
  __syncthreads();
  Unit unit;
  {
    const fx::Num x0 = num(KA_EXP), x1 = num(KA_EXP + 1), x2 = num(KA_EXP + 2);
    const fx::Num mine = num(KA_EXP + k), xp = num(KA_EXP + k1), xq = num(KA_EXP + k2);
    ok = fx::imin(x0.hi, fx::imin(x1.hi, x2.hi)) != fx::kNoExponent;
    unit = Unit(xp.lo & 0xff, xq.hi, xq.lo & 0xff, xp.hi);
    if (ok)
#pragma unroll
      for (int q = KA_DV; q < KA_LA; ++q) num(own + q) = fx::limbs(fx::to_fixed0(sh(own + q), mine.hi - 1075));
  }
  // component k of sums of crosses of an edge or diagonal (slot i) and an adjoint
  // vector (slot j), or (minus) the other way round: the products of the edge's
  // next component and the vector's after it have one scale, the others another
  struct Cross { fx::Acc p, n; };
  auto first = [&](int i, int j) {
    Cross r;
    r.p = fx::mul(num(c1 + i), num(c2 + j));
    r.n = fx::mul(num(c2 + i), num(c1 + j));
    return r;
  };
  auto plus = [&](Cross& r, int i, int j) {
    fx::mac(r.p, num(c1 + i), num(c2 + j));
    fx::mac(r.n, num(c2 + i), num(c1 + j));
  };
  auto minus = [&](Cross& r, int i, int j) {
    fx::msub(r.p, num(c1 + i), num(c2 + j));
    fx::msub(r.n, num(c2 + i), num(c1 + j));
  };
  auto value = [](const Cross& r, const Unit& u) { return (fx::take<3>(r.p) >> u.dp) - (fx::take<3>(r.n) >> u.dn); };
  // the same in doubles, the positions' slots from the tape
  auto at = [&](int j, int i) {
    if (i >= KA_DV) return sh(KA_COMP * j + i);
    auto t = [&](int q) { return a.kin[row(q, E, e)]; };
    if (i < KA_F) return t(3 * j + i - KA_W);
    if (i < KA_D) return fma(-0.5 * dt, t(9 + 3 * j + i - KA_F), t(3 * j + i - KA_F));
    auto d = [&](int q) { return t(45 + 3 * q + j); };
    return i < KA_U ? d(i - KA_D) : d(6 + 2 * (i - KA_U)) + d(7 + 2 * (i - KA_U));
  };
  auto add_cross = [&](double y, int i, int j) { return fma(at(k1, i), at(k2, j), fma(-at(k2, i), at(k1, j), y)); };
  // ---- positions' and velocities' edges: direction d uses A = P x Q, P and Q the
  //      edges after it; C0 = F1 x F2, C1 = F2 x F0, C2 = F0 x F1 ----
  double LW[3], LF[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int b = (i + 1) % 3, c = (i + 2) % 3;  // P of c, Q of b
    if (ok_edges) {
      Cross r = first(KA_W + b, KA_LA + c);
      minus(r, KA_W + c, KA_LA + b);
      LW[i] = fx::to_double(value(r, unit_A), unit_A.k);
      r = first(KA_F + b, KA_LC + c);
      minus(r, KA_F + c, KA_LC + b);
      LF[i] = fx::to_double(value(r, unit_C), unit_C.k);
    } else {
      LW[i] = add_cross(add_cross(0.0, KA_W + b, KA_LA + c), KA_LA + b, KA_W + c);
      LF[i] = add_cross(add_cross(0.0, KA_F + b, KA_LC + c), KA_LC + b, KA_F + c);
    }
  }
  LF[1] = fma(Ldet, C[1], LF[1]);
  {
    double Ldt = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      LW[d] += LF[d];
      LVW[d] = fma(-0.5 * dt, LF[d], LVW[d]);
      Ldt = fma(LF[d], VW[d], Ldt);
    }
    sh(KA_DIR + k) = live ? -0.5 * Ldt : 0.0;
  }
  // the velocity corners (the Walsh transpose), plus the hourglass velocity
  // corners of the cycle after this one
  {
    fx::Float f[11];  // LVW, then the corners: mantissas below 2^59, four to a corner
    int top = fx::kNoExponent;
#pragma unroll
    for (int q = 0; q < 11; ++q) {
      f[q] = fx::to_float(q < 3 ? LVW[q] : a.fV[row(k * 8 + q - 3, E, e)]);
      top = fx::imax(top, f[q].k);
    }
    const int u = top + 2;
    if (good_sum(top, u)) {
      fx::i64 y[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) y[c] = in_unit(f[3 + c], f[3 + c].k, u);
      const fx::i64 w[3] = {in_unit(f[0], f[0].k, u), in_unit(f[1], f[1].k, u), in_unit(f[2], f[2].k, u)};
      walsh1_t(w, y);
      if (live)
#pragma unroll
        for (int c = 0; c < 8; ++c) a.cV[row(k * 8 + c, E, e)] = fx::to_double(y[c], u);
    } else {
      double y[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) y[c] = a.fV[row(k * 8 + c, E, e)];
      walsh1_t(LVW, y);
      if (live)
#pragma unroll
        for (int c = 0; c < 8; ++c) a.cV[row(k * 8 + c, E, e)] = y[c];
    }
  }
  // ---- volume and characteristic length, and the position transpose of the
  //      next cycle's k_force (same positions, same face diagonals) ----
  // dL/dU = Lv12 (V x W) + dV x W + V x dW, dL/dV = W x A + dW x U, dL/dW =
  // A x V + U x dV with A = Lv12 U + dU (V x W is taped). U, V, W of triple t:
  // diagonals 6 + 2 t and 7 + 2 t, iv, iw; the partner of diagonal q in its face
  constexpr int iv[3] = {2, 5, 0}, iw[3] = {3, 1, 4}, partner[12] = {11, 8, 7, 6, 10, 9, 3, 2, 1, 5, 4, 0};
  // corners a diagonal runs from and to
  constexpr int pp[12] = {6, 7, 6, 2, 5, 6, 3, 7, 4, 5, 1, 2}, pq[12] = {1, 0, 3, 0, 0, 4, 1, 2, 3, 7, 4, 5};
  double vw[3], tm[4], LX[8];
#pragma unroll
  for (int t = 0; t < 3; ++t) vw[t] = Lv12 * tk(81 + 3 * t + k);
  // the next cycle's hourglass modes
#pragma unroll
  for (int m = 0; m < 4; ++m) tm[m] = a.sLhm[row(k * 4 + m, E, e)];
  __syncthreads();
  bool summed = false;
  if (ok) {
    fx::i64 X[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // below 3 2^60
    auto onto = [&](int q, fx::i64 y) { X[pp[q]] += y; X[pq[q]] -= y; };
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      const int v = iv[t], w = iw[t];
      // (the slots of dW hold -dW)
      Cross r = first(KA_D + w, KA_DV + t);
      plus(r, KA_D + v, KA_DW + t);
      const fx::i64 gU = value(r, unit);
#pragma unroll
      for (int q = 6 + 2 * t; q < 8 + 2 * t; ++q) onto(q, -(gU + value(first(KA_D + partner[q], KA_LN + partner[q]), unit)));
      r = first(KA_D + w, KA_A + t);
      plus(r, KA_U + t, KA_DW + t);
      plus(r, KA_D + partner[v], KA_LN + v);
      onto(v, value(r, unit));
      r = first(KA_U + t, KA_DV + t);
      minus(r, KA_D + v, KA_A + t);
      plus(r, KA_D + partner[w], KA_LN + w);
      onto(w, value(r, unit));
    }
    // the other terms' mantissas below 2^58, ten to a corner
    fx::Float f[10];
    int top = fx::kNoExponent;
#pragma unroll
    for (int q = 0; q < 10; ++q) {
      f[q] = fx::to_float(q < 3 ? vw[q] : q < 6 ? LW[q - 3] : tm[q - 6]);
      top = fx::imax(top, f[q].k);
    }
    const int u = fx::imax(unit.k, top + 3);
    summed = good_sum(top, u);
    if (summed) {
      fx::i64 i[10], y[8];
#pragma unroll
      for (int q = 0; q < 10; ++q) i[q] = in_unit(f[q], f[q].k, u);
      const fx::i64 t[4] = {i[6], i[7], i[8], i[9]}, w[3] = {i[3], i[4], i[5]};
      walsh_modes_t(t, y);
      walsh1_t(w, y);
#pragma unroll
      for (int q = 6; q < 12; ++q) { y[pp[q]] += i[(q - 6) / 2]; y[pq[q]] -= i[(q - 6) / 2]; }
      const int down = fx::imin(u - unit.k, 63);
#pragma unroll
      for (int c = 0; c < 8; ++c) LX[c] = fx::to_double((X[c] >> down) + y[c], u);
    } else {
#pragma unroll
      for (int c = 0; c < 8; ++c) LX[c] = fx::to_double(X[c], unit.k);
    }
  } else {
#pragma unroll
    for (int c = 0; c < 8; ++c) LX[c] = 0.0;
    auto onto = [&](int q, double y) { LX[pp[q]] += y; LX[pq[q]] -= y; };
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      const int v = iv[t], w = iw[t];
      const double gU = add_cross(add_cross(0.0, KA_DV + t, KA_D + w), KA_DW + t, KA_D + v);
#pragma unroll
      for (int q = 6 + 2 * t; q < 8 + 2 * t; ++q) onto(q, add_cross(gU, KA_LN + partner[q], KA_D + partner[q]));
      onto(v, add_cross(add_cross(add_cross(0.0, KA_D + w, KA_A + t), KA_U + t, KA_DW + t), KA_D + partner[v], KA_LN + v));
      onto(w, add_cross(add_cross(add_cross(0.0, KA_A + t, KA_D + v), KA_U + t, KA_DV + t), KA_D + partner[w], KA_LN + w));
    }
  }
  if (!summed) {
    double y[8];
    walsh_modes_t(tm, y);
    walsh1_t(LW, y);
#pragma unroll
    for (int q = 6; q < 12; ++q) { y[pp[q]] += vw[(q - 6) / 2]; y[pq[q]] -= vw[(q - 6) / 2]; }
#pragma unroll
    for (int c = 0; c < 8; ++c) LX[c] += y[c];
  }
  if (live)
#pragma unroll
    for (int c = 0; c < 8; ++c) a.cX[row(k * 8 + c, E, e)] = LX[c];
  if (k == 2) {
    double Ldt = (sh(KA_DIR) + sh(KA_DIR + 1)) + sh(KA_DIR + 2);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) Ldt += __shfl_down_sync(0xffffffffu, Ldt, o);
    if (lane == 0) a.part_dt[blockIdx.x] = Ldt;
  }
}

// Sums the force corner buffers into node adjoints (added to what is there):
// the last step of a reverse sweep (each cycle's ka_node gathers the previous
// transposed cycle's force corners itself).
__global__ void __launch_bounds__(kAdjBlock) ka_gather_corners(AdjDev a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.N) return;
  const int s = a.nodeElemStart[i], t = a.nodeElemStart[i + 1];
  const long long E8 = 8ll * a.E;
  double gx = 0, gy = 0, gz = 0, hx = 0, hy = 0, hz = 0;
  for (int j = s; j < t; ++j) {
    const int c = a.cornerList[j];
    gx += a.fX[c]; gy += a.fX[E8 + c]; gz += a.fX[2 * E8 + c];
    hx += a.fV[c]; hy += a.fV[E8 + c]; hz += a.fV[2 * E8 + c];
  }
  a.lx[i] += gx; a.ly[i] += gy; a.lz[i] += gz;
  a.lxd[i] += hx; a.lyd[i] += hy; a.lzd[i] += hz;
}

// ---------------------------------------------------------------------------
// ka_node: transpose of k_node (position and velocity update with the
// velocity snap, acceleration = force / mass with the symmetry BCs).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kAdjBlock) ka_node(AdjDev a, const CycleRec* rec) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  wait_for_last_kernel();
  const double dt = rec->dt;
  double Ldt = 0.0;
  if (i < a.N) {
    const unsigned bc = a.nodeBC[i];
    const double im = a.inv_nodalMass[i];
    double* Lx[3] = {a.lx, a.ly, a.lz};
    double* Lxd[3] = {a.lxd, a.lyd, a.lzd};
    double* Lf[3] = {a.lfx, a.lfy, a.lfz};
    const double* xd1[3] = {a.xd1, a.yd1, a.zd1};
    const double* acc[3] = {a.ax, a.ay, a.az};
    // the end-state adjoints gather this cycle's kinematics transpose and
    // (added per corner by ka_kinematics) the force transpose of the cycle
    // after this one
    double gx[3] = {0.0, 0.0, 0.0}, gv[3] = {0.0, 0.0, 0.0};
    {
      const int s = a.nodeElemStart[i], t = a.nodeElemStart[i + 1];
      const long long E8 = 8ll * a.E;
      for (int j = s; j < t; ++j) {
        const int c = a.cornerList[j];
#pragma unroll
        for (int k = 0; k < 3; ++k) { gx[k] += a.cX[k * E8 + c]; gv[k] += a.cV[k * E8 + c]; }
      }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double lxn = Lx[k][i] + gx[k];
      const double v1 = xd1[k][i];
      double lv = (Lxd[k][i] + gv[k]) + lxn * dt;   // x1 = x0 + xd1*dt
      Ldt += lxn * v1;
      double lf = 0.0;
      if (v1 == 0.0) {
        lv = 0.0;                        // snapped to zero (|v| < u_cut)
      } else {
        const double acc_k = acc[k][i];
        Ldt += lv * acc_k;               // xd1 = xd0 + a*dt
        if (!(bc & (1u << k))) lf = lv * dt * im;
      }
      Lx[k][i] = lxn;
      Lxd[k][i] = lv;
      Lf[k][i] = lf;
    }
  }
  block_sum_to(Ldt, a.part_dtn);
}

// Transpose of timeIncrement! (src/domain.jl:920-961) for the recorded
// inputs: Ldt is the adjoint of the new deltatime; adds to the adjoints of
// the previous time, deltatime, dtcourant and dthydro along the branch taken.
__host__ __device__ inline void time_increment_reverse(const CycleRec& r, const Params& prm, double Ldt,
                                                       double& Ltime, double& Ldt_prev, double& Ldtc,
                                                       double& Ldth) {
  double targetdt = prm.stoptime - r.time_prev;
  double dt_pre = r.dt_prev;
  int which = 0, rb = 0;
  bool mb = false;
  const bool adaptive = prm.dtfixed <= 0.0 && r.cycle_prev != 0;
  if (adaptive) {
    const double olddt = r.dt_prev;
    double gnewdt = (double)INFINITY;
    if (r.dtc_in < gnewdt) { gnewdt = r.dtc_in / 2.0; which = 1; }
    if (r.dth_in < gnewdt) { gnewdt = r.dth_in * 2.0 / 3.0; which = 2; }
    double newdt = gnewdt;
    const double ratio = newdt / olddt;
    if (ratio >= 1.0) {
      if (ratio < prm.deltatimemultlb) { newdt = olddt; rb = 1; }
      else if (ratio > prm.deltatimemultub) { newdt = olddt * prm.deltatimemultub; rb = 2; }
    }
    if (!(newdt != newdt) && (prm.dtmax != prm.dtmax || prm.dtmax < newdt)) { newdt = prm.dtmax; mb = true; }
    dt_pre = newdt;
  }
  bool t1 = false;
  if (dt_pre < targetdt && targetdt < 4.0 * dt_pre / 3.0) { targetdt = 2.0 * dt_pre / 3.0; t1 = true; }
  const bool t2 = targetdt < dt_pre;
  double Lpre = 0.0;
  if (t2) {
    if (t1) Lpre += (2.0 / 3.0) * Ldt;
    else Ltime += -Ldt;  // dt = stoptime - time
  } else {
    Lpre += Ldt;
  }
  if (!adaptive) { Ldt_prev += Lpre; return; }
  if (mb) return;
  if (rb == 1) { Ldt_prev += Lpre; return; }
  if (rb == 2) { Ldt_prev += prm.deltatimemultub * Lpre; return; }
  if (which == 1) Ldtc += 0.5 * Lpre;
  else if (which == 2) Ldth += (2.0 / 3.0) * Lpre;
}

// Closes the transpose of one cycle's time (one block of 3 kFixedElems threads):
// sums the kernels' partial adjoints of dt in a fixed order (each thread its
// strided share of both, a warp tree, then the warps in order), then transposes
// time += dt and timeIncrement! on the carried scalar adjoints.
__device__ __noinline__ void cycle_close(const AdjDev& a, int ge, int gn, const CycleRec* rec, AdjScal* sc,
                                         const Params& prm) {
  constexpr int kBlock = 3 * kFixedElems;
  double t_kin = 0.0, t_node = 0.0;
  for (int j = threadIdx.x; j < ge; j += kBlock) t_kin += a.part_dt[j];
  for (int j = threadIdx.x; j < gn; j += kBlock) t_node += a.part_dtn[j];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    t_kin += __shfl_down_sync(0xffffffffu, t_kin, o);
    t_node += __shfl_down_sync(0xffffffffu, t_node, o);
  }
  __shared__ double wsum[2][kBlock / 32];
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) { wsum[0][w] = t_kin; wsum[1][w] = t_node; }
  __syncthreads();
  if (threadIdx.x != 0) return;
  double s_kin = wsum[0][0], s_node = wsum[1][0];
#pragma unroll
  for (int k = 1; k < kBlock / 32; ++k) { s_kin += wsum[0][k]; s_node += wsum[1][k]; }
  const CycleRec r = *rec;
  AdjScal v = *sc;
  // a minimum the cycle did not reach leaves the scalar as it was
  double Ldtc_prev = r.active_c ? 0.0 : v.Ldtc, Ldth_prev = r.active_h ? 0.0 : v.Ldth;
  // time_n = time_{n-1} + dt_n
  const double Ldt_tot = v.Ldt + (s_kin + s_node) + v.Ltime;
  double Ldt_prev = 0.0;
  time_increment_reverse(r, prm, Ldt_tot, v.Ltime, Ldt_prev, Ldtc_prev, Ldth_prev);
  v.Ldt = Ldt_prev;
  v.Ldtc = Ldtc_prev;
  v.Ldth = Ldth_prev;
  *sc = v;
}

// ---------------------------------------------------------------------------
// Transpose of k_force, in two kernels: ka_hourglass (the FB hourglass force
// onto the velocities, ss, v, hgcoef and the two geometric factors) and
// ka_force_geo (the stress force and those geometric factors onto the
// positions).
// ---------------------------------------------------------------------------

// Hourglass transpose. With hg[n][m] = gamma[n][m] - sum_j dv_j[n] hms_j[m]
// (hms = the modes over 12*determ), S_k = hg^T V_k, T_k = hg^T lf_k (lf the
// force adjoints) and coef the hourglass coefficient, the forward force is
// F_k = coef hg S_k and its transpose needs only
//   dL/dV_k   = coef hg T_k,
//   dL/ddv_j  = -coef sum_k (lf_k (S_k . hms_j) + V_k (T_k . hms_j)),
//   dL/dhms_j = -coef sum_k (S_k (lf_k . dv_j) + T_k (V_k . dv_j)),
//   dL/dcoef  = sum_k S_k . T_k,
// where hg^T u = Gamma(u) - sum_j hms_j (dv_j . u): 3x3 dot-product tables
// replace the 8x4 matrices hg and dL/dhg.
//
// Three threads per element, one per coordinate k of V and lf. The sums over
// the 8 corners and onto them run on the integer pipes: derivatives share one
// scale per coordinate, velocities and force adjoints enter by their differences
// to corner 0 (the derivatives sum to zero over the corners, the modes' signs do
// too). dL/ddv is formed up to the same constant for every corner, which the
// differences it is used by do not see. A sum of products with coefficients of
// different size takes the largest term's unit, the others' mantissas shifted. Values
// outside 2^-400..2^400, infinities and NaN take the same sums in doubles, from
// the tape.
// Bound by FP64 issue (451 slots per element, the pipe 76 % busy; ALU 18 %,
// multiply-adds 10 %). At 48^3 155 us with every sum on the FP64 pipe (81 %
// busy), 113 us so; a gradient of 40 cycles at 48^3 went from 22.9 to 21.7 ms by
// this form, of 24 cycles at 15^3 from 2.97 to 2.93 ms. Five blocks per SM (128
// registers, no spills) against six and seven: 21.63, 21.71, 21.78 ms.
//
// The last block closes the cycle's time beside the elements (nothing here reads
// it). As a launch of one block it took 10 us of the chain at 48^3; a gradient of
// 40 cycles 19.80 -> 19.35 ms without it, of 24 cycles at 15^3 2.78 -> 2.65.
enum : int {
  HA_DV = 0,                 // 8 j + c: limbs of the volume derivatives of coordinate j
  HA_V = 24, HA_L = 48,      // 8 k + c: limbs of the corner differences of the velocities and force
                             // adjoints, in place of corner 0 their exponent and whether they are in range
  HA_HMS = 72,               // 4 j + m
  HA_P = 84,                 // 12 k + 4 j + m: coordinate k's part of P_j[m]
  HA_NA = 120, HA_NB = 129,  // 3 k + j
  HA_DVK = 138,              // j: the derivatives' exponent, and whether they are in range
  HA_COEF = 141,             // coef, -coef vi12
  HA_SUM = 143,              // k: S_k . T_k; 3 + j: P_j . hms_j; 6 + k: normals' part of the stress
  HA_COUNT = 152
};

// Limbs of the corner differences u[c] - u[0], c = 1..7, below 2^59, and in
// place of corner 0 their scale's exponent and whether they are in range.
template <class Put>
__device__ __forceinline__ void corner_differences(const double u[8], Put put) {
  int ev = fx::extent_field(u);
  // (all zero, or in range)
  const bool ok = ev == 0 || (ev >= fx::kMinSpeed && ev <= fx::kMaxSpeed);
  ev = ok ? fx::imax(ev, fx::kMinSpeed) : 0x7ff;
  fx::Num x;
  x.lo = 1081 - ev;
  x.hi = ok;
  put(0, x);
  const fx::i64 u0 = fx::to_fixed0(u[0], 6 - ev);
#pragma unroll
  for (int c = 1; c < 8; ++c) put(c, fx::limbs(fx::sub(fx::to_fixed0(u[c], 6 - ev), u0)));
}

template <int MODE>
__global__ void __launch_bounds__(3 * kFixedElems, 5)
    ka_hourglass(AdjDev a, double hgcoef, int gn, const CycleRec* rec, AdjScal* sc, Params prm) {
  __shared__ double column[HA_COUNT * kFixedElems];
  const int E = a.E;
  if (blockIdx.x == gridDim.x - 1) {
    wait_for_last_kernel();
    cycle_close(a, gridDim.x - 1, gn, rec, sc, prm);
    return;
  }
  const int lane = threadIdx.x % kFixedElems, k = threadIdx.x / kFixedElems;
  const int slot = blockIdx.x * kFixedElems + lane;
  const bool live = slot < E;
  const int e = live ? slot : E - 1;  // threads past the end repeat the last element and store nothing
  auto sh = [&](int i) -> double& { return column[i * kFixedElems + lane]; };
  auto num = [&](int i) -> fx::Num& { return reinterpret_cast<fx::Num*>(column)[i * kFixedElems + lane]; };
  const double* const V = k == 0 ? a.xd0 : k == 1 ? a.yd0 : a.zd0;
  const double* const Lf = k == 0 ? a.lfx : k == 1 ? a.lfy : a.lfz;
  int nd[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) nd[c] = a.nodelist[c * E + e];
  wait_for_last_kernel();
  double lf[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) lf[c] = Lf[nd[c]];
  double Lhg_coef = 0.0;
  if (!(hgcoef > 0.0)) {
    if (live) {
#pragma unroll
      for (int c = 0; c < 8; ++c) { a.fV[row(k * 8 + c, E, e)] = 0.0; a.sLdv[row(k * 8 + c, E, e)] = 0.0; }
#pragma unroll
      for (int m = 0; m < 4; ++m) a.sLhm[row(k * 4 + m, E, e)] = 0.0;
    }
  } else {
    double inv_det = 0.0, vi12 = 0.0, ss = 0.0, mass = 0.0, r = 0.0;  // thread 0
    double S[4], v[8], dv[8];
    {
      // the forward kernel's volume derivatives, scaled modes and mode sums
#pragma unroll
      for (int c = 0; c < 8; ++c) dv[c] = a.geo[row(k * 8 + c, E, e)];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        sh(HA_HMS + 4 * k + m) = a.geo[row(24 + 4 * k + m, E, e)];
        S[m] = a.geo[row(36 + 4 * k + m, E, e)];
      }
      unsigned top = 0;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        v[c] = V[nd[c]];
        top = fx::umax(top, (unsigned)fx::hi_word(dv[c]) & 0x7fffffffu);
      }
      corner_differences(v, [&](int c, fx::Num x) { num(HA_V + 8 * k + c) = x; });
      corner_differences(lf, [&](int c, fx::Num x) { num(HA_L + 8 * k + c) = x; });
      // below 2^60
      int ed = fx::exponent_field(top);
      const bool ok = ed == 0 || (ed >= fx::kMinSpeed && ed <= fx::kMaxSpeed);
      ed = ok ? fx::imax(ed, fx::kMinSpeed) : 0x7ff;
#pragma unroll
      for (int c = 0; c < 8; ++c) num(HA_DV + 8 * k + c) = fx::limbs(fx::to_fixed(dv[c], 7 - ed));
      fx::Num x;
      x.lo = 1082 - ed;
      x.hi = ok;
      num(HA_DVK + k) = x;
      if (k == 0) {
        const double determ = a.volo[e] * a.v0[e];
        inv_det = 1.0 / determ;
        vi12 = inv_det * (1.0 / 12.0);
        ss = a.ss0[e];
        mass = a.elemMass[e];
        r = inv_cbrt(determ);
        const double coef = ((-hgcoef * 0.01 * ss) * mass) * r;
        sh(HA_COEF) = coef;
        sh(HA_COEF + 1) = -coef * vi12;
      }
    }
    __syncthreads();
    // D[j] = V . dv_j, C[j] = lf . dv_j, w2 = the modes of lf
    const bool ok = num(HA_DVK).hi & num(HA_DVK + 1).hi & num(HA_DVK + 2).hi & num(HA_V).hi & num(HA_V + 8).hi &
                    num(HA_V + 16).hi & num(HA_L).hi & num(HA_L + 8).hi & num(HA_L + 16).hi;
    double D[3], C[3], w2[4];
    if (ok) {
      const int su = num(HA_V + 8 * k).lo, sl = num(HA_L + 8 * k).lo;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        fx::Acc x = fx::mul(num(HA_DV + 8 * j + 1), num(HA_V + 8 * k + 1));
        fx::Acc y = fx::mul(num(HA_DV + 8 * j + 1), num(HA_L + 8 * k + 1));
#pragma unroll
        for (int c = 2; c < 8; ++c) {
          fx::mac(x, num(HA_DV + 8 * j + c), num(HA_V + 8 * k + c));
          fx::mac(y, num(HA_DV + 8 * j + c), num(HA_L + 8 * k + c));
        }
        const int sd = num(HA_DVK + j).lo;
        D[j] = fx::to_double(fx::take<3>(x), 61 - sd - su);
        C[j] = fx::to_double(fx::take<3>(y), 61 - sd - sl);
      }
      fx::i64 t[4] = {0, 0, 0, 0};
#pragma unroll
      for (int c = 1; c < 8; ++c) {
        const fx::Num x = num(HA_L + 8 * k + c);
        const fx::i64 d = fx::shl((fx::i64)x.hi, 32) + x.lo;
#pragma unroll
        for (int m = 0; m < 4; ++m) t[m] += (fx::kGammaSigns >> (4 * c + m)) & 1u ? -d : d;
      }
#pragma unroll
      for (int m = 0; m < 4; ++m) w2[m] = fx::to_double(t[m], -sl);
    } else {
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        D[j] = C[j] = 0.0;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const double g = a.geo[row(j * 8 + c, E, e)];
          D[j] = fma(g, v[c], D[j]);
          C[j] = fma(g, lf[c], C[j]);
        }
      }
      double w1[3];
      walsh7(lf, w1, w2);
    }
    const double coef = sh(HA_COEF);
    // T = hg^T lf, A[j] = S . hms_j, B[j] = T . hms_j
    double T[4], Lcoef = 0.0, nA[3], nB[3];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      T[m] = fma(-sh(HA_HMS + 8 + m), C[2], fma(-sh(HA_HMS + 4 + m), C[1], fma(-sh(HA_HMS + m), C[0], w2[m])));
      Lcoef = fma(S[m], T[m], Lcoef);
    }
    sh(HA_SUM + k) = Lcoef;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      double x = 0.0, y = 0.0;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const double h = sh(HA_HMS + 4 * j + m);
        x = fma(S[m], h, x);
        y = fma(T[m], h, y);
        sh(HA_P + 12 * k + 4 * j + m) = fma(S[m], C[j], T[m] * D[j]);
      }
      // the coefficient folded into the tables
      nA[j] = -coef * x;
      nB[j] = -coef * y;
      sh(HA_NA + 3 * k + j) = nA[j];
      sh(HA_NB + 3 * k + j) = nB[j];
    }
    // dL/dV = coef (Gamma^T T - sum_j dv_j B[j]) = Gamma^T (coef T) + sum_j dv_j nB[j]
    {
      double cT[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) cT[m] = coef * T[m];
      // products over 2^62 below 2^60.6, the modes' mantissas over 4
      fx::Float fT[4], fB[3];
      int u = fx::kNoExponent, top = u;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        fT[m] = fx::to_float(cT[m]);
        top = fx::imax(top, fT[m].k);
        u = fx::imax(u, fT[m].k + 2);
      }
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        fB[j] = fx::to_float(nB[j]);
        top = fx::imax(top, fB[j].k);
        fB[j].k += 62 - num(HA_DVK + j).lo;
        u = fx::imax(u, fB[j].k);
      }
      if (ok && good_sum(top, u)) {
        fx::Num B[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) B[j] = fx::limbs(in_unit(fB[j], fB[j].k, u));
        fx::i64 t[4], q[8];
#pragma unroll
        for (int m = 0; m < 4; ++m) t[m] = in_unit(fT[m], fT[m].k, u);
        walsh_modes_t(t, q);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          fx::Acc x = fx::mul(num(HA_DV + c), B[0]);
          fx::mac(x, num(HA_DV + 8 + c), B[1]);
          fx::mac(x, num(HA_DV + 16 + c), B[2]);
          if (live) a.fV[row(k * 8 + c, E, e)] = fx::to_double(fx::take<2>(x) + q[c], u);
        }
      } else {
        double q[8];
        walsh_modes_t(cT, q);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          double f = q[c];
#pragma unroll
          for (int j = 0; j < 3; ++j) f = fma(a.geo[row(j * 8 + c, E, e)], nB[j], f);
          if (live) a.fV[row(k * 8 + c, E, e)] = f;
        }
      }
    }
    __syncthreads();
    // coordinate k as the derivatives' j. dL/dhms_j = -coef P_j with P_j[m] the
    // sums below; dL/dhm_j = vi12 dL/dhms_j (hms = vi12 hm); dL/dvi12 = sum_j
    // dL/dhms_j . hms_j / vi12
    double Pvi = 0.0;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const double P = (sh(HA_P + 4 * k + m) + sh(HA_P + 12 + 4 * k + m)) + sh(HA_P + 24 + 4 * k + m);
      Pvi = fma(P, sh(HA_HMS + 4 * k + m), Pvi);
      if (live) a.sLhm[row(k * 4 + m, E, e)] = sh(HA_COEF + 1) * P;
    }
    sh(HA_SUM + 3 + k) = Pvi;
    // dL/ddv_j = -coef sum_k (lf_k A[k][j] + V_k B[k][j]) = sum_k (lf_k nA[k][j] + V_k nB[k][j])
    {
      fx::Float fA[3], fB[3];
      int u = fx::kNoExponent, top = u;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        fA[q] = fx::to_float(sh(HA_NA + 3 * q + k));
        fB[q] = fx::to_float(sh(HA_NB + 3 * q + k));
        top = fx::imax(top, fx::imax(fA[q].k, fB[q].k));
        fA[q].k += 61 - num(HA_L + 8 * q).lo;
        fB[q].k += 61 - num(HA_V + 8 * q).lo;
        u = fx::imax(u, fx::imax(fA[q].k, fB[q].k));
      }
      if (ok && good_sum(top, u)) {
        fx::Num A[3], B[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          A[q] = fx::limbs(in_unit(fA[q], fA[q].k, u));
          B[q] = fx::limbs(in_unit(fB[q], fB[q].k, u));
        }
        if (live) a.sLdv[row(k * 8, E, e)] = 0.0;
#pragma unroll
        for (int c = 1; c < 8; ++c) {
          fx::Acc x = fx::mul(num(HA_L + c), A[0]);
          fx::mac(x, num(HA_V + c), B[0]);
#pragma unroll
          for (int q = 1; q < 3; ++q) {
            fx::mac(x, num(HA_L + 8 * q + c), A[q]);
            fx::mac(x, num(HA_V + 8 * q + c), B[q]);
          }
          if (live) a.sLdv[row(k * 8 + c, E, e)] = fx::to_double(fx::take<3>(x), u);
        }
      } else {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const int n = a.nodelist[c * E + e];
          const double l3[3] = {a.lfx[n], a.lfy[n], a.lfz[n]};
          const double v3_[3] = {a.xd0[n], a.yd0[n], a.zd0[n]};
          double t = 0.0;
#pragma unroll
          for (int q = 0; q < 3; ++q)
            t = fma(l3[q], sh(HA_NA + 3 * q + k), fma(v3_[q], sh(HA_NB + 3 * q + k), t));
          if (live) a.sLdv[row(k * 8 + c, E, e)] = t;
        }
      }
    }
    __syncthreads();
    if (live && k == 0) {
      // coef = c0 ss mass determ^(-1/3), vi12 = 1/(12 determ), determ = volo v
      const double c0 = -hgcoef * 0.01;
      const double Lc = (sh(HA_SUM) + sh(HA_SUM + 1)) + sh(HA_SUM + 2);
      const double Lvi12 = -coef * ((sh(HA_SUM + 3) + sh(HA_SUM + 4)) + sh(HA_SUM + 5));
      a.lss[e] += Lc * c0 * mass * r;
      Lhg_coef = Lc * (-0.01) * ss * mass * r;
      const double Ldeterm = (Lc * c0 * ss * mass * (-1.0 / 3.0) * r - Lvi12) * inv_det;
      a.lv[e] += Ldeterm * a.volo[e];
    }
  }
  // stress part of the force, f = s8 * B with s8 = (-p - q)/8. The forward
  // forms B0..B3 from faces 0-4 (node n's three face cross products) and
  // the opposite corners as B6 = -B0, B7 = -B1, B4 = -B2, B5 = -B3 (the face
  // normals of a closed surface sum to zero), so face 5 carries no adjoint:
  // sum_n lf_n . B_n = sum_f N_f . LU_f. The face terms LU go to sLU for
  // the position transpose; p and q get -1/8 sum_f N_f . LU_f here, before
  // the material transpose of the cycle before reads them.
  {
    // w_n = lf_n - lf_opposite(n) for the corners 0..3 (opposites 6, 7, 4, 5),
    // which touch faces {0,1,4} {0,1,2} {0,2,3} {0,3,4}
    const double w0 = lf[0] - lf[6], w1 = lf[1] - lf[7], w2 = lf[2] - lf[4], w3 = lf[3] - lf[5];
    const double w01 = w0 + w1, w23 = w2 + w3;
    double LU[5] = {w01 + w23, w01, w1 + w2, w23, w0 + w3};
    // src/domain.jl:1050-1055: node 1 (corner 0) takes face 5's areaY twice
    // and no areaZ; its opposite corner has the plain sum
    if (!(MODE & 1) && k != 0) LU[4] += k == 1 ? lf[0] : -lf[0];
    double part = 0.0;
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      // face normals 0..4 (the forward's cross products, from the tape)
      part = fma(a.geo[row(48 + 6 * k + f, E, e)], LU[f], part);
      if (live) a.sLU[row(3 * f + k, E, e)] = LU[f];
    }
    sh(HA_SUM + 6 + k) = part;
    __syncthreads();
    if (live && k == 1) {
      const double Lpq = -0.125 * ((sh(HA_SUM + 6) + sh(HA_SUM + 7)) + sh(HA_SUM + 8));
      a.lp[e] += Lpq;
      a.lq[e] += Lpq;
    }
  }
  // the block's sum over the cycles so far
  if (k == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) Lhg_coef += __shfl_down_sync(0xffffffffu, Lhg_coef, o);
    if (lane == 0) a.part_hg[blockIdx.x] += Lhg_coef;
  }
}

// Position transpose of one element's k_force, added into LX:
//  * the hourglass modes: Gamma^T of dL/dhm;
//  * the volume derivatives: the forward's dv is the gradient of 12*volume
//    (calcElemVolume's three triple products U.(V x W) of face diagonals), so
//    the transpose of G -> sum <G, dv> is the Hessian-vector product of those
//    triple products along G (the faithful slots 1 and 3 swapped back);
//  * the stress force f_n = s8 B_n with B_n the node's face-diagonal cross
//    products, through the face terms LU (see ka_hourglass).
// All three use the 12 face diagonals of the element (force order d20 d31
// d50 d14 d61 d25 d72 d36 d43 d07 d64 d57); the hourglass transpose of the
// same cycle left dL/dhm, dL/ddv and LU in sLhm, sLdv and sLU.
template <int MODE>
__device__ __forceinline__ void force_geo_t(const AdjDev& a, int e, const V3 dgs[12], double s8, double LX[3][8]) {
  const int E = a.E;
  const V3 d20 = dgs[0], d31 = dgs[1], d50 = dgs[2], d14 = dgs[3], d61 = dgs[4], d25 = dgs[5];
  const V3 d72 = dgs[6], d36 = dgs[7], d43 = dgs[8], d07 = dgs[9], d64 = dgs[10], d57 = dgs[11];
  // hourglass modes hm_k = Gamma(X_k)
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    double t[4], q[8];
#pragma unroll
    for (int m = 0; m < 4; ++m) t[m] = a.sLhm[row(k * 4 + m, E, e)];
    walsh_modes_t(t, q);
#pragma unroll
    for (int c = 0; c < 8; ++c) LX[k][c] = q[c];
  }
  auto add = [&](int c, const V3& v) { LX[0][c] += v.x; LX[1][c] += v.y; LX[2][c] += v.z; };
  auto sub = [&](int c, const V3& v) { LX[0][c] -= v.x; LX[1][c] -= v.y; LX[2][c] -= v.z; };
  // volume derivatives: Hessian-vector product of the triple products
  {
    double G[3][8];
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int c = 0; c < 8; ++c) G[j][c] = a.sLdv[row(j * 8 + c, E, e)];
    if (!(MODE & 2)) {
      // the faithful forward stores node 3's derivative in slot 1 and node 1's in slot 3
#pragma unroll
      for (int j = 0; j < 3; ++j) { const double t = G[j][1]; G[j][1] = G[j][3]; G[j][3] = t; }
    }
    auto gd = [&](int p, int q) { return v3(G[0][p] - G[0][q], G[1][p] - G[1][q], G[2][p] - G[2][q]); };
    auto hvp = [&](const V3& U, const V3& V, const V3& W, const V3& dU, const V3& dV, const V3& dW,
                   int u0, int u1, int u2, int u3, int v0, int v1, int w0, int w1) {
      V3 gU = vcross(dV, W); vadd(gU, vcross(V, dW));
      V3 gV = vcross(W, dU); vadd(gV, vcross(dW, U));
      V3 gW = vcross(dU, V); vadd(gW, vcross(U, dV));
      add(u0, gU); sub(u1, gU); add(u2, gU); sub(u3, gU);
      add(v0, gV); sub(v1, gV);
      add(w0, gW); sub(w1, gW);
    };
    // 12*volume = (d31 + d72).(d63 x d20) + (d43 + d57).(d64 x d70) + (d14 + d25).(d61 x d50)
    {
      V3 U = d31; vadd(U, d72);
      V3 dU = gd(3, 1); vadd(dU, gd(7, 2));
      const V3 V = v3(-d36.x, -d36.y, -d36.z);
      hvp(U, V, d20, dU, gd(6, 3), gd(2, 0), 3, 1, 7, 2, 6, 3, 2, 0);
    }
    {
      V3 U = d43; vadd(U, d57);
      V3 dU = gd(4, 3); vadd(dU, gd(5, 7));
      const V3 W = v3(-d07.x, -d07.y, -d07.z);
      hvp(U, d64, W, dU, gd(6, 4), gd(7, 0), 4, 3, 5, 7, 6, 4, 7, 0);
    }
    {
      V3 U = d14; vadd(U, d25);
      V3 dU = gd(1, 4); vadd(dU, gd(2, 5));
      hvp(U, d61, d50, dU, gd(6, 1), gd(5, 0), 1, 4, 2, 5, 6, 1, 5, 0);
    }
  }
  // stress part: with N_f = d1 x d2 for (d1, d2) = (p0 - p1, p2 - p3) of the
  // face's corners, sum_n lf_n . f_n = s8 sum_f N_f . LU_f
  {
    V3 LU[5];
#pragma unroll
    for (int f = 0; f < 5; ++f) LU[f] = v3(a.sLU[row(f * 3, E, e)], a.sLU[row(f * 3 + 1, E, e)], a.sLU[row(f * 3 + 2, E, e)]);
    auto face_t = [&](int f, const V3& d1, const V3& d2, int p0, int p1, int p2, int p3) {
      const V3 LN = v3(s8 * LU[f].x, s8 * LU[f].y, s8 * LU[f].z);
      const V3 L1 = vcross(d2, LN), L2 = vcross(LN, d1);
      add(p0, L1); sub(p1, L1); add(p2, L2); sub(p3, L2);
    };
    face_t(0, d20, d31, 2, 0, 3, 1);
    face_t(1, d50, d14, 5, 0, 1, 4);
    face_t(2, d61, d25, 6, 1, 2, 5);
    face_t(3, d72, d36, 7, 2, 3, 6);
    face_t(4, d43, d07, 4, 3, 0, 7);
  }
}

// The position transpose of the first cycle's k_force (the other cycles'
// is part of ka_kinematics of the cycle before), from the face diagonals
// taped at the segment's start (diag0), into the force corner buffer that
// ka_gather_corners sums.
template <int MODE>
__global__ void __launch_bounds__(kAdjBlock, 3) ka_force_geo(AdjDev a) {
  const int E = a.E;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= E) return;
  V3 dgs[12];
#pragma unroll
  for (int q = 0; q < 12; ++q) dgs[q] = v3(a.diag0[row(3 * q, E, e)], a.diag0[row(3 * q + 1, E, e)], a.diag0[row(3 * q + 2, E, e)]);
  const double s8 = ((-a.p0[e]) - a.q0[e]) * 0.125;
  double LX[3][8];
  force_geo_t<MODE>(a, e, dgs, s8, LX);
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int c = 0; c < 8; ++c) a.fX[row(k * 8 + c, E, e)] = LX[k][c];
}

// Sum of `n` partials in a fixed order by one block of BS threads; every
// thread gets it.
template <int BS>
__device__ double block_fixed_sum(const double* part, int n) {
  __shared__ double sh[BS];
  double s = 0.0;
  for (int j = threadIdx.x; j < n; j += BS) s += part[j];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int w = BS / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  const double r = sh[0];
  __syncthreads();
  return r;
}

// Sums `n` partials in a fixed order (one block).
__global__ void __launch_bounds__(kAdjBlock) ka_sum(const double* part, int n, double* out) {
  const double s = block_fixed_sum<kAdjBlock>(part, n);
  if (threadIdx.x == 0) *out = s;
}

// Copies the 11 state fields (node fields n < N, element fields n < E).
// A field whose destination is null is not copied (a tape set's per-cycle
// states keep only the fields the transposes read).
__device__ __forceinline__ void copy_state_at(int i, const StateSet& src, const StateSet& dst, int E, int N) {
  if (i < N) {
#pragma unroll
    for (int k = 0; k < 6; ++k)
      if (dst.f[k]) dst.f[k][i] = src.f[k][i];
  }
  if (i < E) {
#pragma unroll
    for (int k = 6; k < 11; ++k)
      if (dst.f[k]) dst.f[k][i] = src.f[k][i];
  }
}

__global__ void __launch_bounds__(kAdjBlock) ka_copy_state(StateSet src, StateSet dst, int E, int N) {
  copy_state_at(blockIdx.x * blockDim.x + threadIdx.x, src, dst, E, N);
}

// Start of a taped cycle: every thread copies the cycle's start state to its
// slot; thread 0 folds the previous cycle's minima, records timeIncrement!'s
// inputs, advances time and records the new dt. A run that has reached
// stoptime (the examples/benchmark.jl loop condition) or an earlier error
// makes the cycle a no-op (done / status, which the step kernels check).
__global__ void __launch_bounds__(kAdjBlock) ka_tape_begin(StateSet src, StateSet dst, int E, int N, DevState* st,
                                                            CycleRec* rec, Params prm) {
  wait_for_last_kernel();
  copy_state_at(blockIdx.x * blockDim.x + threadIdx.x, src, dst, E, N);
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  if (st->status != 0u || st->done) return;
  if (dt_registers(st->acc_courant)) st->dtcourant = __longlong_as_double((long long)st->acc_courant);
  if (dt_registers(st->acc_hydro)) st->dthydro = __longlong_as_double((long long)st->acc_hydro);
  st->acc_courant = kInfBits;
  st->acc_hydro = kInfBits;
  if (!(st->time < prm.stoptime)) { st->done = 1; return; }
  CycleRec r;
  r.time_prev = st->time;
  r.dt_prev = st->deltatime;
  r.dtc_in = st->dtcourant;
  r.dth_in = st->dthydro;
  r.cycle_prev = st->cycle;
  double time = st->time, dt = st->deltatime;
  long long cycle = st->cycle;
  time_increment(time, dt, cycle, st->dtcourant, st->dthydro, prm);
  st->time = time;
  st->deltatime = dt;
  st->cycle = cycle;
  r.dt = dt;
  r.active_c = r.active_h = 0;
  r.argmin_c = r.argmin_h = INT_MAX;
  *rec = r;
}

// End of a taped cycle: which minima the cycle reached, and the smallest
// element index attaining each (the element the reference's strict-less-than
// scan keeps, src/domain.jl:3003-3008 and :3041-3046).
__global__ void __launch_bounds__(kAdjBlock) ka_tape_close(const double* dtc, const double* dth, int E,
                                                            const DevState* st, CycleRec* rec) {
  wait_for_last_kernel();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned long long bc = st->acc_courant, bh = st->acc_hydro;
  if (i == 0) {
    rec->active_c = dt_registers(bc);
    rec->active_h = dt_registers(bh);
  }
  if (i >= E) return;
  if (dt_registers(bc) && (unsigned long long)__double_as_longlong(dtc[i]) == bc) atomicMin(&rec->argmin_c, i);
  if (dt_registers(bh) && (unsigned long long)__double_as_longlong(dth[i]) == bh) atomicMin(&rec->argmin_h, i);
}

// Loss seed and value: L = sum_e w_e e + sum_n 0.5 w_n |u|^2 with
// w_e = mask*elemMass, w_n = mask*nodalMass (masks from the reference mesh).
__global__ void __launch_bounds__(kAdjBlock) ka_loss_elem(const double* we, const double* e, int E, double* le,
                                                           double* part) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double s = 0.0;
  if (i < E) {
    s = we[i] * e[i];
    if (le) le[i] = we[i];
  }
  block_sum_to(s, part);
}

__global__ void __launch_bounds__(kAdjBlock) ka_loss_node(const double* wn, const double* xd, const double* yd,
                                                           const double* zd, int N, double* lxd, double* lyd,
                                                           double* lzd, double* part) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double s = 0.0;
  if (i < N) {
    const double w = wn[i], u = xd[i], v = yd[i], z = zd[i];
    s = 0.5 * w * fma(u, u, fma(v, v, z * z));
    if (lxd) { lxd[i] = w * u; lyd[i] = w * v; lzd[i] = w * z; }
  }
  block_sum_to(s, part);
}

}  // namespace lulesh
