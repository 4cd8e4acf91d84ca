// The force and kinematics phases of lulesh_fixed_force.cuh and
// lulesh_fixed_kin.cuh in FP64, for the elements the fixed-point form does not
// take: inverted, flat or not finite ones, whose volume errors these record, turned
// slender ones (kinematics), and numbers outside 2^-400..2^400.
//
// The same three threads, slots and barriers: a thread's component takes about
// 190 FP64 slots (forces) or 110 (kinematics), 6 and 4 us for a block that has
// such an element; one thread for the whole element took 18.
#pragma once

#include "lulesh_device.cuh"
#include "lulesh_fixed_force.cuh"
#include "lulesh_fixed_kin.cuh"

namespace lulesh {

// One element's column of slots as doubles.
struct RealSlots {
  double* p;
  int stride;
  __device__ __forceinline__ double& operator[](int i) const { return p[i * stride]; }
};

// The face diagonals of one coordinate, as fx::diagonals.
__device__ __forceinline__ void diagonals_fp64(const double v[8], double g[12]) {
  constexpr int pa[12] = {2, 3, 5, 1, 6, 2, 7, 3, 4, 0, 6, 5};
  constexpr int pb[12] = {0, 1, 0, 4, 1, 5, 2, 6, 3, 7, 4, 7};
#pragma unroll
  for (int q = 0; q < 12; ++q) g[q] = v[pa[q]] - v[pb[q]];
}

// Component k of the cross product of the vectors in slots a and b (i1, i2:
// where the next two coordinates' slots begin).
__device__ __forceinline__ double cross_fp64(const RealSlots& sh, int i1, int i2, int a, int b) {
  return fma(sh[i1 + a], sh[i2 + b], -sh[i2 + a] * sh[i1 + b]);
}

struct ForceScalars {
  double v, vi12, coef, s8;
  bool hourglass;  // hgcoef > 0
};

// Every thread of the block calls this; `mine` marks the threads of elements
// it is for. x, v: corner positions and velocities of coordinate k. out(n,
// value), tape and errors as in the fixed-point phases.
template <int MODE, class Out, class Tape>
__device__ __forceinline__ void force_fp64(int k, const RealSlots& sh, const double x[8], const double v[8],
                                           const ForceScalars& c, bool mine, unsigned* status, Out out, Tape tape) {
  using namespace fx;
  const int at = FS_GEO + 18 * k, i1 = FS_GEO + 18 * (k == 2 ? 0 : k + 1), i2 = FS_GEO + 18 * (k == 0 ? 2 : k - 1);
  double hm[4], w1;
  {
    double g[12];
    diagonals_fp64(x, g);
#pragma unroll
    for (int q = 0; q < 12; ++q) sh[at + q] = g[q];
    sh[at + 12] = g[1] + g[6];
    sh[at + 13] = g[8] + g[11];
    sh[at + 14] = g[3] + g[5];
    const double a = x[6] - x[0], b = x[5] - x[3], cc = x[7] - x[1], dd = x[4] - x[2];
    const double apb = a + b, cpd = cc + dd, amb = a - b, cmd = cc - dd;
    w1 = amb + cmd;
    sh[at + 15] = apb - cpd;
    sh[at + 16] = w1;
    sh[at + 17] = apb + cpd;
    hm[0] = (g[10] - g[11]) - (g[0] + g[1]);
    const double pp = g[9] + g[4], qq = g[8] + g[5];
    hm[1] = pp - qq;
    hm[2] = pp + qq;
    hm[3] = amb - cmd;
  }
  __syncthreads();
  auto cr = [&](int a, int b) { return cross_fp64(sh, i1, i2, a, b); };
  double B[4], B0;
  {
    double n[5];
#pragma unroll
    for (int f = 0; f < 5; ++f) n[f] = cr(2 * f, 2 * f + 1);
    const double p01 = n[0] + n[1];
    B[0] = p01 + n[4];
    B[1] = p01 + n[2];
    B[2] = (n[0] + n[2]) + n[3];
    B[3] = (n[0] + n[3]) + n[4];
    B0 = (MODE & 1) || k == 0 ? B[0] : k == 1 ? B[0] + n[4] : p01;
  }
  {
    const double u0 = cr(0, 7), v0 = cr(0, 12), w0 = cr(7, 12);
    const double u1 = cr(9, 10), v1 = cr(13, 9), w1_ = cr(13, 10);
    const double u2 = cr(4, 2), v2 = cr(2, 14), w2 = cr(14, 4);
    const double t12 = u2 - u0, t37 = u0 - u1, t45 = u1 - u2;
    const double dv[8] = {-((w0 + w1_) + w2), t12 - v2, t12 + w0, t37 - v0, t45 - v1, t45 + w2, (v0 + v1) + v2, t37 + w1_};
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int src = (MODE & 2) ? n : (n == 1 ? 3 : n == 3 ? 1 : n);
      sh[FS_DV + 12 * k + n] = dv[src];
      if (Tape::on && mine && c.hourglass) tape.derivative(k, n, dv[src]);
    }
  }
  sh[FS_DET + k] = w1 * cr(17, 15);
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const double h = hm[m] * c.vi12;
    sh[FS_DV + 12 * k + 8 + m] = h;
    if (Tape::on && mine && c.hourglass) tape.mode(k, m, h);
  }
  __syncthreads();
  if (mine && k == 0) {
    if (le_zero(sh[FS_DET] + sh[FS_DET + 1] + sh[FS_DET + 2])) atomicOr(status, ST_EARLY);
    if (le_zero(c.v)) atomicOr(status, ST_HOURGLASS);
  }
#pragma unroll
  for (int j = 0; j < 11; ++j) {
    const int i = 3 * j + k, n = (i >> 2) & 7, m = i & 3;
    const double gam = (kGammaSigns >> (i & 31)) & 1u ? -1.0 : 1.0;
    const double g = fma(-sh[FS_DV + 24 + n], sh[FS_DV + 32 + m],
                         fma(-sh[FS_DV + 12 + n], sh[FS_DV + 20 + m], fma(-sh[FS_DV + n], sh[FS_DV + 8 + m], gam)));
    if (i < 32) sh[FS_HG + i] = g;
  }
  __syncthreads();
  if (!mine) return;
  double h[4] = {0.0, 0.0, 0.0, 0.0};
  if (c.hourglass) {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      double s = sh[FS_HG + m] * v[0];
#pragma unroll
      for (int n = 1; n < 8; ++n) s = fma(sh[FS_HG + 4 * n + m], v[n], s);
      if (Tape::on) tape.sum(k, m, s);
      h[m] = c.coef * s;
    }
  }
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    double f = c.s8 * (n == 0 ? B0 : n < 4 ? B[n] : -B[n == 4 ? 2 : n == 5 ? 3 : n == 6 ? 0 : 1]);
    if (c.hourglass)
#pragma unroll
      for (int m = 3; m >= 0; --m) f = fma(sh[FS_HG + 4 * n + m], h[m], f);
    out(n, f);
  }
}

// What the quotients of an element's kinematics are formed from.
struct KinSums {
  double volume12;      // 12 * volume
  double face;          // the largest squared face vector
  int place;            // its place in the reference's face order
  double area, flow;    // direction k: squared cross product of the edges, its product with the velocity difference
  double rate, jacobian;
  double own_rate;      // coordinate k's part of the rate
};

// Coordinate k's taped components.
struct KinTaped {
  double g[12], w[3], vw[3], n[6], gU[3], A[3], C[3];
};

// Every thread of the block calls this.
__device__ __forceinline__ void kin_fp64(int k, const RealSlots& sh, const double x[8], const double v[8], double dt,
                                         KinSums& s, KinTaped& t) {
  using namespace fx;
  const int at = KS_GEO + 18 * k, i1 = KS_GEO + 18 * (k == 2 ? 0 : k + 1), i2 = KS_GEO + 18 * (k == 0 ? 2 : k - 1);
  double half[3];
  diagonals_fp64(x, t.g);
  walsh1(x, t.w);
  walsh1(v, t.vw);
#pragma unroll
  for (int q = 0; q < 12; ++q) sh[at + q] = t.g[q];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    half[a] = fma(-0.5 * dt, t.vw[a], t.w[a]);
    sh[at + 12 + a] = t.w[a];
    sh[at + 15 + a] = half[a];
  }
  __syncthreads();
  auto cr = [&](int a, int b) { return cross_fp64(sh, i1, i2, a, b); };
#pragma unroll
  for (int f = 0; f < 6; ++f) t.n[f] = cr(2 * f, 2 * f + 1);
  t.gU[0] = cr(0, 7);
  t.gU[1] = cr(9, 10);
  t.gU[2] = cr(4, 2);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    t.A[a] = cr(12 + (a + 1) % 3, 12 + (a + 2) % 3);
    t.C[a] = cr(15 + (a + 1) % 3, 15 + (a + 2) % 3);
  }
  __syncthreads();
  const int to = KS_SUM + kSums * k;
  sh[to + SUM_VOLUME] = fma(t.g[1] + t.g[6], t.gU[0], fma(t.g[8] + t.g[11], t.gU[1], (t.g[3] + t.g[5]) * t.gU[2]));
#pragma unroll
  for (int f = 0; f < 6; ++f) sh[to + SUM_FACE + f] = t.n[f] * t.n[f];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    sh[to + SUM_AREA + a] = t.A[a] * t.A[a];
    sh[to + SUM_FLOW + a] = t.A[a] * t.vw[a];
  }
  s.own_rate = fma(t.C[0], t.vw[0], fma(t.C[1], t.vw[1], t.C[2] * t.vw[2]));
  sh[to + SUM_RATE] = s.own_rate;
  sh[to + SUM_JAC] = half[1] * t.C[1];
  __syncthreads();
  auto sum = [&](int i) { return (sh[KS_SUM + i] + sh[KS_SUM + kSums + i]) + sh[KS_SUM + 2 * kSums + i]; };
  s.volume12 = sum(SUM_VOLUME);
  s.face = 0.0;
  s.place = 0;
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    // squares and their sums are >= +0: their bit patterns order them
    const double a = sum(SUM_FACE + (q == 0 ? 0 : q == 1 ? 5 : q - 1));
    if (q == 0 || __double_as_longlong(a) > __double_as_longlong(s.face)) {
      s.face = a;
      s.place = q;
    }
  }
  s.area = sum(SUM_AREA + k) + 256.e-36;
  s.flow = sum(SUM_FLOW + k);
  s.rate = sum(SUM_RATE);
  s.jacobian = sum(SUM_JAC);
}

}  // namespace lulesh
