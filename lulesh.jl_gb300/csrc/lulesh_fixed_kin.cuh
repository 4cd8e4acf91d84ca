// Kinematics of one element (volume, characteristic length, velocity
// divergence, monotonic-Q gradients; src/domain.jl:1874-2320) in the
// fixed-point arithmetic of lulesh_fixed.cuh, by three threads, one per
// coordinate, as lulesh_fixed_force.cuh does the forces.
//
// A thread converts its coordinate's positions and velocities, forms its
// component of every cross product and its terms of every dot product; the
// terms are added in shared memory and the roots and quotients, in FP64, are
// divided among the three.
#pragma once

#include "lulesh_fixed.cuh"

namespace lulesh {
namespace fx {

enum : int {
  KS_GEO = 0,    // 18 k + q: limbs of diagonal q (12), mean edge (3), half-step edge (3) of coordinate k
  KS_SUM = 0,    // kSums k + i: coordinate k's terms, over the diagonals once those are read
  KS_DET = 57,   // k: a term of the Jacobian determinant
  KS_EXT = 60,   // k: exponent fields of the position and velocity extents
  KS_MID = 63,   // 1/(64 volume), then the divergence's factor and the divergence
  KS_COUNT = 66
};
// sums over the coordinates
enum : int {
  SUM_VOLUME = 0,  // 12 volume over 2^62
  SUM_FACE = 1,    // 6: squared face vectors over 2^61, force order
  SUM_AREA = 7,    // 3: squared cross products of the mean edges over 2^61
  SUM_FLOW = 10,   // 3: those cross products times velocity differences
  SUM_RATE = 13,   // cofactors times velocity differences
  SUM_JAC = 14,    // half-step determinant
  SUM_EXPO = 15,   // 4: exponents of flow d (low word) and area d (high word); the rate's, and over 2^8 the faces', with the
                   // determinant's below
  kSums = 19
};
// exponent of a term that is exactly zero
constexpr int kNoTerm = -16384;
static_assert(3 * kSums <= KS_DET, "the sums overlay the diagonals");

// What a thread keeps over the phases: its components (unscaled integers) of
// the face vectors, the volume's V x W, the edges' cross products (over
// 2^(64 - up)), the cofactors (over 2^62), and its velocity differences and
// edges. A component of a cross product is in the other two coordinates' units,
// a triple product in all three, whichever the component.
struct KinLane {
  double x[8], v[8];
  int s, sv, all;  // scales of this coordinate's positions and velocities; sum of the three positions'
  int least;       // the least determinant is 2^least
  int up[3];
  bool ok_x, ok;  // positions taken; positions and velocities taken
  i64 g[12], w[3], vw[3];
  i64 n[6], gU[3], A[3], C[3];
  Num half_eta;
};

// a^2 over 2^61; all four limb products, as the squares of the low limbs do
// not average out
LULESH_FX i64 square(Num a) {
  const i64 h = mulw(a.hi, a.hi), m = mulw(a.hi, a.lo);
  const u64 l = (u64)mulw(a.lo, a.lo);
  return shl(h, 3) + ((m + (i64)(l >> 33)) >> 28);
}

// 1: r.x and r.v hold coordinate k's corner values.
LULESH_FX void kin_extents(int k, Slots sh, const KinLane& r) {
  Num m;
  extent_fields(r.x, r.v, m.lo, m.hi);
  sh[KS_EXT + k] = m;
}

// 2: diagonals, mean edges, velocity differences and half-step edges (edge -
// dt/2 velocity difference, half_dt = dt/2). Each coordinate's positions and
// velocities have their own scale: a thin element keeps its thin direction's
// bits, and in flow along one axis the others' differences, which alone make up
// the monotonic-Q gradients across it, are as small as they please.
LULESH_FX void kin_edges(int k, Slots sh, double half_dt, KinLane& r, Range range = narrow()) {
  const Num m0 = sh[KS_EXT], m1 = sh[KS_EXT + 1], m2 = sh[KS_EXT + 2];
  const Scales s = scales_of(m0.lo, m1.lo, m2.lo, range);
  r.ok_x = s.ok;
  r.s = k == 0 ? s.s[0] : k == 1 ? s.s[1] : s.s[2];
  r.all = s.s[0] + s.s[1] + s.s[2];
  r.least = s.least(range.kin_det, range);
  int ev[3] = {m0.hi, m1.hi, m2.hi};
  const bool wild = imax(ev[0], imax(ev[1], ev[2])) > kMaxSpeed;  // not finite, or far beyond any flow
  int fastest = kNoExponent;
  LULESH_UNROLL
  for (int j = 0; j < 3; ++j) {
    ev[j] = imax(ev[j], kMinSpeed);
    fastest = imax(fastest, s.s[j] - 1083 + ev[j]);
  }
  r.sv = 1083 - (k == 0 ? ev[0] : k == 1 ? ev[1] : ev[2]);
  // dt/2 in units of the edges over those of the velocities, T.m 2^tx: taken
  // while corners move less than an eighth of the scale's 2^61
  const Float T = to_float(half_dt);
  const int tx = T.k + r.s - r.sv;
  r.ok = r.ok_x && !wild && T.k + fastest <= -64 && exponent_field((unsigned)hi_word(half_dt)) != 0x7ff;
  const Num tau = limbs(T.m >> (r.ok ? imin(-64 - tx, 63) : 63));
  i64 c[8];
  LULESH_UNROLL
  for (int i = 0; i < 8; ++i) c[i] = to_fixed(r.x[i], r.s - 1075);
  diagonals(c, r.g);
  walsh(c, r.w, nullptr);
  LULESH_UNROLL
  for (int i = 0; i < 8; ++i) c[i] = to_fixed0(r.v[i], r.sv - 1075);
  walsh(c, r.vw, nullptr);
  const int at = KS_GEO + 18 * k;
  LULESH_UNROLL
  for (int q = 0; q < 12; ++q) sh[at + q] = limbs(r.g[q]);
  LULESH_UNROLL
  for (int a = 0; a < 3; ++a) {
    sh[at + 12 + a] = limbs(r.w[a]);
    const Num h = limbs(r.w[a] - product(limbs(r.vw[a]), tau));
    sh[at + 15 + a] = h;
    if (a == 1) r.half_eta = h;
  }
}

// 3: component k of the cross products; i1, i2 the slots of the next two
// coordinates. Reads the diagonals, so a barrier separates it from 4.
LULESH_FX void kin_products(int k, Slots sh, KinLane& r) {
  const int i1 = KS_GEO + 18 * (k == 2 ? 0 : k + 1), i2 = KS_GEO + 18 * (k == 0 ? 2 : k - 1);
  auto cross_k = [&](int a, int b) {
    return take<0>(mul_minus(sh[i1 + a], sh[i2 + b], sh[i2 + a], sh[i1 + b]));
  };
  LULESH_UNROLL
  for (int f = 0; f < 6; ++f) r.n[f] = cross_k(2 * f, 2 * f + 1);
  // V x W of the three products: (-g7, g0), (g10, -g9), (g4, g2)
  r.gU[0] = cross_k(0, 7);
  r.gU[1] = cross_k(9, 10);
  r.gU[2] = cross_k(4, 2);
  // eta x zeta, zeta x xi, xi x eta of the mean edges and of the half-step edges
  LULESH_UNROLL
  for (int d = 0; d < 3; ++d) {
    const int a = 12 + (d + 1) % 3, b = 12 + (d + 2) % 3;
    r.A[d] = take_all(mul_minus_full(sh[i1 + a], sh[i2 + b], sh[i2 + a], sh[i1 + b]), r.up[d]);
    r.C[d] = take<2>(mul_minus(sh[i1 + a + 3], sh[i2 + b + 3], sh[i2 + a + 3], sh[i1 + b + 3]));
  }
  sh.put(KS_DET + k, product(limbs(r.w[1]), limbs(r.A[1] >> r.up[1])));
}

// 4: coordinate k's terms of the sums.
LULESH_FX void kin_terms(int k, Slots sh, const KinLane& r) {
  const int at = KS_SUM + kSums * k;
  {
    Acc a = {0, 0};
    mac_full(a, limbs(r.g[1] + r.g[6]), limbs(r.gU[0]));
    mac_full(a, limbs(r.g[8] + r.g[11]), limbs(r.gU[1]));
    mac_full(a, limbs(r.g[3] + r.g[5]), limbs(r.gU[2]));
    sh.put(at + SUM_VOLUME, take<2>(a));
  }
  // The terms of the other sums differ in scale by coordinate: each is brought
  // to 2^60 and carries its exponent, and the sum takes the largest's. (Of the
  // faces only the largest counts: a coordinate's six share an exponent.)
  const int two = r.all - r.s;
  Num last;
  {
    unsigned used = 0;
    LULESH_UNROLL
    for (int f = 0; f < 6; ++f) {
      const int h = (int)(r.n[f] >> 32);
      used |= (unsigned)(h ^ (h >> 31));
    }
    const int c = imax(leading_zeros(used) - 3, 0);
    LULESH_UNROLL
    for (int f = 0; f < 6; ++f) sh.put(at + SUM_FACE + f, square(limbs(shl(r.n[f], c))));
    last.hi = -2 * (two + c);
  }
  auto put_term = [&](int i, i64 t, int shift) {
    const int c = room(t);
    sh.put(at + i, shl(t, c));
    return t != 0 ? -(r.sv + two + shift + c) : kNoTerm;
  };
  Acc rate = {0, 0};
  LULESH_UNROLL
  for (int d = 0; d < 3; ++d) {
    const Num a = limbs(r.A[d]), u = limbs(r.vw[d]), c = limbs(r.C[d]);
    sh.put(at + SUM_AREA + d, square(a));
    Num e;
    e.hi = -2 * (two + r.up[d]);  // (with up 29 and scales within 2^28 of one another, zeros stay below the rest)
    Acc flow = {0, 0};
    mac_full(flow, a, u);
    e.lo = put_term(SUM_FLOW + d, take<3>(flow), r.up[d]);
    sh[at + SUM_EXPO + d] = e;
    mac_full(rate, c, u);
  }
  last.lo = put_term(SUM_RATE, take<1>(rate), 0);
  Acc jac = {0, 0};
  mac_full(jac, r.half_eta, limbs(r.C[1]));
  int c;
  sh.put(at + SUM_JAC, take_all(jac, c));
  last.hi = (int)((unsigned)last.hi << 8) | c;
  sh[at + SUM_EXPO + 3] = last;
}

LULESH_FX i64 kin_sum(Slots sh, int i) {
  return add(add(sh.get(KS_SUM + i), sh.get(KS_SUM + kSums + i)), sh.get(KS_SUM + 2 * kSums + i));
}

// the sum of the terms with exponents e, times 2^k
LULESH_FX double kin_aligned(Slots sh, int sum, int e0, int e1, int e2, int k) {
  const int top = imax(e0, imax(e1, e2));
  const i64 t = (sh.get(KS_SUM + sum) >> imin(top - e0, 63)) + (sh.get(KS_SUM + kSums + sum) >> imin(top - e1, 63)) +
                (sh.get(KS_SUM + 2 * kSums + sum) >> imin(top - e2, 63));
  return to_double(t, k + top);
}
LULESH_FX Num kin_expo(Slots sh, int j, int d) { return sh[KS_SUM + kSums * j + SUM_EXPO + d]; }

LULESH_FX i64 kin_determinant(Slots sh) { return sh.get(KS_DET) + sh.get(KS_DET + 1) + sh.get(KS_DET + 2); }

// 5: whether the element is taken (by its determinant and volume too), and the
// sums in FP64 with their true scales.
LULESH_FX bool kin_positions_taken(Slots sh, const KinLane& r) {
  return r.ok_x && kin_determinant(sh) >= shl(1, r.least);
}
LULESH_FX void kin_accept(Slots sh, KinLane& r) {
  r.ok_x = kin_positions_taken(sh, r);
  r.ok = r.ok && r.ok_x && kin_sum(sh, SUM_VOLUME) >= shl(1, r.least + 4);
}
LULESH_FX double kin_volume12(Slots sh, const KinLane& r) { return to_double(kin_sum(sh, SUM_VOLUME), 126 - r.all); }
// the largest squared face vector and its place in the reference's face order
// (0, 5, 1, 2, 3, 4 of the force order)
LULESH_FX double kin_largest_face(Slots sh, const KinLane& r, int& place) {
  const int e0 = kin_expo(sh, 0, 3).hi >> 8, e1 = kin_expo(sh, 1, 3).hi >> 8, e2 = kin_expo(sh, 2, 3).hi >> 8;
  const int top = imax(e0, imax(e1, e2));
  const int d0 = imin(top - e0, 63), d1 = imin(top - e1, 63), d2 = imin(top - e2, 63);
  i64 best = -1;
  place = 0;
  LULESH_UNROLL
  for (int q = 0; q < 6; ++q) {
    const int f = SUM_FACE + (q == 0 ? 0 : q == 1 ? 5 : q - 1);
    const i64 a = (sh.get(KS_SUM + f) >> d0) + (sh.get(KS_SUM + kSums + f) >> d1) + (sh.get(KS_SUM + 2 * kSums + f) >> d2);
    if (a > best) {
      best = a;
      place = q;
    }
  }
  return to_double(best, 189 + top);
}
LULESH_FX double kin_area(Slots sh, const KinLane&, int d) {
  return kin_aligned(sh, SUM_AREA + d, kin_expo(sh, 0, d).hi, kin_expo(sh, 1, d).hi, kin_expo(sh, 2, d).hi, 197);
}
LULESH_FX double kin_flow(Slots sh, const KinLane&, int d) {
  return kin_aligned(sh, SUM_FLOW + d, kin_expo(sh, 0, d).lo, kin_expo(sh, 1, d).lo, kin_expo(sh, 2, d).lo, 131);
}
LULESH_FX double kin_rate(Slots sh, const KinLane&) {
  return kin_aligned(sh, SUM_RATE, kin_expo(sh, 0, 3).lo, kin_expo(sh, 1, 3).lo, kin_expo(sh, 2, 3).lo, 131);
}
// coordinate k's part of it
LULESH_FX double kin_own_rate(Slots sh, const KinLane&, int k) {
  return to_double(sh.get(KS_SUM + kSums * k + SUM_RATE), 131 + kin_expo(sh, k, 3).lo);
}
LULESH_FX double kin_jacobian(Slots sh, const KinLane& r) {
  auto e = [&](int j) { return -(kin_expo(sh, j, 3).hi & 0xff); };
  return kin_aligned(sh, SUM_JAC, e(0), e(1), e(2), 132 - r.all);
}

}  // namespace fx
}  // namespace lulesh
