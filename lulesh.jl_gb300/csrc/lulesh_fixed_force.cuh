// Corner forces of one element (stress plus Flanagan-Belytschko hourglass,
// src/domain.jl:1069-1110 and 1258-1694) in the fixed-point arithmetic of
// lulesh_fixed.cuh, by three threads, one per coordinate.
//
// A thread converts its coordinate's positions and velocities, forms its
// component of every cross product, of the node normals and of the volume
// derivatives, a third of the hourglass base vectors, and its component of
// the forces; diagonals, derivatives and base vectors change hands in shared
// memory. Beside one thread for the whole element (4,800 instructions and 204
// registers) the work is the same, but a warp's instruction stream is a third
// as long and its registers allow twice the warps, which is what bounds this
// integer code: dependent wide multiply-adds are 8 to 16 cycles apart and
// straight-line instructions have to be fetched.
//
// The phases are written for one (element, coordinate) each, with a barrier
// of the element's three threads between them.
#pragma once

#include "lulesh_fixed.cuh"

namespace lulesh {
namespace fx {

// gamma of calcFBHourglassForceForElems (src/domain.jl:1490-1499): bit 4 n + m
// is set where entry m of corner n's hourglass base vector is -1.
constexpr unsigned gamma_signs() {
  unsigned r = 0;
  for (int n = 0; n < 8; ++n)
    for (int m = 0; m < 4; ++m) {
      const bool x = n == 1 || n == 2 || n == 5 || n == 6, y = n == 2 || n == 3 || n == 6 || n == 7, z = n >= 4;
      const bool neg = m == 0 ? y != z : m == 1 ? x != z : m == 2 ? x != y : !((x != y) != z);
      if (neg) r |= 1u << (4 * n + m);
    }
  return r;
}
constexpr unsigned kGammaSigns = gamma_signs();

// A finite double that is zero or has a magnitude in 2^-400 .. 2^400.
LULESH_FX bool ordinary(double x) {
  const unsigned h = (unsigned)hi_word(x) & 0x7fffffffu;
  return (h | lo_word(x)) == 0u || (h >= ((unsigned)kMinSpeed << 20) && h < ((unsigned)(kMaxSpeed + 1) << 20));
}

enum : int {
  FS_GEO = 0,      // 18 k + q: limbs of diagonal q (12), U vector (3), mean edge (3) of coordinate k
  FS_HG = 0,       // 4 n + m: limbs of the base vectors, over the diagonals once those are read
  FS_DV = 54,      // 12 k + n: limbs of the volume derivatives (8) and scaled modes (4)
  FS_EXT = 90,     // k: extent's exponent field; whether the velocities are out of range
  FS_USED = 93,    // k: bits used by the modes' high words
  FS_K = 96,       // mantissas of 1/(12 determ), the coefficient and the stress, then their exponents
  FS_C = 97,
  FS_S = 98,
  FS_EXPO = 99,    // K.k and C.k; Sg.k and whether the scalars are in range
  FS_DET = 101,    // k: a term of the Jacobian determinant
  FS_SMALL = 104,  // k: bits used by the derivatives' high words, where the base vectors outgrow their scale
  FS_COUNT = 107
};

// places the base vectors may outgrow their scale by at the cost of their last bits
constexpr int kFewPlaces = 1;

// What a thread keeps over the phases.
struct ForceLane {
  double x[8];
  Num V[8];
  int ev, s, all, q;  // (s: this coordinate's scale, all: the sum of the three)
  int least;          // the least determinant is 2^least
  bool ok;
  i64 w1;
  Num B[4], B0;
};

// 1: positions x and velocities v of coordinate k.
LULESH_FX void force_load(int k, Slots sh, const double v[8], ForceLane& r) {
  int ev;
  Num m;
  extent_fields(v, r.x, ev, m.lo);
  const bool wild = ev > kMaxSpeed;  // not finite, or far beyond any flow
  r.ev = wild ? 0x7ff : imax(ev, kMinSpeed);
  const i64 v0 = to_fixed(v[0], 7 - r.ev);
  LULESH_UNROLL
  for (int n = 1; n < 8; ++n) r.V[n] = limbs(sub(to_fixed(v[n], 7 - r.ev), v0));
  m.hi = wild;
  sh[FS_EXT + k] = m;
}
// 1, by one thread: vi12 = 1 / (12 volo v) and the hourglass coefficient (0
// for none); by another, s8 = (-p - q) / 8.
LULESH_FX void force_scales(Slots sh, double vi12, double coef) {
  const Float K = to_float(vi12), C = to_float(coef);
  sh.put(FS_K, K.m);
  sh.put(FS_C, C.m);
  Num e;
  e.lo = K.k;
  // an exponent no ordinary number has marks an element that is not taken
  e.hi = K.m > 0 && ordinary(vi12) && ordinary(coef) ? C.k : 1 << 20;
  sh[FS_EXPO] = e;
}
LULESH_FX void force_stress(Slots sh, double s8) {
  const Float S = to_float(s8);
  sh.put(FS_S, shl(S.m, 1));
  Num e;
  e.lo = S.k - 1;
  e.hi = ordinary(s8);
  sh[FS_EXPO + 1] = e;
}

// 2: the coordinate's diagonals, U vectors, mean edges and hourglass modes.
LULESH_FX void force_diagonals(int k, Slots sh, ForceLane& r, i64 hm[4], Range range = narrow()) {
  const Num m0 = sh[FS_EXT], m1 = sh[FS_EXT + 1], m2 = sh[FS_EXT + 2];
  const Scales s = scales_of(m0.lo, m1.lo, m2.lo, range);
  r.ok = s.ok && (m0.hi | m1.hi | m2.hi) == 0 && sh[FS_EXPO].hi != 1 << 20 && sh[FS_EXPO + 1].hi != 0;
  r.s = k == 0 ? s.s[0] : k == 1 ? s.s[1] : s.s[2];
  r.all = s.s[0] + s.s[1] + s.s[2];
  r.least = s.least(range.force_det, range);
  i64 v[8], g[12], w[3];
  LULESH_UNROLL
  for (int c = 0; c < 8; ++c) v[c] = to_fixed(r.x[c], r.s - 1075);
  diagonals(v, g);
  walsh(v, w, &hm[3]);
  even_modes(g, hm);
  r.w1 = w[1];
  const int at = FS_GEO + 18 * k;
  LULESH_UNROLL
  for (int q = 0; q < 12; ++q) sh[at + q] = limbs(g[q]);
  sh[at + 12] = limbs(g[1] + g[6]);
  sh[at + 13] = limbs(g[8] + g[11]);
  sh[at + 14] = limbs(g[3] + g[5]);
  LULESH_UNROLL
  for (int a = 0; a < 3; ++a) sh[at + 15 + a] = limbs(w[a]);
  unsigned used = 0;
  LULESH_UNROLL
  for (int m = 0; m < 4; ++m) {
    const int h = (int)(hm[m] >> 32);
    used |= (unsigned)(h ^ (h >> 31));
  }
  Num u;
  u.lo = (int)used;
  u.hi = 0;
  sh[FS_USED + k] = u;
}

// 3: component k of the cross products: node normals (times -8) of corners
// 0..3 as sums of their faces' diagonal cross products (corners 6, 7, 4, 5 are
// minus corners 0, 1, 2, 3), volume derivatives in the reference's slots (node
// 3's in slot 1 and node 1's in slot 3 unless MODE bit 1), the determinant of
// the mean edges, and the scaled modes.
//
// Each coordinate's positions have their own scale: a cross product's component
// is in the other two's units, derivative * mode and the determinant in all
// three, whichever the component. A thin element's forces along its thin
// direction, and across it, keep their bits.
//
// The modes are scaled by 1/(12 determ) so that derivative * mode is in units
// 2^(q - 58) of the base vectors. The scale's exponent L is taken as a left
// shift of the modes as far as they leave room (below 2^61) and, up to 4
// places, of the product; q is 0 unless the distortion needs more, and more
// than the range has is left to the FP64 form. A derivative is at most 3 E^2 (its bilinear
// form over the corners of a box), below 2^59.6, so the base vectors stay
// below 2^59.8. Where q is more than a few places, what the derivatives leave of that
// is taken off it in phase 4: a slender element's are as far below its box's areas as its base
// vectors' terms are above their scale.
template <int MODE, class Tape>
LULESH_FX void force_products(int k, Slots sh, ForceLane& r, const i64 hm[4], Tape tape, Range range = narrow()) {
  const int i1 = FS_GEO + 18 * (k == 2 ? 0 : k + 1), i2 = FS_GEO + 18 * (k == 0 ? 2 : k - 1);
  auto cross_k = [&](int a, int b) {
    return take<0>(mul_minus(sh[i1 + a], sh[i2 + b], sh[i2 + a], sh[i1 + b]));
  };
  {
    i64 n[5];
    LULESH_UNROLL
    for (int f = 0; f < 5; ++f) n[f] = cross_k(2 * f, 2 * f + 1);
    const i64 p01 = n[0] + n[1], p03 = n[0] + n[3], p014 = p01 + n[4];
    r.B[0] = limbs(p014);
    r.B[1] = limbs(p01 + n[2]);
    r.B[2] = limbs(p03 + n[2]);
    r.B[3] = limbs(p03 + n[4]);
    // corner 0 takes face 4's y area twice and its z area not at all in the
    // reference (MODE bit 0 clear)
    r.B0 = (MODE & 1) ? r.B[0] : limbs(k == 0 ? p014 : k == 1 ? p014 + n[4] : p01);
  }
  {
    // V, W of the three products: (-g7, g0), (g10, -g9), (g4, g2)
    const i64 u0 = cross_k(0, 7), v0 = cross_k(0, 12), w0 = cross_k(7, 12);
    const i64 u1 = cross_k(9, 10), v1 = cross_k(13, 9), w1 = cross_k(13, 10);
    const i64 u2 = cross_k(4, 2), v2 = cross_k(2, 14), w2 = cross_k(14, 4);
    const i64 t12 = u2 - u0, t37 = u0 - u1, t45 = u1 - u2;
    const i64 d[8] = {-((w0 + w1) + w2), t12 - v2, t12 + w0, t37 - v0, t45 - v1, t45 + w2, (v0 + v1) + v2, t37 + w1};
    LULESH_UNROLL
    for (int n = 0; n < 8; ++n) {
      const int src = (MODE & 2) ? n : (n == 1 ? 3 : n == 3 ? 1 : n);
      sh[FS_DV + 12 * k + n] = limbs(d[src]);
      if (Tape::on) tape.derivative(k, n, to_double(d[src], 64 - (r.all - r.s)));
    }
  }
  sh.put(FS_DET + k, product(limbs(r.w1), limbs(cross_k(17, 15))));

  const Num expo = sh[FS_EXPO];
  const unsigned modes_used = (unsigned)(sh[FS_USED].lo | sh[FS_USED + 1].lo | sh[FS_USED + 2].lo);
  const int room = leading_zeros(modes_used) - 3, L = expo.lo + 252 - r.all;
  r.q = imax(L - (room + 4), 0);
  r.ok = r.ok && L >= 0 && r.q <= range.distortion;
  r.q = r.ok ? r.q : 0;
  const int Lq = r.ok ? L - r.q : 0, left = imin(Lq, room), rest = Lq - left;
  if (r.q > kFewPlaces) {
    Num small = {0, 0};
    for (int n = 0; n < 8; ++n) {
      const int h = sh[FS_DV + 12 * k + n].hi;
      small.lo |= h ^ (h >> 31);
    }
    sh[FS_SMALL + k] = small;
  }
  const Num kl = limbs(sh.get(FS_K));
  LULESH_UNROLL
  for (int m = 0; m < 4; ++m) {
    const i64 h = shl(product(limbs(shl(hm[m], left)), kl), rest);
    sh[FS_DV + 12 * k + 8 + m] = limbs(h);
    if (Tape::on) tape.mode(k, m, to_double(h, r.all - r.s - 186 + r.q));
  }
}

// 4: every third entry of the base vectors, gamma - sum_k derivative_k mode_k.
LULESH_FX void force_base(int k, Slots sh, ForceLane& r) {
  r.ok = r.ok && sh.get(FS_DET) + sh.get(FS_DET + 1) + sh.get(FS_DET + 2) >= shl(1, r.least);
  int up = 0;
  if (r.q > kFewPlaces) {
    const int used = sh[FS_SMALL].lo | sh[FS_SMALL + 1].lo | sh[FS_SMALL + 2].lo;
    up = imin(imax(leading_zeros((unsigned)used) - 4, 0), r.q);  // (derivatives stay below 2^60)
    r.q -= up;
  }
  const i64 one = 1ll << (58 - r.q);
  auto entry = [&](int i, auto take_sum) {
    const int n = (i >> 2) & 7, m = i & 3;
    Acc a = mul(sh[FS_DV + n], sh[FS_DV + 8 + m]);
    mac(a, sh[FS_DV + 12 + n], sh[FS_DV + 20 + m]);
    mac(a, sh[FS_DV + 24 + n], sh[FS_DV + 32 + m]);
    const Num g = limbs(((kGammaSigns >> (i & 31)) & 1u ? -one : one) - take_sum(a));
    if (i < 32) sh[FS_HG + i] = g;
  };
  if (up == 0) {
    LULESH_UNROLL
    for (int j = 0; j < 11; ++j) entry(3 * j + k, [](const Acc& a) { return take<0>(a); });
  } else {
    LULESH_ROLLED
    for (int j = 0; j < 11; ++j) entry(3 * j + k, [&](const Acc& a) { return take_up(a, up); });
  }
}

// 5: component k of the forces; out(n, value) takes corner n's. Elements with
// r.ok clear are the caller's.
template <class Out, class Tape>
LULESH_FX void force_corners(int k, Slots sh, const ForceLane& r, Out out, Tape tape) {
  const int sv = 1082 - r.ev;
  // Mode sums (the base vectors sum to zero over the corners, so differences
  // to corner 0 do), brought to 2^62 together: a smooth flow has sums far
  // below the velocities' extent.
  i64 S[4];
  unsigned used = 0, low = 0;
  LULESH_UNROLL
  for (int m = 0; m < 4; ++m) {
    Acc a = mul(sh[FS_HG + 4 + m], r.V[1]);
    LULESH_UNROLL
    for (int n = 2; n < 8; ++n) mac(a, sh[FS_HG + 4 * n + m], r.V[n]);
    S[m] = take<4>(a);
    if (Tape::on) tape.sum(k, m, to_double(S[m], 2 + r.q - sv));
    const int h = (int)(S[m] >> 32);
    used |= (unsigned)(h ^ (h >> 31));
    low |= (unsigned)(u64)S[m];
  }
  const int room = imax(leading_zeros(used) - 2, 0);
  const i64 Cm = sh.get(FS_C), Sm = sh.get(FS_S);
  const int Ck = sh[FS_EXPO].hi, Sk = sh[FS_EXPO + 1].lo;
  // both parts of the force in the larger of their units, 2^u
  const int uh = Cm != 0 && (used | low) != 0u ? 67 + 2 * r.q - room - sv + Ck : kNoExponent;
  const int us = Sm != 0 ? 125 - (r.all - r.s) + Sk : kNoExponent;
  const int u = imax(uh, us);
  const Num Cl = limbs(Cm >> imin(u - uh, 63)), Sl = limbs(Sm >> imin(u - us, 63));
  Num H[4];
  LULESH_UNROLL
  for (int m = 0; m < 4; ++m) H[m] = limbs(product(limbs(shl(S[m], room)), Cl));
#ifdef __CUDA_ARCH__
  // the base vectors are read again, not held: 64 registers
  asm volatile("" ::: "memory");
#endif
  i64 SB[4];
  LULESH_UNROLL
  for (int n = 0; n < 4; ++n) SB[n] = take<3>(mul(r.B[n], Sl));
  const i64 S0 = take<3>(mul(r.B0, Sl));
  LULESH_UNROLL
  for (int n = 0; n < 8; ++n) {
    Acc a = mul(sh[FS_HG + 4 * n], H[0]);
    mac(a, sh[FS_HG + 4 * n + 1], H[1]);
    mac(a, sh[FS_HG + 4 * n + 2], H[2]);
    mac(a, sh[FS_HG + 4 * n + 3], H[3]);
    const i64 st = n == 0 ? S0 : n < 4 ? SB[n] : -SB[n == 4 ? 2 : n == 5 ? 3 : n == 6 ? 0 : 1];
    out(n, to_double(take<5>(a) + st, u));
  }
}

}  // namespace fx
}  // namespace lulesh
