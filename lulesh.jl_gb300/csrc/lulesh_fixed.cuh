// 64-bit fixed-point arithmetic for the element kernels' geometry.
//
// GB300 issues 2 FP64 instructions per clock and SM. Measured beside that
// (independent chains, 12 warps per SM, lanes per ns and SM): DFMA 3.9,
// 32x32+64-bit integer multiply-add 114, 64-bit integer add 116, 32-bit
// integer add 237; double<->integer conversions take an FP64 slot each. So
// sums and products of quantities that share one scale run on the integer
// pipes at about six (products) to thirty times (sums) the FP64 rate. What an
// element kernel forms from its eight corners is such a set: differences of one
// coordinate's positions or velocities within one element.
//
// Numbers are integers X with an exponent for each coordinate of an element:
// x = X 2^-s. The scale puts the coordinate's extent over the corners in [2^60,
// 2^61), so a difference of corners keeps 60 bits below the extent where a double
// keeps 52 below the (larger) coordinate itself. Conversion is modulo 2^64: a corner
// far from the origin wraps, and the differences, which is all that is used,
// are exact. A product keeps the upper 64 of its 128 bits.
//
// Products are taken on balanced 32-bit limbs, x = hi 2^32 + lo with lo
// signed: hi*hi and the two cross products, three wide multiply-adds; lo*lo
// (below a quarter of the last kept bit, of either sign) is dropped. Sums of
// products share one pair of accumulators and one rounding.
//
// Error: a difference 2^-61 of the coordinate's extent, a cross product's component
// about 2^-57 of the product of the other two's, the volume about 2^-56 of the
// product of all three, each at or below what the FP64 expressions leave (tested
// beside them). What is inverted, flat, not finite or of a size no mesh has is left
// to the FP64 expressions by the callers (Range).
//
// Everything here also compiles for the host, where the tests compare it with
// exact rational arithmetic.
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define LULESH_FX __host__ __device__ __forceinline__
#else
#define LULESH_FX inline
#endif
#ifdef __CUDA_ARCH__
#define LULESH_UNROLL _Pragma("unroll")
#define LULESH_ROLLED _Pragma("unroll 1")
#else
#define LULESH_UNROLL
#define LULESH_ROLLED
#endif

namespace lulesh {
namespace fx {

typedef long long i64;
typedef unsigned long long u64;

LULESH_FX int hi_word(double x) {
#ifdef __CUDA_ARCH__
  return __double2hiint(x);
#else
  i64 b;
  memcpy(&b, &x, sizeof b);
  return (int)(b >> 32);
#endif
}
LULESH_FX unsigned lo_word(double x) {
#ifdef __CUDA_ARCH__
  return (unsigned)__double2loint(x);
#else
  i64 b;
  memcpy(&b, &x, sizeof b);
  return (unsigned)b;
#endif
}
LULESH_FX double from_words(int hi, unsigned lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double(hi, (int)lo);
#else
  const i64 b = (i64)(((u64)(unsigned)hi << 32) | lo);
  double x;
  memcpy(&x, &b, sizeof x);
  return x;
#endif
}
LULESH_FX int leading_zeros(unsigned x) {  // 32 for x = 0
#ifdef __CUDA_ARCH__
  return __clz((int)x);
#else
  return x ? __builtin_clz(x) : 32;
#endif
}
LULESH_FX int imin(int a, int b) { return a < b ? a : b; }
LULESH_FX int imax(int a, int b) { return a > b ? a : b; }

// wrapping sums
LULESH_FX i64 add(i64 a, i64 b) { return (i64)((u64)a + (u64)b); }
LULESH_FX i64 sub(i64 a, i64 b) { return (i64)((u64)a - (u64)b); }
LULESH_FX i64 shl(i64 a, int n) { return (i64)((u64)a << n); }

// --- products ---------------------------------------------------------------
struct alignas(8) Num {
  int lo, hi;  // hi 2^32 + lo, both signed
};
LULESH_FX Num limbs(i64 x) {
  Num r;
  r.lo = (int)(unsigned)(u64)x;
  r.hi = (int)((unsigned)((u64)x >> 32) + ((unsigned)r.lo >> 31));
  return r;
}
// h 2^64 + m 2^32; |m| must stay below 2^63 - 2^31
struct Acc {
  i64 h, m;
};
// c + a b; written as the instruction, which the compiler otherwise takes apart
// once it sees that a limb was cut from a 64-bit value
LULESH_FX i64 mad(int a, int b, i64 c) {
#ifdef __CUDA_ARCH__
  i64 r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
#else
  return c + (i64)a * b;
#endif
}
LULESH_FX i64 mulw(int a, int b) {
#ifdef __CUDA_ARCH__
  i64 c;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(c) : "r"(a), "r"(b));
  return c;
#else
  return (i64)a * b;
#endif
}
// 1 the compiler does not know, so that x.hi + y is one multiply-add and not
// a sign extension and two adds.
#ifdef __CUDACC__
static __constant__ int kOne = 1;
#endif
LULESH_FX int one() {
#ifdef __CUDA_ARCH__
  return kOne;
#else
  return 1;
#endif
}
LULESH_FX Acc mul(Num a, Num b) {
  Acc r;
  r.h = mulw(a.hi, b.hi);
  r.m = mad(a.lo, b.hi, mulw(a.hi, b.lo));
  return r;
}
LULESH_FX void mac(Acc& r, Num a, Num b) {
  r.h = mad(a.hi, b.hi, r.h);
  r.m = mad(a.lo, b.hi, mad(a.hi, b.lo, r.m));
}
LULESH_FX void msub(Acc& r, Num a, Num b) {
  r.h -= mulw(a.hi, b.hi);
  r.m -= mad(a.lo, b.hi, mulw(a.hi, b.lo));
}
// with lo*lo too, for sums whose terms cancel or are far below their scale
LULESH_FX void mac_full(Acc& r, Num a, Num b) {
  mac(r, a, b);
  r.m = mad((int)(mulw(a.lo, b.lo) >> 32), one(), r.m);
}
// a b - c d
LULESH_FX Acc mul_minus(Num a, Num b, Num c, Num d) {
  Acc r = mul(a, b);
  r.h -= mulw(c.hi, d.hi);
  r.m -= mad(c.lo, d.hi, mulw(c.hi, d.lo));
  return r;
}
// the same with lo*lo too
LULESH_FX Acc mul_minus_full(Num a, Num b, Num c, Num d) {
  Acc r = mul_minus(a, b, c, d);
  r.m = mad((int)(mulw(a.lo, b.lo) >> 32), one(), r.m);
  r.m -= mulw(c.lo, d.lo) >> 32;
  return r;
}
// the accumulated sum over 2^(64 - B), rounded down (a rounding addend would
// cost two moves; what it would save, half a unit, is below the dropped lo*lo)
template <int B>
LULESH_FX i64 take(Acc a) {
  return B == 0 ? mad((int)(a.m >> 32), one(), a.h) : shl(a.h, B) + (a.m >> (32 - B));
}
LULESH_FX i64 product(Num a, Num b) { return take<0>(mul(a, b)); }
// How far |x| < 2^61 can be shifted left and stay below 2^61, at most 29 (from
// the high word alone).
LULESH_FX int room(i64 x) {
  const int h = (int)(x >> 32);
  return imax(leading_zeros((unsigned)(h ^ (h >> 31))) - 3, 0);
}
LULESH_FX i64 take_up(Acc a, int B) { return shl(a.h, B) + (a.m >> (32 - B)); }
// The accumulated sum over 2^(64 - B), B as large as it stays below 2^61 with:
// a component far below the others of its vector keeps its bits.
LULESH_FX i64 take_all(Acc a, int& B) {
  B = room(take<0>(a));
  return take_up(a, B);
}
// --- conversions ------------------------------------------------------------
// Exponent field of a bound on the extent of eight doubles, from their high
// words: max - min with the low words rounded outwards. NaN and infinities
// give 0x7ff. The bound is at least 2^-21 of the largest magnitude.
// Signed and unsigned minima order sign-magnitude words well enough: with any
// negative value the unsigned maximum is the most negative one, with none the
// signed and unsigned orders agree.
LULESH_FX unsigned extent_hi(const double v[8]) {
  int smax = hi_word(v[0]);
  unsigned umax = (unsigned)smax, umin = (unsigned)smax;
LULESH_UNROLL
  for (int c = 1; c < 8; ++c) {
    const int h = hi_word(v[c]);
    const unsigned u = (unsigned)h;
    smax = imax(smax, h);
    umax = u > umax ? u : umax;
    umin = u < umin ? u : umin;
  }
  const int top = smax < 0 ? (int)umin : smax;
  const int bot = (int)umax < 0 ? (int)umax : (int)umin;
  const double ext = from_words(top, top < 0 ? 0u : 0xffffffffu) - from_words(bot, bot < 0 ? 0xffffffffu : 0u);
  return (unsigned)hi_word(ext);
}
LULESH_FX int exponent_field(unsigned hi) { return (int)((hi >> 20) & 0x7ffu); }

// Exponent field of the extent itself, to a factor of two: the bound above is that
// while it is well above 2^-20 of the largest magnitude. Below (a fast uniform
// motion, a mesh far from the origin) it is mostly the rounding of the low words, and
// differences scaled by it would leave up to 32 leading bits of every product empty
// (velocity sums 2e-8 off, forces 1e-13); the extent of the differences to the first
// corner is taken there, or 2^-52 of the magnitude, below which no difference is.
LULESH_FX bool loose(unsigned bound, double v0) {  // (NaN and infinities are not)
  return bound + (16u << 20) < ((unsigned)hi_word(v0) & 0x7fffffffu);
}
LULESH_FX int extent_field(const double v[8]) {
  const unsigned h = extent_hi(v);
  if (!loose(h, v[0])) return exponent_field(h);
  double d[8];
  LULESH_UNROLL
  for (int c = 0; c < 8; ++c) d[c] = v[c] - v[0];
  return imax(exponent_field(extent_hi(d)), exponent_field((unsigned)hi_word(v[0])) - 52);
}
// Of two coordinates' values, with one branch: a cycle at 150^3 2.161 ms with the bounds
// alone, 2.167 so, 2.187 with a branch for each.
LULESH_FX void extent_fields(const double v[8], const double w[8], int& ev, int& ew) {
  const unsigned h = extent_hi(v), g = extent_hi(w);
  ev = exponent_field(h);
  ew = exponent_field(g);
  if (loose(h, v[0]) || loose(g, w[0])) {
    ev = extent_field(v);
    ew = extent_field(w);
  }
}

// x 2^(bias + 1075) modulo 2^64, with bias = 8 - e for the exponent field e of
// the extent (extent below 2^61; 6 - e: below 2^59). Bits below the last
// place are dropped; a negative value is the complement of its magnitude's,
// one unit off for all alike. Shifts stay within 0..63: x's exponent field is at
// most 53 above e, and a zero or subnormal shifts out.
LULESH_FX i64 to_fixed(double x, int bias) {
  const int h = hi_word(x);
  const int n = (int)(((unsigned)h >> 20) & 0x7ffu) + bias;
  const u64 m = ((u64)(((unsigned)h & 0xfffffu) | 0x100000u) << 32) | lo_word(x);
  const u64 r = (m << imax(n, 0)) >> imin(imax(-n, 0), 63);
  return (i64)r ^ (i64)(h >> 31);
}

// The same rounded towards zero: zeros of both signs give zero, and x and -x
// opposite numbers, so that what cancels in doubles that fit cancels here. (A
// velocity divergence that is exactly zero sets no time constraint, and where no
// adjoint has come to an element yet, its sums stay exact zeros.)
LULESH_FX i64 to_fixed0(double x, int bias) { return sub(to_fixed(x, bias), (i64)(hi_word(x) >> 31)); }

// v 2^k, rounded once; the caller keeps the result's exponent in range
LULESH_FX double to_double(i64 v, int k) {
  const double d = (double)v;
  const int h = hi_word(d);
  return from_words(h ? h + (int)((unsigned)k << 20) : h, lo_word(d));
}

// A double as mantissa and exponent: x = m 2^k with |m| in [2^60, 2^61); zero
// and subnormals give m = 0 and an exponent below every other.
constexpr int kNoExponent = -100000;
struct Float {
  i64 m;
  int k;
};
LULESH_FX Float to_float(double x) {
  const int h = hi_word(x);
  const int e = (int)(((unsigned)h >> 20) & 0x7ffu);
  const u64 m = ((u64)(((unsigned)h & 0xfffffu) | 0x100000u) << 32) | lo_word(x);
  const i64 s = (i64)(h >> 31);
  Float r;
  r.m = e ? ((i64)(m << 8) ^ s) - s : 0;
  r.k = e ? e - 1083 : kNoExponent;
  return r;
}

// --- scale of an element ------------------------------------------------------
// Which elements the fixed-point form takes. Extents: exponent fields of the
// least and most an element's largest extent may be. det: the least Jacobian
// determinant (of the mean edges, which are the extents of an undistorted element;
// an undistorted box has 2^52 to 2^55 of its scale, by where its extents lie in
// [2^60, 2^61)) that k_force and k_kinematics take, over the box or over the cube of
// the largest extent. distortion: the powers of two the hourglass base vectors may
// outgrow their scale by.
struct Range {
  int least_extent, most_extent;
  int force_det, kin_det;
  bool over_cube;
  int distortion;
};
// Where every sum is within a few units of 2^-47 of its own size: extents for
// which the guards 1e-36 added to squared areas and to volumes are below half a
// unit, volumes above 1/32 to 1/256 of the cube.
LULESH_FX constexpr Range narrow() { return {1023 - 12, 1023 + 40, 47, 47, true, 4}; }
// Where every sum is at least as good as the FP64 expressions leave it. The kernels
// add the guards. Plates and needles along the axes are boxes; of turned ones the
// kinematics takes those above 1/32 to 1/256 of their box (the cofactors of others
// are too far below its areas), the forces down to 2^-30. What is inverted, flat or
// not finite is the FP64 form's, whose errors the step reports. A cycle at 100^3 of
// plates or needles 1:100, or of edges below 2^-12: 0.81 ms, as of cubes (in a calm
// state), turned plates 1:500 1.38; over the narrow range, both forms one after the
// other, 2.32; the FP64 kernels alone 1.81.
LULESH_FX constexpr Range wide() { return {1023 - 100, 1023 + 100, 24, 47, false, 31}; }
// velocity extents below 2^-400 are taken as that: they move nothing
constexpr int kMinSpeed = 1023 - 400, kMaxSpeed = 1023 + 400;

LULESH_FX unsigned umax(unsigned a, unsigned b) { return a > b ? a : b; }

// The scales s (x = X 2^-s) of an element's three coordinates, each its extent to
// [2^60, 2^61); an extent below 2^-28 of the largest counts as that.
struct Scales {
  int s[3];
  bool ok;  // the largest extent is in range
  LULESH_FX int wide() const { return imin(s[0], imin(s[1], s[2])); }
  // the least determinant is 2^least, in its own units (none reaches 2^58)
  LULESH_FX int least(int det, Range range) const {
    return range.over_cube ? imin(det + s[0] + s[1] + s[2] - 3 * wide(), 58) : det;
  }
};
LULESH_FX Scales scales_of(int ex0, int ex1, int ex2, Range range) {  // exponent fields of the extents
  Scales r = {{ex0, ex1, ex2}, false};
  const int top = imax(ex0, imax(ex1, ex2));
  r.ok = top >= range.least_extent && top <= range.most_extent;
  LULESH_UNROLL
  for (int j = 0; j < 3; ++j) r.s[j] = 1083 - imax(r.s[j], top - 28);
  return r;
}

// --- element geometry -----------------------------------------------------------
// The 12 face diagonals in the FP64 code's order: d20 d31 d50 d14 d61 d25 d72
// d36 d43 d07 d64 d57. Below 2^61.
LULESH_FX void diagonals(const i64 v[8], i64 g[12]) {
  constexpr int pa[12] = {2, 3, 5, 1, 6, 2, 7, 3, 4, 0, 6, 5};
  constexpr int pb[12] = {0, 1, 0, 4, 1, 5, 2, 6, 3, 7, 4, 7};
LULESH_UNROLL
  for (int q = 0; q < 12; ++q) g[q] = sub(v[pa[q]], v[pb[q]]);
}

// First-order Walsh coefficients over 4 (the mean edges; below 2^61) of corner
// values, through the four body diagonals; xez the third-order one over 4.
LULESH_FX void walsh(const i64 v[8], i64 w[3], i64* xez) {
  const i64 a = sub(v[6], v[0]), b = sub(v[5], v[3]), c = sub(v[7], v[1]), d = sub(v[4], v[2]);
  const i64 apb = a + b, cpd = c + d, amb = a - b, cmd = c - d;
  w[0] = (apb - cpd) >> 2;
  w[1] = (amb + cmd) >> 2;
  w[2] = (apb + cpd) >> 2;
  if (xez) *xez = (amb - cmd) >> 2;
}

// The even hourglass modes (eta*zeta, xi*zeta, xi*eta) over 4.
LULESH_FX void even_modes(const i64 g[12], i64 h[3]) {
  h[0] = ((g[10] - g[11]) - (g[0] + g[1])) >> 2;
  const i64 pp = g[9] + g[4], qq = g[8] + g[5];
  h[1] = (pp - qq) >> 2;
  h[2] = (pp + qq) >> 2;
}

// One element's slots in shared memory: a column of 64-bit words.
struct Slots {
  Num* p;
  int stride;
  LULESH_FX Num& operator[](int i) const { return p[i * stride]; }
  LULESH_FX void put(int i, i64 v) const {
    Num n;
    n.lo = (int)(unsigned)(u64)v;
    n.hi = (int)(v >> 32);
    p[i * stride] = n;
  }
  LULESH_FX i64 get(int i) const {
    const Num n = p[i * stride];
    return shl((i64)n.hi, 32) | (i64)(u64)(unsigned)n.lo;
  }
};
}  // namespace fx
}  // namespace lulesh
