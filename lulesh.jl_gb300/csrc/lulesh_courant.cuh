// Which Courant candidates need not be formed (k_material). Also compiled for the
// host, where a test compares it with the candidates over the whole range of doubles.
#pragma once

#include <math.h>

#include "lulesh_fixed.cuh"

namespace lulesh {

// A non-negative double as a float, rounded down; 0 below the float range and
// infinity above it. On the integer pipe (a conversion takes an FP64 slot).
LULESH_FX float coarse(double x) {
  const int h = fx::hi_word(x);
  if (h < 0x38100000) return 0.f;
  const int b = h >= 0x47f00000 ? 0x7f800000 : ((h - 0x38000000) << 3) | (int)(fx::lo_word(x) >> 29);
#ifdef __CUDA_ARCH__
  return __int_as_float(b);
#else
  float f;
  memcpy(&f, &b, sizeof f);
  return f;
#endif
}

// 8 |qqc| for courant_above: infinity (never certain) where it is far from any
// viscosity coefficient, rounded up where it is almost none.
inline float coarse_qqc8(double qqc) {
  const double q = 8.0 * fabs(qqc);
  return q == 0.0 ? 0.f : q < 1e-30 ? 1e-30f : q <= 1e15 ? (float)q : INFINITY;
}

// Whether the candidate arealg / sqrt(ss^2 + [vdov < 0] (8 qqc arealg vdov)^2)
// (src/domain.jl:2996-3005) is certainly above `least` > 0: the estimate, in FP32
// from rounded-down operands, is good to 1e-6, the margin 1e-4. Operands that a
// float does not hold leave it uncertain: a candidate's terms reach over the
// squares of the float range in units no one uses, but what is in use is not for
// this to say. (arealg vdov first: where that underflows, the term does not count
// beside 1e-30.)
LULESH_FX bool courant_above(double arealg, double ss, double vdov, double least, float qqc8) {
  const float fa = coarse(arealg), fs = coarse(ss), fl = coarse(least);
  float f = fs * fs;
  if (fx::hi_word(vdov) < 0) {
    const float fv = coarse(fx::from_words(fx::hi_word(vdov) & 0x7fffffff, fx::lo_word(vdov)));
    if (!(fv > 0.f)) return false;
    const float t = qqc8 * (fa * fv);
    f = fmaf(t, t, f);
  }
  return f > 1e-30f && fl > 0.f && fa > fl * (sqrtf(f) * 1.0001f);
}

}  // namespace lulesh
