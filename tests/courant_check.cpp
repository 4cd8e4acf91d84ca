// Host harness of the coarse comparison of Courant candidates.
#include "../lulesh.jl_gb300/csrc/lulesh_courant.cuh"

#if defined(__x86_64__)
typedef __float128 Q;
#else
typedef long double Q;  // binary128 on aarch64
#endif

// says[i]: certainly above; above[i]: the candidate is at least `least`, in 113 bits
// with a 15-bit exponent (compared without quotient and root)
extern "C" void check_courant(int n, const double* arealg, const double* ss, const double* vdov, const double* least,
                              const double* qqc, int* says, int* above) {
  for (int i = 0; i < n; ++i) {
    says[i] = lulesh::courant_above(arealg[i], ss[i], vdov[i], least[i], lulesh::coarse_qqc8(qqc[i]));
    const Q a = arealg[i], s = ss[i], t = vdov[i] < 0 ? 8 * (Q)qqc[i] * a * (Q)vdov[i] : 0, l = least[i];
    above[i] = a * a >= l * l * (s * s + t * t);
  }
}
