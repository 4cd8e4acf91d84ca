// Host harness of the fixed-point element arithmetic
// (lulesh.jl_gb300/csrc/lulesh_fixed*.cuh): the same functions the kernels
// run, compared with 113-bit floating point, where every product and sum of
// these expressions is exact or rounded far below the bounds tested.
#include "../lulesh.jl_gb300/csrc/lulesh_fixed_force.cuh"
#include "../lulesh.jl_gb300/csrc/lulesh_fixed_kin.cuh"

#include <cmath>
#include <cstdlib>

#if defined(__x86_64__)
typedef __float128 Q;
#else
typedef long double Q;  // binary128 on aarch64
#endif

namespace {
using namespace lulesh::fx;

bool gamma_negative(int n, int m) { return (kGammaSigns >> (4 * n + m)) & 1u; }

Q qabs(Q a) { return a < 0 ? -a : a; }

struct NoTape {
  static constexpr bool on = false;
  void derivative(int, int, double) {}
  void mode(int, int, double) {}
  void sum(int, int, double) {}
};
struct KeepTape {
  static constexpr bool on = true;
  double *dv, *hms, *s;
  void derivative(int k, int n, double v) { dv[8 * k + n] = v; }
  void mode(int k, int m, double v) { hms[4 * k + m] = v; }
  void sum(int k, int m, double v) { s[4 * k + m] = v; }
};

void qcross(const Q a[3], const Q b[3], Q c[3]) {
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}

// The reference's corner forces: normals from the six faces, volume
// derivatives from edge sums (src/domain.jl:1178-1256), base vectors and
// contractions as written there. dv, hms, s: what a tape holds.
void exact_forces(const double p[3][8], const double vel[3][8], double vi12, double coef, double s8, int mode,
                  Q f[3][8], Q dv[3][8], Q hms[3][4], Q S[3][4]) {
  static const int fd[6][4] = {{2, 0, 3, 1}, {5, 0, 1, 4}, {6, 1, 2, 5}, {7, 2, 3, 6}, {4, 3, 0, 7}, {6, 4, 5, 7}};
  static const int nf[8][3] = {{0, 1, 4}, {0, 1, 2}, {0, 2, 3}, {0, 3, 4}, {1, 4, 5}, {1, 2, 5}, {2, 3, 5}, {3, 4, 5}};
  Q n[6][3];
  for (int q = 0; q < 6; ++q) {
    Q a[3], b[3];
    for (int k = 0; k < 3; ++k) {
      a[k] = (Q)p[k][fd[q][0]] - p[k][fd[q][1]];
      b[k] = (Q)p[k][fd[q][2]] - p[k][fd[q][3]];
    }
    qcross(a, b, n[q]);
  }
  Q B[3][8];
  for (int c = 0; c < 8; ++c)
    for (int k = 0; k < 3; ++k) B[k][c] = n[nf[c][0]][k] + n[nf[c][1]][k] + n[nf[c][2]][k];
  if (!(mode & 1)) {
    B[1][0] += n[4][1];
    B[2][0] -= n[4][2];
  }
  static const int call[8][6] = {{1, 2, 3, 4, 5, 7}, {0, 1, 2, 7, 4, 6}, {3, 0, 1, 6, 7, 5}, {2, 3, 0, 5, 6, 4},
                                 {7, 6, 5, 0, 3, 1}, {4, 7, 6, 1, 0, 2}, {5, 4, 7, 2, 1, 3}, {6, 5, 4, 3, 2, 0}};
  static const int owner[8] = {0, 3, 2, 1, 4, 5, 6, 7};
  for (int c = 0; c < 8; ++c) {
    const int* o = call[c];
    auto v = [&](int k, int i) { return (Q)p[k][o[i]]; };
    auto term = [&](int a, int b) {  // the y-z form of voluDer, coordinates a, b
      return (v(a, 1) + v(a, 2)) * (v(b, 0) + v(b, 1)) - (v(a, 0) + v(a, 1)) * (v(b, 1) + v(b, 2)) +
             (v(a, 0) + v(a, 4)) * (v(b, 3) + v(b, 4)) - (v(a, 3) + v(a, 4)) * (v(b, 0) + v(b, 4)) -
             (v(a, 2) + v(a, 5)) * (v(b, 3) + v(b, 5)) + (v(a, 3) + v(a, 5)) * (v(b, 2) + v(b, 5));
    };
    const int slot = (mode & 2) ? owner[c] : c;
    dv[0][slot] = term(1, 2);
    dv[1][slot] = -term(0, 2);
    dv[2][slot] = term(0, 1);
  }
  Q hg[8][4];
  for (int m = 0; m < 4; ++m) {
    for (int k = 0; k < 3; ++k) {
      Q h = 0;
      for (int c = 0; c < 8; ++c) h += gamma_negative(c, m) ? -(Q)p[k][c] : (Q)p[k][c];
      hms[k][m] = h * vi12;
    }
    for (int c = 0; c < 8; ++c)
      hg[c][m] = (gamma_negative(c, m) ? -1 : 1) - (dv[0][c] * hms[0][m] + dv[1][c] * hms[1][m] + dv[2][c] * hms[2][m]);
  }
  for (int k = 0; k < 3; ++k) {
    Q h[4];
    for (int m = 0; m < 4; ++m) {
      h[m] = 0;
      for (int c = 0; c < 8; ++c) h[m] += hg[c][m] * vel[k][c];
      S[k][m] = h[m];
    }
    for (int c = 0; c < 8; ++c) {
      f[k][c] = (Q)s8 * B[k][c];
      for (int m = 0; m < 4; ++m) f[k][c] += hg[c][m] * h[m] * (Q)coef;
    }
  }
}

// The kernel's phases for one element, its three threads in turn.
template <int MODE, class Tape>
bool fixed_forces(const double p[3][8], const double vel[3][8], double vi12, double coef, double s8, double f[3][8],
                  Tape tape) {
  Num column[FS_COUNT];
  const Slots sh{column, 1};
  ForceLane r[3];
  i64 hm[3][4];
  for (int k = 0; k < 3; ++k) {
    for (int c = 0; c < 8; ++c) r[k].x[c] = p[k][c];
    force_load(k, sh, vel[k], r[k]);
  }
  force_scales(sh, vi12, coef);
  force_stress(sh, s8);
  for (int k = 0; k < 3; ++k) force_diagonals(k, sh, r[k], hm[k]);
  for (int k = 0; k < 3; ++k) force_products<MODE>(k, sh, r[k], hm[k], tape);
  for (int k = 0; k < 3; ++k) force_base(k, sh, r[k]);
  if (r[0].ok != r[1].ok || r[0].ok != r[2].ok) std::abort();
  for (int k = 0; k < 3 && r[0].ok; ++k) force_corners(k, sh, r[k], [&](int n, double v) { f[k][n] = v; }, tape);
  return r[0].ok;
}
}  // namespace

extern "C" {

// Corner forces of n elements (pos, vel: [n][3][8]; scal: [n][3] = vi12, coef,
// s8). taken[i] tells whether the fixed-point form took the element; force:
// [n][3][8]. Per element, err[4 i + 0..3]: the largest error of the forces
// over the scale |s8| E^2 + |coef| dV (E, dV the largest corner extents), of
// the volume derivatives over E^2, of the scaled modes over their bound E vi12
// and of the mode sums over dV.
void check_forces(int mode, int n, const double* pos, const double* vel, const double* scal, int* taken, double* force,
                  double* err) {
  for (int i = 0; i < n; ++i) {
    const double(*p)[8] = reinterpret_cast<const double(*)[8]>(pos + 24 * i);
    const double(*v)[8] = reinterpret_cast<const double(*)[8]>(vel + 24 * i);
    double(*f)[8] = reinterpret_cast<double(*)[8]>(force + 24 * i);
    const double vi12 = scal[3 * i], coef = scal[3 * i + 1], s8 = scal[3 * i + 2];
    auto run = [&](auto t) {
      switch (mode & 3) {
        case 0: return fixed_forces<0>(p, v, vi12, coef, s8, f, t);
        case 1: return fixed_forces<1>(p, v, vi12, coef, s8, f, t);
        case 2: return fixed_forces<2>(p, v, vi12, coef, s8, f, t);
        default: return fixed_forces<3>(p, v, vi12, coef, s8, f, t);
      }
    };
    double dv[24], hms[12], S[12];
    run(KeepTape{dv, hms, S});
    taken[i] = run(NoTape{});
    if (!taken[i]) continue;
    Q qf[3][8], qdv[3][8], qh[3][4], qS[3][4];
    exact_forces(p, v, vi12, coef, s8, mode, qf, qdv, qh, qS);
    auto extent = [](const double a[3][8]) {
      double e = 0;
      for (int k = 0; k < 3; ++k)
        for (int c = 0; c < 8; ++c)
          for (int b = 0; b < 8; ++b) e = std::fmax(e, a[k][c] - a[k][b]);
      return e;
    };
    const double E = extent(p), dV = extent(v);
    Q e[4] = {0, 0, 0, 0};
    auto up = [](Q& a, Q b) { if (b > a) a = b; };
    for (int k = 0; k < 3; ++k) {
      for (int c = 0; c < 8; ++c) {
        up(e[0], qabs(f[k][c] - qf[k][c]));
        up(e[1], qabs(dv[8 * k + c] - qdv[k][c]));
      }
      for (int m = 0; m < 4; ++m) {
        up(e[2], qabs(hms[4 * k + m] - qh[k][m]));
        up(e[3], qabs(S[4 * k + m] - qS[k][m]));
      }
    }
    const double scale[4] = {std::fabs(s8) * E * E + std::fabs(coef) * dV, E * E, E * vi12, dV};
    for (int j = 0; j < 4; ++j) err[4 * i + j] = e[j] == 0 ? 0.0 : (double)(e[j] / (Q)scale[j]);
  }
}

// Kinematics sums of n elements (pos, vel: [n][3][8]) at half step half_dt.
// Per element, taken, and err[13 i + j]: errors over the sums' scales (E, dV
// the largest corner extents): 12 volume over E^3, the largest squared face
// vector over E^4, the squared edge cross products over 256 E^4 (3), their
// products with the velocity differences over 64 E^2 dV (3), the cofactor sum
// over 64 E^2 dV, the half-step determinant over 64 E^3; and of 12 volume and
// the determinant over their own size; then the largest face's place.
void check_kinematics(int n, const double* pos, const double* vel, double half_dt, int* taken, double* err) {
  for (int i = 0; i < n; ++i) {
    const double(*p)[8] = reinterpret_cast<const double(*)[8]>(pos + 24 * i);
    const double(*v)[8] = reinterpret_cast<const double(*)[8]>(vel + 24 * i);
    Num column[KS_COUNT];
    const Slots sh{column, 1};
    KinLane r[3];
    for (int k = 0; k < 3; ++k) {
      for (int c = 0; c < 8; ++c) {
        r[k].x[c] = p[k][c];
        r[k].v[c] = v[k][c];
      }
      kin_extents(k, sh, r[k]);
    }
    for (int k = 0; k < 3; ++k) kin_edges(k, sh, half_dt, r[k]);
    for (int k = 0; k < 3; ++k) kin_products(k, sh, r[k]);
    for (int k = 0; k < 3; ++k) kin_terms(k, sh, r[k]);
    for (int k = 0; k < 3; ++k) kin_accept(sh, r[k]);
    if (r[0].ok != r[1].ok || r[0].ok != r[2].ok) std::abort();
    taken[i] = r[0].ok;
    if (!taken[i]) continue;
    int place;
    const double got[10] = {kin_volume12(sh, r[0]), kin_largest_face(sh, r[0], place),
                            kin_area(sh, r[0], 0), kin_area(sh, r[0], 1), kin_area(sh, r[0], 2),
                            kin_flow(sh, r[0], 0), kin_flow(sh, r[0], 1), kin_flow(sh, r[0], 2),
                            kin_rate(sh, r[0]), kin_jacobian(sh, r[0])};
    Q want[10];
    auto d = [&](int k, int a, int b) { return (Q)p[k][a] - p[k][b]; };
    static const int tv[3][8] = {{3, 1, 7, 2, 6, 3, 2, 0}, {4, 3, 5, 7, 6, 4, 7, 0}, {1, 4, 2, 5, 6, 1, 5, 0}};
    want[0] = 0;
    for (int t = 0; t < 3; ++t) {
      Q U[3], V[3], W[3], c[3];
      for (int k = 0; k < 3; ++k) {
        U[k] = d(k, tv[t][0], tv[t][1]) + d(k, tv[t][2], tv[t][3]);
        V[k] = d(k, tv[t][4], tv[t][5]);
        W[k] = d(k, tv[t][6], tv[t][7]);
      }
      qcross(V, W, c);
      want[0] += U[0] * c[0] + U[1] * c[1] + U[2] * c[2];
    }
    static const int fd[6][4] = {{2, 0, 3, 1}, {6, 4, 5, 7}, {5, 0, 1, 4}, {6, 1, 2, 5}, {7, 2, 3, 6}, {4, 3, 0, 7}};
    want[1] = 0;
    Q face[6];
    for (int q = 0; q < 6; ++q) {
      Q a[3], b[3], c[3];
      for (int k = 0; k < 3; ++k) {
        a[k] = d(k, fd[q][0], fd[q][1]);
        b[k] = d(k, fd[q][2], fd[q][3]);
      }
      qcross(a, b, c);
      face[q] = c[0] * c[0] + c[1] * c[1] + c[2] * c[2];
      if (face[q] > want[1]) want[1] = face[q];
    }
    Q w[3][3], u[3][3], h[3][3];  // [direction][coordinate]
    static const int sg[3][8] = {{-1, 1, 1, -1, -1, 1, 1, -1}, {-1, -1, 1, 1, -1, -1, 1, 1}, {-1, -1, -1, -1, 1, 1, 1, 1}};
    for (int a = 0; a < 3; ++a)
      for (int k = 0; k < 3; ++k) {
        w[a][k] = u[a][k] = 0;
        for (int c = 0; c < 8; ++c) {
          w[a][k] += sg[a][c] * (Q)p[k][c];
          u[a][k] += sg[a][c] * (Q)v[k][c];
        }
        h[a][k] = w[a][k] - (Q)half_dt * u[a][k];
      }
    want[8] = 0;
    for (int a = 0; a < 3; ++a) {
      Q A[3], C[3];
      qcross(w[(a + 1) % 3], w[(a + 2) % 3], A);
      qcross(h[(a + 1) % 3], h[(a + 2) % 3], C);
      want[2 + a] = A[0] * A[0] + A[1] * A[1] + A[2] * A[2];
      want[5 + a] = A[0] * u[a][0] + A[1] * u[a][1] + A[2] * u[a][2];
      want[8] += C[0] * u[a][0] + C[1] * u[a][1] + C[2] * u[a][2];
      if (a == 1) want[9] = C[0] * h[1][0] + C[1] * h[1][1] + C[2] * h[1][2];
    }
    double E = 0, dV = 0;
    for (int k = 0; k < 3; ++k)
      for (int c = 0; c < 8; ++c)
        for (int b = 0; b < 8; ++b) {
          E = std::fmax(E, p[k][c] - p[k][b]);
          dV = std::fmax(dV, v[k][c] - v[k][b]);
        }
    const Q E2 = (Q)E * E, flow = 64 * E2 * dV;
    const Q scale[10] = {E2 * E, E2 * E2, 256 * E2 * E2, 256 * E2 * E2, 256 * E2 * E2, flow, flow, flow, flow, 64 * E2 * E};
    for (int j = 0; j < 10; ++j) {
      const Q e = qabs((Q)got[j] - want[j]);
      err[13 * i + j] = e == 0 ? 0.0 : (double)(e / scale[j]);
    }
    err[13 * i + 10] = (double)(qabs((Q)got[0] - want[0]) / qabs(want[0]));
    err[13 * i + 11] = (double)(qabs((Q)got[9] - want[9]) / qabs(want[9]));
    // how far the chosen face is from the largest
    err[13 * i + 12] = (double)((want[1] - face[place]) / want[1]);
  }
}

// to_fixed and to_float of n doubles
void convert(int n, const double* x, const int* bias, long long* fixed, long long* mant, int* expo) {
  for (int i = 0; i < n; ++i) {
    fixed[i] = to_fixed(x[i], bias[i]);
    const Float f = to_float(x[i]);
    mant[i] = f.m;
    expo[i] = f.k;
  }
}

// extent bound's exponent field of n groups of eight values
void extents(int n, const double* v, int* field) {
  for (int i = 0; i < n; ++i) field[i] = exponent_field(extent_hi(v + 8 * i));
}

}  // extern "C"
