// Host harness of the fixed-point kinematics sums and forces (lulesh_fixed_kin.cuh,
// lulesh_fixed_force.cuh) beside the FP64 expressions the kernels had and still
// have for the elements the fixed-point form does not take (kin_fp64 and force_fp64
// in lulesh_element_fp64.cuh), both against 113-bit floating point.
#include "fixed_check.cpp"

namespace {
// kin_fp64's sums: 12 volume, the largest squared face vector, areas, flows,
// rate, determinant.
void fp64_sums(const double p[3][8], const double v[3][8], double half_dt, double out[10]) {
  static const int pa[12] = {2, 3, 5, 1, 6, 2, 7, 3, 4, 0, 6, 5}, pb[12] = {0, 1, 0, 4, 1, 5, 2, 6, 3, 7, 4, 7};
  auto walsh = [](const double x[8], double w[3]) {
    const double a = x[6] - x[0], b = x[5] - x[3], c = x[7] - x[1], d = x[4] - x[2];
    const double apb = a + b, cpd = c + d;
    w[0] = apb - cpd;
    w[1] = (a - b) + (c - d);
    w[2] = apb + cpd;
  };
  double g[3][12], w[3][3], u[3][3], h[3][3], t[3][15];
  for (int k = 0; k < 3; ++k) {
    for (int q = 0; q < 12; ++q) g[k][q] = p[k][pa[q]] - p[k][pb[q]];
    walsh(p[k], w[k]);
    walsh(v[k], u[k]);
    for (int a = 0; a < 3; ++a) h[k][a] = std::fma(-half_dt, u[k][a], w[k][a]);
  }
  for (int k = 0; k < 3; ++k) {
    const int i = (k + 1) % 3, j = (k + 2) % 3;
    auto cr = [&](const double a1, const double b2, const double a2, const double b1) { return std::fma(a1, b2, -a2 * b1); };
    auto gc = [&](int a, int b) { return cr(g[i][a], g[j][b], g[j][a], g[i][b]); };
    t[k][0] = std::fma(g[k][1] + g[k][6], gc(0, 7),
                       std::fma(g[k][8] + g[k][11], gc(9, 10), (g[k][3] + g[k][5]) * gc(4, 2)));
    for (int f = 0; f < 6; ++f) t[k][1 + f] = gc(2 * f, 2 * f + 1) * gc(2 * f, 2 * f + 1);
    double C[3];
    for (int a = 0; a < 3; ++a) {
      const int b = (a + 1) % 3, c = (a + 2) % 3;
      const double A = cr(w[i][b], w[j][c], w[j][b], w[i][c]);
      C[a] = cr(h[i][b], h[j][c], h[j][b], h[i][c]);
      t[k][7 + a] = A * A;
      t[k][10 + a] = A * u[k][a];
    }
    t[k][13] = std::fma(C[0], u[k][0], std::fma(C[1], u[k][1], C[2] * u[k][2]));
    t[k][14] = h[k][1] * C[1];
  }
  auto sum = [&](int q) { return (t[0][q] + t[1][q]) + t[2][q]; };
  out[0] = sum(0);
  out[1] = 0;
  for (int f = 0; f < 6; ++f) out[1] = std::fmax(out[1], sum(1 + f));
  for (int j = 2; j < 10; ++j) out[j] = sum(5 + j);
}

// force_fp64's corner forces (mode 3: no defects).
void fp64_forces(const double p[3][8], const double v[3][8], double vi12, double coef, double s8, double f[3][8]) {
  static const int pa[12] = {2, 3, 5, 1, 6, 2, 7, 3, 4, 0, 6, 5}, pb[12] = {0, 1, 0, 4, 1, 5, 2, 6, 3, 7, 4, 7};
  double g[3][15], B[3][8], dv[3][8], hm[3][4], hg[8][4];
  for (int k = 0; k < 3; ++k) {
    const double* x = p[k];
    for (int q = 0; q < 12; ++q) g[k][q] = x[pa[q]] - x[pb[q]];
    g[k][12] = g[k][1] + g[k][6];
    g[k][13] = g[k][8] + g[k][11];
    g[k][14] = g[k][3] + g[k][5];
    const double a = x[6] - x[0], b = x[5] - x[3], c = x[7] - x[1], d = x[4] - x[2];
    const double pp = g[k][9] + g[k][4], qq = g[k][8] + g[k][5];
    const double h[4] = {(g[k][10] - g[k][11]) - (g[k][0] + g[k][1]), pp - qq, pp + qq, (a - b) - (c - d)};
    for (int m = 0; m < 4; ++m) hm[k][m] = h[m] * vi12;
  }
  for (int k = 0; k < 3; ++k) {
    const int i = (k + 1) % 3, j = (k + 2) % 3;
    auto cr = [&](int a, int b) { return std::fma(g[i][a], g[j][b], -g[j][a] * g[i][b]); };
    double n[5];
    for (int q = 0; q < 5; ++q) n[q] = cr(2 * q, 2 * q + 1);
    const double p01 = n[0] + n[1];
    B[k][0] = p01 + n[4];
    B[k][1] = p01 + n[2];
    B[k][2] = (n[0] + n[2]) + n[3];
    B[k][3] = (n[0] + n[3]) + n[4];
    static const int opposite[4] = {6, 7, 4, 5};
    for (int c = 0; c < 4; ++c) B[k][opposite[c]] = -B[k][c];
    const double u0 = cr(0, 7), v0 = cr(0, 12), w0 = cr(7, 12), u1 = cr(9, 10), v1 = cr(13, 9), w1 = cr(13, 10);
    const double u2 = cr(4, 2), v2 = cr(2, 14), w2 = cr(14, 4), t12 = u2 - u0, t37 = u0 - u1, t45 = u1 - u2;
    const double d[8] = {-((w0 + w1) + w2), t12 - v2, t12 + w0, t37 - v0, t45 - v1, t45 + w2, (v0 + v1) + v2, t37 + w1};
    for (int c = 0; c < 8; ++c) dv[k][c] = d[c];
  }
  for (int c = 0; c < 8; ++c)
    for (int m = 0; m < 4; ++m)
      hg[c][m] = std::fma(-dv[2][c], hm[2][m], std::fma(-dv[1][c], hm[1][m], std::fma(-dv[0][c], hm[0][m], gamma_negative(c, m) ? -1.0 : 1.0)));
  for (int k = 0; k < 3; ++k) {
    double h[4];
    for (int m = 0; m < 4; ++m) {
      double s = hg[0][m] * v[k][0];
      for (int c = 1; c < 8; ++c) s = std::fma(hg[c][m], v[k][c], s);
      h[m] = coef * s;
    }
    for (int c = 0; c < 8; ++c) {
      f[k][c] = s8 * B[k][c];
      for (int m = 3; m >= 0; --m) f[k][c] = std::fma(hg[c][m], h[m], f[k][c]);
    }
  }
}

// fixed_forces over either range
bool ranged_forces(const double p[3][8], const double vel[3][8], double vi12, double coef, double s8, Range range,
                   double f[3][8], double* largest_base = nullptr) {
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
  for (int k = 0; k < 3; ++k) force_diagonals(k, sh, r[k], hm[k], range);
  for (int k = 0; k < 3; ++k) force_products<3>(k, sh, r[k], hm[k], NoTape{}, range);
  for (int k = 0; k < 3; ++k) force_base(k, sh, r[k]);
  if (r[0].ok != r[1].ok || r[0].ok != r[2].ok) std::abort();
  if (largest_base)
    for (int i = *largest_base = 0; i < 32; ++i)
      *largest_base = std::fmax(*largest_base, std::fabs(sh[FS_HG + i].hi * 4294967296.0 + sh[FS_HG + i].lo));
  for (int k = 0; k < 3 && r[0].ok; ++k) force_corners(k, sh, r[k], [&](int n, double v) { f[k][n] = v; }, NoTape{});
  return r[0].ok;
}

// c = a x b, and p the sums of its products' magnitudes
void cross(const Q a[3], const Q b[3], Q c[3], Q p[3]) {
  for (int k = 0; k < 3; ++k) {
    const Q s = a[(k + 1) % 3] * b[(k + 2) % 3], t = a[(k + 2) % 3] * b[(k + 1) % 3];
    c[k] = s - t;
    p[k] = qabs(s) + qabs(t);
  }
}
}  // namespace

extern "C" {

// Sums of n elements (pos, vel: [n][3][8]) at half step half_dt: per element
// taken, and for sum j (12 volume, the largest squared face vector, the squared
// edge cross products (3), their products with the velocity differences (3), the
// cofactor sum, the half-step determinant) want[10 i + j], the errors of the fixed-point
// form and of the FP64 form, and the sum of the magnitudes of its products.
// (Sums with velocities take 4 of the coordinate's velocity extent for a
// difference, the size of its four body diagonals.) kernels: over the kernels' range.
void check_sizes(int kernels, int n, const double* pos, const double* vel, double half_dt, int* taken, double* want, double* fixed,
                 double* fp64, double* size) {
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
    for (int k = 0; k < 3; ++k) kin_edges(k, sh, half_dt, r[k], kernels ? wide() : narrow());
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
    Q w[10], s[10];
    for (int j = 0; j < 10; ++j) w[j] = s[j] = 0;
    auto d = [&](int k, int a, int b) { return (Q)p[k][a] - p[k][b]; };
    static const int tv[3][8] = {{3, 1, 7, 2, 6, 3, 2, 0}, {4, 3, 5, 7, 6, 4, 7, 0}, {1, 4, 2, 5, 6, 1, 5, 0}};
    for (int t = 0; t < 3; ++t) {
      Q U[3], V[3], W[3], c[3], m[3];
      for (int k = 0; k < 3; ++k) {
        U[k] = d(k, tv[t][0], tv[t][1]) + d(k, tv[t][2], tv[t][3]);
        V[k] = d(k, tv[t][4], tv[t][5]);
        W[k] = d(k, tv[t][6], tv[t][7]);
      }
      cross(V, W, c, m);
      for (int k = 0; k < 3; ++k) {
        w[0] += U[k] * c[k];
        s[0] += qabs(U[k]) * m[k];
      }
    }
    static const int fd[6][4] = {{2, 0, 3, 1}, {6, 4, 5, 7}, {5, 0, 1, 4}, {6, 1, 2, 5}, {7, 2, 3, 6}, {4, 3, 0, 7}};
    for (int q = 0; q < 6; ++q) {
      Q a[3], b[3], c[3], m[3], f = 0, g = 0;
      for (int k = 0; k < 3; ++k) {
        a[k] = d(k, fd[q][0], fd[q][1]);
        b[k] = d(k, fd[q][2], fd[q][3]);
      }
      cross(a, b, c, m);
      for (int k = 0; k < 3; ++k) {
        f += c[k] * c[k];
        g += qabs(c[k]) * m[k];
      }
      if (f > w[1]) {
        w[1] = f;
        s[1] = g;
      }
    }
    Q e[3][3], u[3][3], h[3][3], dV[3];  // [direction][coordinate]
    static const int sg[3][8] = {{-1, 1, 1, -1, -1, 1, 1, -1}, {-1, -1, 1, 1, -1, -1, 1, 1}, {-1, -1, -1, -1, 1, 1, 1, 1}};
    for (int k = 0; k < 3; ++k) {
      dV[k] = 0;
      for (int c = 0; c < 8; ++c)
        for (int b = 0; b < 8; ++b)
          if ((Q)v[k][c] - v[k][b] > dV[k]) dV[k] = (Q)v[k][c] - v[k][b];
      for (int a = 0; a < 3; ++a) {
        e[a][k] = u[a][k] = 0;
        for (int c = 0; c < 8; ++c) {
          e[a][k] += sg[a][c] * (Q)p[k][c];
          u[a][k] += sg[a][c] * (Q)v[k][c];
        }
        h[a][k] = e[a][k] - (Q)half_dt * u[a][k];
      }
    }
    for (int a = 0; a < 3; ++a) {
      Q A[3], Am[3], C[3], Cm[3];
      cross(e[(a + 1) % 3], e[(a + 2) % 3], A, Am);
      cross(h[(a + 1) % 3], h[(a + 2) % 3], C, Cm);
      for (int k = 0; k < 3; ++k) {
        w[2 + a] += A[k] * A[k];
        s[2 + a] += qabs(A[k]) * Am[k];
        w[5 + a] += A[k] * u[a][k];
        s[5 + a] += Am[k] * 4 * dV[k];
        w[8] += C[k] * u[a][k];
        s[8] += Cm[k] * 4 * dV[k];
        if (a == 1) {
          w[9] += C[k] * h[1][k];
          s[9] += Cm[k] * qabs(h[1][k]);
        }
      }
    }
    double plain[10];
    fp64_sums(p, v, half_dt, plain);
    for (int j = 0; j < 10; ++j) {
      want[10 * i + j] = (double)w[j];
      fixed[10 * i + j] = (double)qabs((Q)got[j] - w[j]);
      fp64[10 * i + j] = (double)qabs((Q)plain[j] - w[j]);
      size[10 * i + j] = (double)s[j];
    }
  }
}

// Corner forces (mode 3) of n elements (scal: [n][3] = vi12, coef, s8): per element
// taken, and for coordinate k the largest errors over the corners of the two forms,
// and the size: |s8| times the magnitudes of the products of a corner's three
// faces, plus |coef| times the coordinate's velocity extent.
void check_force_sizes(int kernels, int n, const double* pos, const double* vel, const double* scal, int* taken, double* fixed,
                       double* fp64, double* size) {
  static const int fd[6][4] = {{2, 0, 3, 1}, {5, 0, 1, 4}, {6, 1, 2, 5}, {7, 2, 3, 6}, {4, 3, 0, 7}, {6, 4, 5, 7}};
  for (int i = 0; i < n; ++i) {
    const double(*p)[8] = reinterpret_cast<const double(*)[8]>(pos + 24 * i);
    const double(*v)[8] = reinterpret_cast<const double(*)[8]>(vel + 24 * i);
    const double vi12 = scal[3 * i], coef = scal[3 * i + 1], s8 = scal[3 * i + 2];
    double f[3][8], plain[3][8];
    taken[i] = ranged_forces(p, v, vi12, coef, s8, kernels ? wide() : narrow(), f);
    if (!taken[i]) continue;
    Q qf[3][8], qdv[3][8], qh[3][4], qS[3][4];
    exact_forces(p, v, vi12, coef, s8, 3, qf, qdv, qh, qS);
    fp64_forces(p, v, vi12, coef, s8, plain);
    Q most[3] = {0, 0, 0};
    for (int q = 0; q < 6; ++q) {
      Q a[3], b[3], c[3], m[3];
      for (int k = 0; k < 3; ++k) {
        a[k] = (Q)p[k][fd[q][0]] - p[k][fd[q][1]];
        b[k] = (Q)p[k][fd[q][2]] - p[k][fd[q][3]];
      }
      cross(a, b, c, m);
      for (int k = 0; k < 3; ++k)
        if (m[k] > most[k]) most[k] = m[k];
    }
    for (int k = 0; k < 3; ++k) {
      double dV = 0;
      Q e = 0, g = 0;
      for (int c = 0; c < 8; ++c) {
        for (int b = 0; b < 8; ++b) dV = std::fmax(dV, v[k][c] - v[k][b]);
        if (qabs(f[k][c] - qf[k][c]) > e) e = qabs(f[k][c] - qf[k][c]);
        if (qabs(plain[k][c] - qf[k][c]) > g) g = qabs(plain[k][c] - qf[k][c]);
      }
      fixed[3 * i + k] = (double)e;
      fp64[3 * i + k] = (double)g;
      size[3 * i + k] = (double)(3 * std::fabs(s8) * most[k]) + std::fabs(coef) * dV;
    }
  }
}

// The largest entry of the hourglass base vectors, in their units, over the kernels'
// range (0 for an element that is not taken).
void check_base(int n, const double* pos, const double* vel, const double* scal, double* largest) {
  for (int i = 0; i < n; ++i) {
    double f[3][8];
    if (!ranged_forces(reinterpret_cast<const double(*)[8]>(pos + 24 * i), reinterpret_cast<const double(*)[8]>(vel + 24 * i),
                       scal[3 * i], scal[3 * i + 1], scal[3 * i + 2], wide(), f, largest + i))
      largest[i] = 0;
  }
}

}  // extern "C"
