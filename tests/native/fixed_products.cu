// Host-side accuracy check of the block fixed-point rows of fixed.cuh (device
// and host forms are the same source): chains row(A) B^dag C against long
// double, beside the same chain in fp64, and the fp64 <-> fixed conversions.
// Prints one line per kind: name, fixed rms and max, fp64 rms and max, errors
// relative to the product of the Frobenius norms.
#include <cmath>
#include <complex>
#include <cstdio>
#include <random>

#include "fixed.cuh"

using namespace gf;
typedef std::complex<long double> cl;
typedef std::complex<double> cd;

struct Arr {
  const int4* p;
  int4 operator()(int e) const { return p[e]; }
};

static void unitarise(double* m) {
  cd r[3][3];
  for (int i = 0; i < 9; ++i) r[i / 3][i % 3] = cd(m[2 * i], m[2 * i + 1]);
  for (int i = 0; i < 3; ++i) {
    for (int j = 0; j < i; ++j) {
      cd d = 0;
      for (int k = 0; k < 3; ++k) d += std::conj(r[j][k]) * r[i][k];
      for (int k = 0; k < 3; ++k) r[i][k] -= d * r[j][k];
    }
    double n = 0;
    for (int k = 0; k < 3; ++k) n += std::norm(r[i][k]);
    for (int k = 0; k < 3; ++k) r[i][k] /= std::sqrt(n);
  }
  for (int i = 0; i < 9; ++i) {
    m[2 * i] = r[i / 3][i % 3].real();
    m[2 * i + 1] = r[i / 3][i % 3].imag();
  }
}

// kind 0: unitary, 1: Gaussian at scales 1e-20 .. 1e20, 2: graded entries
static void chain(int kind, std::mt19937_64& g) {
  std::normal_distribution<double> nd;
  double fs = 0, fm = 0, ds = 0, dm = 0, conv = 0;
  long n = 0, shifted = 0;
  for (int t = 0; t < 20000; ++t) {
    double m[3][18];
    int4 f[3][9];
    int E[3];
    double norm = 1;
    for (int q = 0; q < 3; ++q) {
      const double s = kind == 0 ? 1.0 : std::pow(10.0, (t + 7 * q) % 41 - 20);
      double fn = 0, big = 0;
      for (int i = 0; i < 18; ++i) m[q][i] = nd(g) * s * (kind == 2 ? std::pow(10.0, -3 * ((i + t) % 5)) : 1.0);
      if (kind == 0) unitarise(m[q]);
      for (int i = 0; i < 18; ++i) {
        fn += m[q][i] * m[q][i];
        big = std::fmax(big, std::fabs(m[q][i]));
      }
      norm *= std::sqrt(fn);
      E[q] = fx_from_f64(m[q], f[q]);
      shifted += kind == 0 && E[q] != 0;
      for (int i = 0; i < 18; ++i) {
        const int4 v = f[q][i / 2];
        const i64 R = i % 2 ? fx_join(v.z, v.w) : fx_join(v.x, v.y);
        conv = std::fmax(conv, std::fabs(fx_to_f64(R, E[q]) - m[q][i]) / big);
      }
    }
    cl M[3][9];
    cd D[3][9];
    for (int q = 0; q < 3; ++q)
      for (int i = 0; i < 9; ++i) {
        M[q][i] = cl(m[q][2 * i], m[q][2 * i + 1]);
        D[q][i] = cd(m[q][2 * i], m[q][2 * i + 1]);
      }
    for (int r = 0; r < 3; ++r) {
      fx_row a;
      for (int k = 0; k < 3; ++k) {
        const int4 v = f[0][3 * r + k];
        a.ah[k] = v.x;
        a.al[k] = v.y;
        a.bh[k] = v.z;
        a.bl[k] = v.w;
      }
      const fx_acc p = fx_row_mul<false>(fx_operand<0>(fx_row_mul<true>(a, Arr{f[1]})), Arr{f[2]});
      cl x[3], y[3];
      cd u[3], w[3];
      for (int j = 0; j < 3; ++j)
        for (int k = 0; k < 3; ++k) {
          x[j] += M[0][3 * r + k] * std::conj(M[1][3 * j + k]);
          u[j] += D[0][3 * r + k] * std::conj(D[1][3 * j + k]);
        }
      for (int j = 0; j < 3; ++j) {
        for (int k = 0; k < 3; ++k) {
          y[j] += x[k] * M[2][3 * k + j];
          w[j] += u[k] * D[2][3 * k + j];
        }
        const int e = E[0] + E[1] + E[2] - 60;
        const cl z(ldexpl((long double)p.re[j], e), ldexpl((long double)p.im[j], e));
        const double ef = (double)std::abs(z - y[j]) / norm, ed = (double)std::abs(cl(w[j]) - y[j]) / norm;
        fs += ef * ef;
        ds += ed * ed;
        fm = std::fmax(fm, ef);
        dm = std::fmax(dm, ed);
        ++n;
      }
    }
  }
  static const char* name[3] = {"unitary", "gaussian", "graded"};
  std::printf("%s %.4e %.4e %.4e %.4e %.4e %ld\n", name[kind], std::sqrt(fs / n), fm, std::sqrt(ds / n), dm, conv,
              shifted);
}

int main() {
  std::mt19937_64 g(5);
  for (int k = 0; k < 3; ++k) chain(k, g);
  // special values: the largest and smallest doubles, subnormals, zero, non-finite entries
  double m[18] = {0};
  int4 f[9];
  int E = fx_from_f64(m, f), bad = f[0].x || f[8].w || fx_to_f64(0, E) != 0.0;
  m[0] = 1.7976931348623157e308;
  m[3] = -1.0;
  E = fx_from_f64(m, f);
  bad += fx_to_f64(fx_join(f[0].x, f[0].y), E) != m[0];
  m[0] = 4.9406564584124654e-324;
  m[3] = -2.2250738585072014e-308;
  E = fx_from_f64(m, f);
  bad += fx_to_f64(fx_join(f[1].z, f[1].w), E) != m[3];
  m[7] = NAN;
  bad += fx_from_f64(m, f) != GF_FX_BAD;
  m[7] = -INFINITY;
  bad += fx_from_f64(m, f) != GF_FX_BAD;
  bad += fx_to_f64(1, GF_FX_BAD) == fx_to_f64(1, GF_FX_BAD);
  bad += fx_to_f64(1ll << 60, 1024) != INFINITY || fx_to_f64(-(1ll << 60), 1024) != -INFINITY;
  std::printf("special %d\n", bad);
  return 0;
}
