// Which matrices fx_encode (fixed.cuh) keeps in fp64, on the host. One line per
// kind: name, matrices, graded ones, slots that do not give their matrix back.
#include <cmath>
#include <complex>
#include <cstdio>
#include <random>

#include "fixed.cuh"

using namespace gf;
typedef std::complex<double> cd;

static void unitarise(cd r[3][3]) {
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
}

int main() {
  std::mt19937_64 g(5);
  std::normal_distribution<double> nd;
  const char* names[] = {"haar", "gaussian", "identity", "weak", "diagonal", "su2", "exact_su2", "real", "thin_row"};
  for (int kind = 0; kind < 9; ++kind) {
    const int N = kind < 2 ? 2000000 : 2000;
    int graded = 0, wrong = 0;
    for (int t = 0; t < N; ++t) {
      cd r[3][3];
      const double eps = kind == 0 || kind == 1 ? 1.0 : std::pow(10.0, -7 - t % 6), big = std::pow(2.0, t % 41 - 20);
      for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
          cd x(nd(g), nd(g));
          const bool block = i < 2 && j < 2;
          if (kind == 2) x = i == j;
          if (kind == 3) x = (i == j ? 1.0 : 0.0) + eps * x;
          if (kind == 4) x = i == j ? x : eps * x;
          if (kind == 5) x = block || i == j ? x : eps * x;
          if (kind == 6) x = block ? x : cd(i == j);
          if (kind == 7) x = cd(x.real(), eps * x.imag());
          if (kind == 8 && i == t % 3) x *= eps;
          r[i][j] = x;
        }
      if (kind != 1 && kind != 8) unitarise(r);
      double m[18];
      for (int i = 0; i < 9; ++i) {
        m[2 * i] = big * r[i / 3][i % 3].real();
        m[2 * i + 1] = big * r[i / 3][i % 3].imag();
      }
      int4 f[9];
      const int e = fx_encode(m, f);
      graded += e == GF_FX_F64;
      bool bad = fx_has_f64(e) != (e == GF_FX_F64) || fx_has_f64(6 * GF_FX_BAD + 7000) || !fx_has_f64(GF_FX_F64 - 7000);
      for (int i = 0; i < 18; ++i) {
        const int4 v = f[i / 2];
        const int h = i % 2 ? v.z : v.x, l = i % 2 ? v.w : v.y;
        if (e == GF_FX_F64) bad = bad || fx_unpack64(h, l) != m[i];
        // in fixed point: to half a unit, 2^(e - 61), and a rounding to fp64
        else bad = bad || std::fabs(fx_to_f64(fx_join(h, l), e) - m[i]) > std::ldexp(1.0, e - 61) + 1.2e-16 * std::fabs(m[i]);
      }
      wrong += bad;
    }
    std::printf("%s %d %d %d\n", names[kind], N, graded, wrong);
  }
  // results around the smallest normal number: within half a unit of 2^-1074, or of fp64's rounding
  int wrong = 0;
  for (int t = 0; t < 200000; ++t) {
    const i64 R = (i64)(g() >> (4 + t % 60)) * (t & 1 ? 1 : -1);
    const int E = -1020 - (int)(g() % 70);
    const long double x = ldexpl((long double)R, E - 60), y = fx_to_f64(R, E);
    const long double unit = fmaxl(ldexpl(1.0L, -1074), fabsl(x) * ldexpl(1.0L, -52));
    wrong += !(fabsl(x - y) <= 0.5L * unit);
  }
  std::printf("subnormal 200000 0 %d\n", wrong);
  return 0;
}
