// The fp64 twins of the fixed-point kernels' arithmetic, by rows too, for links
// whose products hold a graded matrix (fixed.cuh): the small parts of weak or
// nearly diagonal fields keep the digits of their own that fp64 gives them.
// All of it is out of line and run by blocks that meet such a link only; a
// thread 3 link + row forms its row for those links and sits out for the rest.
// The rows stay within the registers that the calling kernels have. Fields that
// are graded throughout are bound by the fp64 pipe: weak links at 24^4, force
// 3.57 ms, plaquette + rectangle force 18.7, plaquette 0.92, two-level stout
// force 43.1, link update 1.08, where kernels in fp64 altogether took 4.78, 30.4,
// 1.22, 46.3 and 0.95, and fixed point alone, with 10^-9 of the small parts
// wrong, 0.74, 3.4, 0.29, 7.3 and 0.28. Generic links pay up to 2% for the test
// and the call beside it (24^4 force 705 -> 711 us, 32^4 stout force 23.49 ->
// 23.64 ms): a called function's registers count in its caller.
#pragma once
#include "fxlat.cuh"

namespace gf {

struct row64 {
  double re[3], im[3];
};
// a matrix of the block's links in shared memory (FxOperand or FxRaw storage)
struct Sh64 {
  double2 (*v)[GF_FX_LINKS];
  int link;
  __device__ __forceinline__ double2 operator()(int el) const { return v[el][link]; }
};
template <class STORE>
__device__ __forceinline__ Sh64 sh64(STORE& m, int link) {
  static_assert(sizeof(STORE) >= 9 * GF_FX_LINKS * sizeof(double2), "a matrix per link");
  return Sh64{reinterpret_cast<double2(*)[GF_FX_LINKS]>(&m), link};
}
__device__ __forceinline__ void share64(const Sh64& sh, int r, const row64& a) {
#pragma unroll
  for (int j = 0; j < 3; ++j) sh.v[3 * r + j][sh.link] = make_double2(a.re[j], a.im[j]);
}
// row r of M or of its dagger
template <bool DAG, class MAT>
__device__ __forceinline__ row64 load_row64(const MAT& M, int r) {
  row64 a;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double2 v = M(DAG ? 3 * k + r : 3 * r + k);
    a.re[k] = v.x;
    a.im[k] = DAG ? -v.y : v.y;
  }
  return a;
}
// a M or a M^dag
template <bool DAG, class MAT>
__device__ __forceinline__ row64 mul64(const row64& a, const MAT& M) {
  row64 c;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    double re = 0.0, im = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      double2 b = M(DAG ? 3 * j + k : 3 * k + j);
      if (DAG) b.y = -b.y;
      re = fma(a.re[k], b.x, re);
      im = fma(a.re[k], b.y, im);
      re = fma(-a.im[k], b.y, re);
      im = fma(a.im[k], b.x, im);
    }
    c.re[j] = re;
    c.im[j] = im;
  }
  return c;
}
template <class MAT>
__device__ __forceinline__ row64 mul64(const row64& a, const MAT& M, bool dag) {
  return dag ? mul64<true>(a, M) : mul64<false>(a, M);
}
__device__ __forceinline__ row64 zero64() { return row64{{0, 0, 0}, {0, 0, 0}}; }
// acc += s a
__device__ __forceinline__ void add64(row64& acc, const row64& a, double s = 1.0) {
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    acc.re[j] = fma(s, a.re[j], acc.re[j]);
    acc.im[j] = fma(s, a.im[j], acc.im[j]);
  }
}
// acc += (sr + i si) a
__device__ __forceinline__ void cadd64(row64& acc, double sr, double si, const row64& a) {
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    acc.re[j] = fma(sr, a.re[j], fma(-si, a.im[j], acc.re[j]));
    acc.im[j] = fma(sr, a.im[j], fma(si, a.re[j], acc.im[j]));
  }
}
__device__ __forceinline__ double pick64(double a, double b, double c, int r) { return r == 0 ? a : (r == 1 ? b : c); }

// row r of V = S^dag, the staple sum (fx_add_staples)
__device__ __forceinline__ row64 staple_row64(const FxField& U, const Geom& g, const Site& st, int s, int mu, int r) {
  const int V = g.vol, mu_up = fx_up(g, st, mu);
  const int xpm = eo_of_lex(g, st.lex + mu_up, st.par ^ 1);
  row64 acc = zero64();
#pragma unroll 1
  for (int k = 1; k < 4; ++k) {
    const int nu = (mu + k) & 3, dn = fx_down(g, st, nu);
    const int xpn = eo_of_lex(g, st.lex + fx_up(g, st, nu), st.par ^ 1);
    const int xmn = eo_of_lex(g, st.lex + dn, st.par ^ 1);
    const int xpm_mn = eo_of_lex(g, st.lex + mu_up + dn, st.par);
    row64 t = mul64<false>(load_row64<false>(fx_mat64(U, nu, s, V), r), fx_mat64(U, mu, xpn, V));
    add64(acc, mul64<true>(t, fx_mat64(U, nu, xpm, V)));
    t = mul64<false>(load_row64<true>(fx_mat64(U, nu, xmn, V), r), fx_mat64(U, mu, xmn, V));
    add64(acc, mul64<false>(t, fx_mat64(U, nu, xpm_mn, V)));
  }
  return acc;
}

// fx_update_mom for the links that it leaves out: P <- keep P + coef c(M), M the
// block's fp64 matrices
__device__ __forceinline__ void update_mom64(const Sh64& m, const int* se, double* __restrict__ P, int mu, int s0,
                                             int V, double coef, double keep) {
  const int part = threadIdx.x >> 5, s = s0 + m.link;
  if (s >= V || !fx_has_f64(se[m.link])) return;
  const int i = part == 2 ? 1 : 0, j = part == 0 ? 1 : 2;
  const double2 x = m(3 * i + j), y = m(3 * j + i);
  const double d1 = m(0).y, d2 = m(4).y, d3 = m(8).y;
  const double c[3] = {x.y + y.y, x.x - y.x, part == 0 ? d1 - d2 : (d1 + d2 - 2.0 * d3) * 0.57735026918962576451};
  const int a0 = part == 0 ? 0 : (part == 1 ? 3 : 5);
  const int a[3] = {a0, a0 + 1, part == 0 ? 2 : 7};
  double* p = P + (size_t)mu * 8 * V + s;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    if (q == 2 && part == 2) break;
    double* d = p + (size_t)a[q] * V;
    const double old = keep != 0.0 ? keep * *d : 0.0;
    *d = fma(coef, c[q], old);
  }
}

// a link's matrix, or its dagger, into a field
__device__ __forceinline__ void store_field64(const Sh64& m, char* p, int mu, int s, int V, bool dag = false) {
  double e[18];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const double2 v = m(dag ? 3 * (k % 3) + k / 3 : k);
    e[2 * k] = v.x;
    e[2 * k + 1] = dag ? -v.y : v.y;
  }
  fx_store64(p, mu, s, V, e);
}

// halvings that bring |X| to 1, from |X|^2 <= (2/3) tr X^2; at most one more than
// leave the phases of exp(iX) any digit, and none for what is not finite
__device__ __forceinline__ int halvings64(double trx2) {
  int n = 0;
  for (double x = trx2 * (2.0 / 3.0); x > 1.0 && n <= GF_FX_MAX_POW2 && x <= 1.7976931348623157e308; x *= 0.25) ++n;
  return n;
}
__device__ __forceinline__ double halve64(int n) {
  return n > GF_FX_MAX_POW2 ? __longlong_as_double(0x7FF8000000000000ll) : scalbn(1.0, -n);
}
// X = -i TA(rho m) of a matrix, Hermitian, and the halvings that bring |X| to 1
__device__ __forceinline__ mat3<double> ta_herm64(const Sh64& m, double rho, int& halvings) {
  mat3<double> q;
  const double d[3] = {m(0).y, m(4).y, m(8).y}, tr = (d[0] + d[1] + d[2]) * (1.0 / 3.0);
  double n2 = 0.0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    q.e[i][i] = mk(rho * (d[i] - tr), 0.0);
    n2 += q.e[i][i].re * q.e[i][i].re;
#pragma unroll
    for (int j = i + 1; j < 3; ++j) {
      const double2 x = m(3 * i + j), y = m(3 * j + i);
      q.e[i][j] = mk(0.5 * rho * (x.y + y.y), -0.5 * rho * (x.x - y.x));
      q.e[j][i] = conj(q.e[i][j]);
      n2 += 2.0 * (q.e[i][j].re * q.e[i][j].re + q.e[i][j].im * q.e[i][j].im);
    }
  }
  halvings = halvings64(n2);
  return scale(halve64(halvings), q);
}

}  // namespace gf
