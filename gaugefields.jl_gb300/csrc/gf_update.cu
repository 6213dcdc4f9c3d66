// Link update U <- exp(i eps P) U (update_gaugefields!,
// src/molecular_dynamics.jl:513-531; exptU!, src/4D/TA_gaugefields_4D_serial.jl:760)
// with the Cayley-Hamilton exponential, optional re-unitarisation
// (normalize3!, src/AbstractGaugefields.jl:3378) and an optional fp32
// 12-real shadow copy for the mixed-precision force path. One kernel for every
// precision form: fp64 storage, fixed-point arithmetic of fp64 class.
#include "gf_internal.h"
#include "fxrows64.cuh"

namespace gf {

// In block fixed point (fixed.cuh), a thread per link.
struct FxRegMat {
  const int4* m;
  __device__ __forceinline__ int4 operator()(int el) const { return m[el]; }
};
struct FxHermMat {
  const fx_herm& q;
  __device__ __forceinline__ int4 operator()(int el) const { return fx_herm_element(q, el / 3, el % 3); }
};
__device__ __forceinline__ fx_row fx_reg_row(const int4* m) {
  fx_row a;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    a.ah[k] = m[k].x;
    a.al[k] = m[k].y;
    a.bh[k] = m[k].z;
    a.bl[k] = m[k].w;
  }
  return a;
}
__device__ __forceinline__ void fx_reg_store(int4* m, const fx_acc& v) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    fx_split<0>(v.re[k], m[k].x, m[k].y);
    fx_split<0>(v.im[k], m[k].z, m[k].w);
  }
}
// E <- E^(2^n), out of line: only |X| > 2 comes here
__device__ __noinline__ void fx_square_often(int4* E, int n) {
  int4 T[9];
#pragma unroll 1
  for (int k = 0; k < n; ++k) {
#pragma unroll 1
    for (int r = 0; r < 3; ++r) fx_reg_store(T + 3 * r, fx_row_mul<false>(fx_reg_row(E + 3 * r), FxRegMat{E}));
#pragma unroll 1
    for (int i = 0; i < 9; ++i) E[i] = T[i];
  }
}

// unit row: v / |v|; false for a zero row
__device__ __forceinline__ bool fx_unit_row(fx_acc& v) {
  const float f = fx_square(v);
  const int d = fx_norm_shift(f, 0);
  fx_sum n2 = fx_zero_sum();
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    v.re[j] = fx_shift(v.re[j], d);
    v.im[j] = fx_shift(v.im[j], d);
    const fx_num a = fx_pre(v.re[j]), b = fx_pre(v.im[j]);
    fx_mac(n2, a, a);
    fx_mac(n2, b, b);
  }
  // |v|^2 in (1/16, 1]: to [1/2, 2) by powers of 4
  i64 m = fx_get(n2);
  const int k = m >= (1ll << 59) ? 0 : (m >= (1ll << 57) ? 1 : 2);
  m <<= 2 * k;
  const fx_num y = fx_pre(fx_rsqrt(m, rsqrtf((float)(int)(m >> 32) * 3.7252902984619140625e-9f)));
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    v.re[j] = fx_mul(fx_pre(v.re[j] << k), y);
    v.im[j] = fx_mul(fx_pre(v.im[j] << k), y);
  }
  return f > 0.f;
}
// X = eps sum_a p_a lambda_a / 2 as entries and exponent
__device__ __forceinline__ fx_herm fx_mom_herm(const double* __restrict__ P, int mu, int s, int V, fx_scalar eps,
                                               int& e) {
  double p[8];
  int emax = 1;
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    p[a] = P[((size_t)mu * 8 + a) * V + s];
    emax = max(emax, fx_exponent_field(p[a]));
  }
  i64 R[8];
#pragma unroll
  for (int a = 0; a < 8; ++a) R[a] = fx_mantissa(p[a], emax, 1);
  const i64 c7 = fx_mul(fx_pre(R[7]), fx_pre(665639541039271463ll));  // 2^60 / sqrt(3)
  const i64 h[9] = {(R[2] + c7) >> 1, (c7 - R[2]) >> 1, 0, R[0] >> 1, R[3] >> 1, R[5] >> 1,
                    -(R[1] >> 1),     -(R[4] >> 1),     -(R[6] >> 1)};
  fx_herm q;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    q.d[k] = fx_mul(fx_pre(h[k]), fx_num_of(eps));
    q.re[k] = fx_mul(fx_pre(h[3 + k]), fx_num_of(eps));
    q.im[k] = fx_mul(fx_pre(h[6 + k]), fx_num_of(eps));
  }
  q.d[2] = -q.d[0] - q.d[1];
  e = emax == 0x7FF ? GF_FX_BAD : emax - 1022 + eps.e;
  return q;
}

// b <- unit row of b - <a, b> a, a a unit row; false when nothing is left
__device__ __forceinline__ bool fx_orthonormal_row(fx_acc& b, const fx_acc& a) {
  fx_num ar[3], ai[3];
  // relative to its own size, so that the projection keeps its digits
  const int d = fx_norm_shift(fx_square(b), 0);
  fx_sum pr = fx_zero_sum(), pi = fx_zero_sum();
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    b.re[j] = fx_shift(b.re[j], d);
    b.im[j] = fx_shift(b.im[j], d);
    ar[j] = fx_pre(a.re[j]);
    ai[j] = fx_pre(a.im[j]);
    fx_cmac(pr, pi, fx_pre(b.re[j]), fx_pre(b.im[j]), ar[j], fx_neg(ai[j]));
  }
  const fx_num xr = fx_pre(fx_get(pr)), xi = fx_pre(fx_get(pi));
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    fx_sum yr = fx_zero_sum(), yi = fx_zero_sum();
    fx_cmac(yr, yi, xr, xi, ar[j], ai[j]);
    b.re[j] -= fx_get(yr);
    b.im[j] -= fx_get(yi);
  }
  return fx_unit_row(b);
}
// conj(a x b)
__device__ __forceinline__ fx_acc fx_cross_row(const fx_acc& a, const fx_acc& b) {
  const fx_row x = fx_operand<0>(a), y = fx_operand<0>(b);
  fx_acc c;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int k = (j + 1) % 3, l = (j + 2) % 3;
    const fx_num ark{x.ah[k], x.al[k]}, aik{x.bh[k], x.bl[k]}, arl{x.ah[l], x.al[l]}, ail{x.bh[l], x.bl[l]};
    const fx_num brk{y.ah[k], y.al[k]}, bik{y.bh[k], y.bl[k]}, brl{y.ah[l], y.al[l]}, bil{y.bh[l], y.bl[l]};
    fx_sum re = fx_zero_sum(), im = fx_zero_sum();
    fx_cmac(re, im, ark, aik, brl, bil);
    fx_cmac(re, im, fx_neg(arl), fx_neg(ail), brk, bik);
    c.re[j] = fx_get(re);
    c.im[j] = -fx_get(im);
  }
  return c;
}
// rows a, b -> orthonormal, c = conj(a x b) (normalize3!,
// src/AbstractGaugefields.jl:3378). Returns how many rows are defined.
__device__ __forceinline__ int fx_unitarise(fx_acc w[3]) {
  if (!fx_unit_row(w[0])) return 0;
  if (!fx_orthonormal_row(w[1], w[0])) return 1;
  w[2] = fx_cross_row(w[0], w[1]);
  return 3;
}

// whether a link's update takes the fp64 path (update_link64)
__device__ __forceinline__ bool fx_patterned(const double* m, int unit) {
  unsigned small = 0;
#pragma unroll
  for (int i = 0; i < 18; ++i) small |= (unsigned)fx_is_small(m[i], unit) << i;
  return fx_small_pattern(small);
}
// links of a matrix from fp64, the exponent from its Frobenius norm
// the same out of line, of a stored link
__device__ __noinline__ bool fx_patterned(const double2* U, int mu, int s, int V, int unit) {
  const double2* b = U + (size_t)mu * 9 * V + s;
  unsigned small = 0;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const double2 v = b[(size_t)k * V];
    small |= (unsigned)fx_is_small(v.x, unit) << (2 * k) | (unsigned)fx_is_small(v.y, unit) << (2 * k + 1);
  }
  return fx_small_pattern(small);
}
// small: how many entries are below 2^-7 of the unit, unit: for fx_patterned
__device__ __forceinline__ int fx_from_f64_fast(const double* m, int4 out[9], int& small, int& unit) {
  int emax = 1;
#pragma unroll
  for (int i = 0; i < 18; ++i) emax = max(emax, fx_exponent_field(m[i]));
  float n = 0.f, f[18];
#pragma unroll
  for (int i = 0; i < 18; ++i) {
    f[i] = fx_leading(m[i], emax);
    n = fmaf(f[i], f[i], n);
  }
  const int up = (n > 0.999f) + (n > 3.996f) + (n > 15.98f) + (n > 63.9f);
  const bool bad = emax == 0x7FF;
  // entries below 2^-7 of the spectral norm, half the Frobenius norm's power of two
  const float tiny = 0.00390625f * (float)(1 << up);
  small = 0;
#pragma unroll
  for (int i = 0; i < 18; ++i) small += fabsf(f[i]) < tiny;
  if (bad) small = 0;
  unit = emax + up - 1;
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    fx_split<0>(bad ? 0 : fx_mantissa(m[2 * i], emax, up), out[i].x, out[i].y);
    fx_split<0>(bad ? 0 : fx_mantissa(m[2 * i + 1], emax, up), out[i].z, out[i].w);
  }
  return bad ? GF_FX_BAD : emax - 1023 + up;
}

// an element of a unitary matrix, exponent 0, or kept in fp64
__device__ __forceinline__ int4 fx_unitary_element(double2 v, bool ok, bool f64) {
  int4 o;
  if (f64) return fx_pack64(v.x, v.y);
  fx_split<0>(ok ? fx_mantissa(v.x, 1023, 0) : 0, o.x, o.y);
  fx_split<0>(ok ? fx_mantissa(v.y, 1023, 0) : 0, o.z, o.w);
  return o;
}
__device__ __forceinline__ fx_acc fx_shared_row(const FxRaw& m, int link, int r) {
  fx_acc v;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    v.re[j] = m.v[2 * (3 * r + j)][link];
    v.im[j] = m.v[2 * (3 * r + j) + 1][link];
  }
  return v;
}

// W = exp(i eps P) U of one link in fp64, where U is near the identity or has
// another pattern of small entries (fx_small_pattern; exact zeros count, for
// what the momentum puts in their place): stored like the others.
template <bool REUNIT>
__device__ __noinline__ void update_link64(const double2* Uin, double2* Uout, const double* __restrict__ P, int mu,
                                           int s, int V, double eps, float4* sh32, char* fx) {
  mat3<double> u;
  const double2* b = Uin + (size_t)mu * 9 * V + s;
#pragma unroll
  for (int k = 0; k < 9; ++k) u.e[k / 3][k % 3] = mk(b[(size_t)k * V].x, b[(size_t)k * V].y);
  const double* p = P + (size_t)mu * 8 * V + s;
  double c[8];
#pragma unroll
  for (int a = 0; a < 8; ++a) c[a] = 0.5 * eps * p[(size_t)a * V];
  mat3<double> q;
  const double d = c[7] * 0.57735026918962576451;
  q.e[0][0] = mk(c[2] + d, 0.0);
  q.e[1][1] = mk(d - c[2], 0.0);
  q.e[2][2] = mk(-2.0 * d, 0.0);
  q.e[0][1] = mk(c[0], -c[1]);
  q.e[0][2] = mk(c[3], -c[4]);
  q.e[1][2] = mk(c[5], -c[6]);
  double n2 = 2.0 * (c[0] * c[0] + c[1] * c[1] + c[3] * c[3] + c[4] * c[4] + c[5] * c[5] + c[6] * c[6]);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    n2 += q.e[i][i].re * q.e[i][i].re;
#pragma unroll
    for (int j = 0; j < i; ++j) q.e[i][j] = conj(q.e[j][i]);
  }
  // halved to |X| <= 1, and squared afterwards
  const int halvings = halvings64(n2);
  mat3<double> E = expiq(scale(halve64(halvings), q));
#pragma unroll 1
  for (int k = 0; k < halvings; ++k) E = mul_nn(E, E);
  u = mul_nn(E, u);
  if (REUNIT) reunitarize(u);
  LinkFull<double>::store(Uout, mu, s, V, u);
  if (sh32) {
    mat3<float> h;
#pragma unroll
    for (int k = 0; k < 6; ++k) h.e[k / 3][k % 3] = mk((float)u.e[k / 3][k % 3].re, (float)u.e[k / 3][k % 3].im);
    Link12f::store(sh32, mu, s, V, h);
  }
  if (fx) fx_store64(fx, mu, s, V, &u.e[0][0].re);
}
// blocks per SM of the link update
#ifndef GF_FX_UPDATE_MINB
#define GF_FX_UPDATE_MINB 4
#endif
// W = exp(i eps P) U on fp64 links (Uin, Uout may be the same field). Bound by
// integer issue: 48^4 4.55 ms, where the double-float kernel took 7.18 ms and
// the fp64 one 20 ms; four blocks per SM (128 registers) against 4.88 ms with
// two or three, and 7.85 ms for a row of the link per thread, whose series and
// row-after-row re-unitarisation leave warps waiting at barriers. Against
// 113-bit arithmetic the result is off by 4.9e-17 (the final rounding), the
// fp64 kernel's by 1.6e-16, the double-float one's by 6.2e-15.
template <bool REUNIT>
__global__ void __launch_bounds__(128, GF_FX_UPDATE_MINB)
    k_link_update_fx(const double2* Uin, double2* Uout, const double* __restrict__ P, const __grid_constant__ Geom g,
                     fx_scalar eps, double eps64, float4* __restrict__ sh32, char* __restrict__ fx) {
  const int V = g.vol, mu = blockIdx.y, s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V) return;
  constexpr int rows = REUNIT ? 2 : 3;  // re-unitarisation rebuilds row 3
  int e;
  fx_herm q = fx_mom_herm(P, mu, s, V, eps, e);
  const fx_plan plan = fx_exp_plan<false>(q, e);
  i64 f[6];
  {
    i64 c0, c1;
    fx_invariants(q, c0, c1);
    fx_ch_both(c_fx_kappa.k[plan.series], plan.guard - fx_kappa_base(plan.series), plan.terms, c0, c1, f);
  }
  int4 u[9];
  int eu, small, unit;
  {
    const double2* b = Uin + (size_t)mu * 9 * V + s;
    double m[18];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const double2 v = b[(size_t)k * V];
      m[2 * k] = v.x;
      m[2 * k + 1] = v.y;
    }
    eu = fx_from_f64_fast(m, u, small, unit);
  }
  if (e > GF_FX_BAD / 2 || plan.pow2 > GF_FX_MAX_POW2) eu = GF_FX_BAD;
  fx_acc w[3];
  const FxHermMat qm{q};
  if (plan.squares == 0) {
#pragma unroll
    for (int r = 0; r < rows; ++r) {
      const int4 row[3] = {qm(3 * r), qm(3 * r + 1), qm(3 * r + 2)};
      const fx_acc E = fx_exp_row(f, plan.guard, fx_reg_row(row), qm, r);
      w[r] = fx_row_mul<false>(fx_operand<0>(E), FxRegMat{u});
    }
  } else {
    int4 E[9];
#pragma unroll 1
    for (int r = 0; r < 3; ++r) {
      const int4 row[3] = {r == 0 ? qm(0) : (r == 1 ? qm(3) : qm(6)), r == 0 ? qm(1) : (r == 1 ? qm(4) : qm(7)),
                           r == 0 ? qm(2) : (r == 1 ? qm(5) : qm(8))};
      fx_reg_store(E + 3 * r, fx_exp_row(f, plan.guard, fx_reg_row(row), qm, r));
    }
    fx_square_often(E, plan.squares);
#pragma unroll
    for (int r = 0; r < rows; ++r) w[r] = fx_row_mul<false>(fx_reg_row(E + 3 * r), FxRegMat{u});
  }
  int fine = 3;
  if (REUNIT) {
    fine = eu > GF_FX_BAD / 2 ? 0 : fx_unitarise(w);
    eu = 0;
  }
  // here, where least is alive across the calls
  if (small >= GF_FX_PATTERN_MIN && fx_patterned(Uin, mu, s, V, unit)) {
    update_link64<REUNIT>(Uin, Uout, P, mu, s, V, eps64, sh32, fx);
    return;
  }
  double2* o = Uout + (size_t)mu * 9 * V + s;
  double2 v[9];
  const bool tiny = eu <= GF_FX_NORMAL;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int ew = k / 3 < fine ? (tiny ? eu + 1000 : eu) : GF_FX_BAD;
    v[k] = make_double2(fx_to_normal(w[k / 3].re[k % 3], ew), fx_to_normal(w[k / 3].im[k % 3], ew));
  }
  if (tiny) {
#pragma unroll
    for (int k = 0; k < 9; ++k) v[k] = make_double2(v[k].x * 0x1p-1000, v[k].y * 0x1p-1000);
  }
#pragma unroll
  for (int k = 0; k < 9; ++k) o[(size_t)k * V] = v[k];
  if (sh32) {
    float4* q4 = sh32 + (size_t)mu * 3 * V + s;
#pragma unroll
    for (int k = 0; k < 3; ++k)
      q4[(size_t)k * V] =
          make_float4((float)v[2 * k].x, (float)v[2 * k].y, (float)v[2 * k + 1].x, (float)v[2 * k + 1].y);
  }
  if (fx) {
    // the fixed-point copy of what was stored, as k_to_fx makes it
    int4 el[9];
    const size_t off = fx_offset(mu, s, V);
    bool few;
    int ef;
    if (REUNIT) {
      // a unitary matrix has exponent 0
      int n = 0;
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        el[k] = fx_unitary_element(v[k], fine == 3, false);
        n += fx_is_small(v[k].x, 1023) + fx_is_small(v[k].y, 1023);
      }
      ef = fine == 3 ? 0 : GF_FX_BAD;
      few = n >= GF_FX_PATTERN_MIN && fine == 3;
    } else {
      double m[18];
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        m[2 * k] = v[k].x;
        m[2 * k + 1] = v[k].y;
      }
      ef = fx_from_f64(m, el, few);
    }
    fx_store_exp(fx, off, s, ef);
#pragma unroll
    for (int k = 0; k < 9; ++k) *reinterpret_cast<int4*>(fx + off + 512 * k) = el[k];
    if (few) fx_regrade(Uout, fx, mu, s, V, ef);
  }
}

// The same with a warp per row of 32 links, for lattices that do not fill the
// GPU with a thread per link: there the update takes as long as one thread's
// instructions, some 6,000 of them (GF_FX_ROWS_MAX has the figures). Warps 0
// and 1 form the real and imaginary parts of the series while warp 2 brings U to
// fixed point. Same results as above.
struct FxUpdateRows {
  FxExp x;      // x.m: the finished rows
  FxOperand u;  // U, then (no re-unitarisation) the fp64 result
  int eu[GF_FX_LINKS];
  int fine[GF_FX_LINKS];
  int patterned[GF_FX_LINKS];     // the link's update runs in fp64
  unsigned small[3][GF_FX_LINKS];  // by rows: small entries of the result, bit 6 if one is not zero
};
template <bool REUNIT>
__global__ void __launch_bounds__(GF_FX_THREADS, 4)
    k_link_update_rows_fx(const double2* Uin, double2* Uout, const double* __restrict__ P, const __grid_constant__ Geom g,
                          fx_scalar eps, double eps64, float4* __restrict__ sh32, char* __restrict__ fx) {
  __shared__ FxUpdateRows sh;
  const int V = g.vol, mu = blockIdx.y, link = threadIdx.x & 31, r = threadIdx.x >> 5;
  const int sx = blockIdx.x * GF_FX_LINKS + link, s = min(sx, V - 1);
  if (r < 2) {
    int e;
    fx_herm q = fx_mom_herm(P, mu, s, V, eps, e);
    const fx_plan plan = fx_exp_plan<false>(q, e);
    i64 c0, c1, f[3], b1[3], b2[3];
    fx_invariants(q, c0, c1);
    fx_ch<false>(c_fx_kappa.k[plan.series], plan.guard - fx_kappa_base(plan.series), plan.terms, r, c0, c1, f, b1, b2);
#pragma unroll
    for (int j = 0; j < 3; ++j) sh.x.f[2 * j + r][link] = f[j];
    if (r == 0) {
#pragma unroll
      for (int el = 0; el < 9; ++el) sh.x.q.v[el][link] = fx_herm_element(q, el / 3, el % 3);
      sh.x.e[link] = plan.pow2 > GF_FX_MAX_POW2 ? GF_FX_BAD : e;
      sh.x.g[link] = plan.guard;
      sh.x.sq[link] = plan.squares;
      const int most = __reduce_max_sync(0xffffffffu, plan.squares);
      if (link == 0) sh.x.most = most;
    }
  } else {
    const double2* b = Uin + (size_t)mu * 9 * V + s;
    double m[18];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const double2 v = b[(size_t)k * V];
      m[2 * k] = v.x;
      m[2 * k + 1] = v.y;
    }
    int4 u[9];
    int small, unit;
    sh.eu[link] = fx_from_f64_fast(m, u, small, unit);
    sh.patterned[link] = small >= GF_FX_PATTERN_MIN && fx_patterned(m, unit);
#pragma unroll
    for (int k = 0; k < 9; ++k) sh.u.v[k][link] = u[k];
  }
  __syncthreads();
  const fx_acc E = fx_exp_row_squared(sh.x, link, r);
  fx_acc w = {{0, 0, 0}, {0, 0, 0}};
  if (!REUNIT || r < 2) w = fx_row_mul<false>(fx_operand<0>(E), FxShMat{&sh.u, link});
  int eu = sh.x.e[link] > GF_FX_BAD / 2 ? GF_FX_BAD : sh.eu[link], fine = 3;
  if (REUNIT) {
    if (r == 0) {
      const bool ok = fx_unit_row(w);
      sh.fine[link] = ok && eu <= GF_FX_BAD / 2 ? 3 : 0;
      fx_share(sh.x.m, link, 0, w);
    }
    __syncthreads();
    if (r == 1) {
      if (!fx_orthonormal_row(w, fx_shared_row(sh.x.m, link, 0)) && sh.fine[link] == 3) sh.fine[link] = 1;
      fx_share(sh.x.m, link, 1, w);
    }
    __syncthreads();
    if (r == 2) w = fx_cross_row(fx_shared_row(sh.x.m, link, 0), fx_shared_row(sh.x.m, link, 1));
    fine = sh.fine[link];
    eu = 0;
  }
  double2 v[3];
  const bool tiny = eu <= GF_FX_NORMAL;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int ew = r < fine ? (tiny ? eu + 1000 : eu) : GF_FX_BAD;
    v[j] = make_double2(fx_to_normal(w.re[j], ew), fx_to_normal(w.im[j], ew));
    if (tiny) v[j] = make_double2(v[j].x * 0x1p-1000, v[j].y * 0x1p-1000);
  }
  const size_t off = fx_offset(mu, s, V);
  int4 el[3];
  int ef = fine == 3 ? 0 : GF_FX_BAD;
  if (fx && REUNIT) {
    unsigned small = 0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      small |= (unsigned)fx_is_small(v[j].x, 1023) << (2 * j) | (unsigned)fx_is_small(v[j].y, 1023) << (2 * j + 1);
      small |= (unsigned)(fx_small_nonzero(v[j].x, 1023) || fx_small_nonzero(v[j].y, 1023)) << 6;
    }
    sh.small[r][link] = small;
    __syncthreads();
    const unsigned a = sh.small[0][link], b = sh.small[1][link], c = sh.small[2][link];
    const bool f64 =
        fine == 3 && ((a | b | c) & 64) && fx_small_pattern((a & 63) | (b & 63) << 6 | (c & 63) << 12);
    if (f64) ef = GF_FX_F64;
#pragma unroll
    for (int j = 0; j < 3; ++j) el[j] = fx_unitary_element(v[j], fine == 3, f64);
  } else if (fx) {
    double2* x = reinterpret_cast<double2*>(sh.u.v) + link;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 3; ++j) x[(3 * r + j) * GF_FX_LINKS] = v[j];
    __syncthreads();
    double m[18];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      m[2 * k] = x[k * GF_FX_LINKS].x;
      m[2 * k + 1] = x[k * GF_FX_LINKS].y;
    }
    int emax, up, small;
    const bool bad = !fx_exponent_of(m, emax, up, small);
    const bool f64 = !bad && small >= GF_FX_PATTERN_MIN && fx_graded(m, emax + up);
    ef = bad ? GF_FX_BAD : (f64 ? GF_FX_F64 : emax - 1023 + up);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      fx_split<0>(bad ? 0 : fx_mantissa(v[j].x, emax, up), el[j].x, el[j].y);
      fx_split<0>(bad ? 0 : fx_mantissa(v[j].y, emax, up), el[j].z, el[j].w);
      if (f64) el[j] = fx_pack64(v[j].x, v[j].y);
    }
  }
  if (sx >= V) return;
  if (sh.patterned[link]) {
    if (r == 2) update_link64<REUNIT>(Uin, Uout, P, mu, s, V, eps64, sh32, fx);
    return;
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int k = 3 * r + j;
    Uout[((size_t)mu * 9 + k) * V + s] = v[j];
    if (sh32 && r < 2)  // complex element k of float4 [3][V]
      reinterpret_cast<float2*>(sh32)[2 * ((size_t)(mu * 3 + k / 2) * V + s) + (k & 1)] =
          make_float2((float)v[j].x, (float)v[j].y);
    if (fx) *reinterpret_cast<int4*>(fx + off + 512 * k) = el[j];
  }
  if (fx && r == 0) *reinterpret_cast<int*>(fx + off + 9 * 512 - 12 * (s & 31)) = ef;
}

// The update writes the fixed-point copy itself: a launch and the copy's pass
// over the links less. A copy kernel after it against this one: trajectories
// 8^4 (10 steps) 445 / 389 us, 16^4 2.37 / 2.31 ms, 24^4 11.25 / 10.92, 40^4 (2
// steps) 22.0 / 21.6. Without re-unitarisation (flows) the copy needs the
// bound of its exponent, for which this kernel has no registers left: 8^4 (3 steps)
// 284 / 247 us, 12^4 742 / 706, 16^4 1.86 / 1.85 ms, but on 166,320 sites (5
// steps) 7.17 / 7.25, 32^4 (2 steps) 18.52 / 18.62.
#ifndef GF_FX_FUSE_PLAIN_MAX
#define GF_FX_FUSE_PLAIN_MAX (1 << 16)
#endif
// Sites up to which a link gets a warp lane in each of three warps. Trajectory
// of 20 steps (without re-unitarisation, flow of 5 steps), a thread per link
// against rows: 4^4 502 (311) against 462 (251) us, 6^4 572 (343) against 522
// (282), 8^4 710 (437) against 674 (406); at 10^4 the GPU is full and the
// rows' barriers cost, 1134 (737) against 1167 (763), at 32^4 the update takes
// 0.91 against 1.54 ms.
#ifndef GF_FX_ROWS_MAX
#define GF_FX_ROWS_MAX 6144
#endif
static void update_links(gf_ctx* ctx, gf_field* W, const gf_field* P, double eps, const gf_field* U, int reunit,
                         gf_field* shadow32, gf_field* fx) {
  const int V = ctx->geom.vol;
  const bool rows = V <= GF_FX_ROWS_MAX, fused = reunit || V <= GF_FX_FUSE_PLAIN_MAX;
  const int threads = rows ? GF_FX_THREADS : 128;
  dim3 grid(blocks_for(V, rows ? GF_FX_LINKS : 128), 4);
  auto kern = rows ? (reunit ? k_link_update_rows_fx<true> : k_link_update_rows_fx<false>)
                   : (reunit ? k_link_update_fx<true> : k_link_update_fx<false>);
  kern<<<grid, threads, 0, ctx->stream>>>((const double2*)U->ptr, (double2*)W->ptr, (const double*)P->ptr, ctx->geom,
                                      fx_scalar_of(eps), eps, shadow32 ? (float4*)shadow32->ptr : nullptr,
                                      fx && fused ? (char*)fx->ptr : nullptr);
  GF_CHECK_LAUNCH();
  if (fx && !fused) to_fx(ctx, fx, W);
}

void link_update(gf_ctx* ctx, gf_field* U, const gf_field* P, double eps, int reunit, gf_field* shadow32, bool df,
                 gf_field* fx) {
  if (U->kind != GF_LINK64) throw gf_error(GF_EINVAL, "link update: U must be LINK64");
  if (P->kind != GF_MOM64) throw gf_error(GF_EINVAL, "link update: P must be MOM64");
  ProfScope prof(ctx, df ? GF_K_LINK_UPDATE_DF : GF_K_LINK_UPDATE);
  update_links(ctx, U, P, eps, U, reunit, shadow32, fx);
}

// exp_aF_U!(W, a, F, U) (src/AbstractGaugefields.jl:2810-2842): W_mu = exp(a F_mu) U_mu
// with F in su(3) coefficients, i.e. exp(i a sum_a F_a lambda_a / 2) U.
void exp_mom_links(gf_ctx* ctx, gf_field* W, const gf_field* P, double a, const gf_field* U, bool df, gf_field* fx) {
  ProfScope prof(ctx, df ? GF_K_LINK_UPDATE_DF : GF_K_LINK_UPDATE);
  update_links(ctx, W, P, a, U, 0, nullptr, fx);
}

__global__ void k_reunit(double2* __restrict__ U, int V) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  int mu = blockIdx.y;
  if (s >= V) return;
  mat3<double> u = LinkFull<double>::load(U, mu, s, V);
  reunitarize(u);
  LinkFull<double>::store(U, mu, s, V, u);
}

void reunitarize_links(gf_ctx* ctx, gf_field* U) {
  if (U->kind != GF_LINK64) throw gf_error(GF_EINVAL, "reunitarize: U must be LINK64");
  dim3 grid(blocks_for(ctx->geom.vol, 128), 4);
  k_reunit<<<grid, 128, 0, ctx->stream>>>((double2*)U->ptr, ctx->geom.vol);
  GF_CHECK_LAUNCH();
}

}  // namespace gf
