// Block fixed-point arithmetic on the integer pipes, for fp64-class 3x3 work.
//
// GB300 issues one fp64 multiply-add per 64 fp32 ones, but a 32 x 32 + 64 bit
// integer multiply-add (IMAD.WIDE) per four (measured: 3.95 cycles per warp
// and scheduler). A product of two 60-bit fixed-point numbers kept as limbs of
// 30 bits needs three of them (high x high and the two cross terms), so a
// real multiply-add costs 12 issue slots instead of 64, with an absolute
// error of about 2^-59 of the operands' norms, below fp64's rounding of anything
// but entries under 2^-7 of the norm (fx_graded).
//
// A matrix is 18 integers R with one exponent E: value = R 2^(E - 60). E is
// chosen so that the matrix's spectral norm is at most 1 + 2^-11 in units of
// 2^E (unitary links have E = 0 and lose no bit): every entry, every row and
// every column norm is then at most about 2^60, a product of such matrices is
// again one (the spectral norm is submultiplicative), and the 64-bit sums
// below cannot overflow. An operand holds R as h 2^30 + l with l in
// [0, 2^30); |h| <= 2^30 (1 + 2^-10).
//
// Products are formed by rows: a thread owns row r of the left factor and
// multiplies it by whole matrices, row(A) B, so chains of products
// row(A) B C ... need no exchange between the threads of a link, keep their
// state in registers (12 + 12 words) and give three threads per link.
// The complex products take three real ones (Gauss): with a = Re A, b = Im A,
// c = Re B, d = Im B,
//   k = a (c + d),  Re = k - d (a + b),  Im = k + c (b - a),
// exact in integer arithmetic (intermediate wrap-around cancels modulo 2^64
// because the final sums fit). 27 multiply-adds per entry instead of 36.
#pragma once
#include "lattice.cuh"

namespace gf {

typedef long long i64;
typedef unsigned long long u64;

#define GF_FX_MASK 0x3FFFFFFF
// exponent of a matrix holding a NaN or an infinity; sums of exponents keep
// it recognisable (every regular exponent sum is far below GF_FX_BAD / 2)
#define GF_FX_BAD (1 << 24)
// "exponent" of a matrix whose slot holds its fp64 entries (fx_graded). A sum of
// exponents with one among them is at least GF_FX_F64_SUM, any other (up to
// seven GF_FX_BAD) below.
#define GF_FX_F64 (1 << 27)
#define GF_FX_F64_SUM (15 << 23)

struct fx_row {  // operand: row of a left factor, a = Re, b = Im
  int ah[3], al[3], bh[3], bl[3];
};
struct fx_acc {  // raw 64-bit row
  i64 re[3], im[3];
};

GF_HD i64 fx_join(int h, int l) { return ((i64)h << 30) + l; }

// limbs of R / 2^K
template <int K>
GF_HD void fx_split(i64 R, int& h, int& l) {
  h = (int)(R >> (30 + K));
  l = (int)(R >> K) & GF_FX_MASK;
}
template <int K>
GF_HD fx_row fx_operand(const fx_acc& v) {
  fx_row r;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    fx_split<K>(v.re[j], r.ah[j], r.al[j]);
    fx_split<K>(v.im[j], r.bh[j], r.bl[j]);
  }
  return r;
}

// a b + c, the product in PTX: written in C, with limbs that the compiler knows
// not to be negative, it measured slower, and so did mad.wide.
GF_HD i64 fx_mad(int a, int b, i64 c) {
#ifdef __CUDA_ARCH__
  i64 d;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(d) : "r"(a), "r"(b));
  return d + c;
#else
  return (i64)a * b + c;
#endif
}

// row(A) op(B), op = identity or dagger; B(e) returns element e of the
// row-major matrix as int4 (re.h, re.l, im.h, im.l). Unit 2^(EA + EB - 60).
template <bool DAG, class MAT>
GF_HD fx_acc fx_row_mul(const fx_row& A, const MAT& B) {
  int ph[3], pl[3], qh[3], ql[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    ph[k] = DAG ? A.ah[k] + A.bh[k] : -A.ah[k] - A.bh[k];
    pl[k] = DAG ? A.al[k] + A.bl[k] : -A.al[k] - A.bl[k];
    qh[k] = A.bh[k] - A.ah[k];
    ql[k] = A.bl[k] - A.al[k];
  }
  fx_acc out;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    int4 b[3];
    i64 kh = 0, kx = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      b[k] = B(DAG ? 3 * j + k : 3 * k + j);
      const int sh = DAG ? b[k].x - b[k].z : b[k].x + b[k].z;
      const int sl = DAG ? b[k].y - b[k].w : b[k].y + b[k].w;
      kh = fx_mad(A.ah[k], sh, kh);
      kx = fx_mad(A.ah[k], sl, kx);
      kx = fx_mad(A.al[k], sh, kx);
    }
    i64 rh = kh, rx = kx, mh = kh, mx = kx;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      rh = fx_mad(b[k].z, ph[k], rh);
      rx = fx_mad(b[k].z, pl[k], rx);
      rx = fx_mad(b[k].w, ph[k], rx);
      mh = fx_mad(b[k].x, qh[k], mh);
      mx = fx_mad(b[k].x, ql[k], mx);
      mx = fx_mad(b[k].y, qh[k], mx);
    }
    out.re[j] = rh + (rx >> 30);
    out.im[j] = mh + (mx >> 30);
  }
  return out;
}

// acc (unit exponent ea) += v (unit exponent ev). Equal exponents, as for
// unitary links, are plain adds; otherwise the smaller one is shifted down.
GF_HD int fx_clamp_shift(int d) { return d < 0 ? 0 : (d > 63 ? 63 : d); }
GF_HD void fx_add(fx_acc& acc, int& ea, fx_acc v, int ev) {
  if (ev != ea) {
    const int da = fx_clamp_shift(ev - ea), dv = fx_clamp_shift(ea - ev);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      acc.re[j] >>= da;
      acc.im[j] >>= da;
      v.re[j] >>= dv;
      v.im[j] >>= dv;
    }
    ea = ev > ea ? ev : ea;
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    acc.re[j] += v.re[j];
    acc.im[j] += v.im[j];
  }
}

// ---------------------------------------------------------------------------
// scalars in units of 2^-60 (|value| < 2), and sums of their products
// ---------------------------------------------------------------------------
struct fx_num {
  int h, l;
};
GF_HD fx_num fx_pre(i64 R) {
  fx_num n;
  fx_split<0>(R, n.h, n.l);
  return n;
}
GF_HD fx_num fx_neg(fx_num n) {
  n.h = -n.h;
  n.l = -n.l;
  return n;
}
struct fx_sum {
  i64 hh, x;
};
GF_HD fx_sum fx_zero_sum() { return fx_sum{0, 0}; }
GF_HD void fx_mac(fx_sum& s, fx_num a, fx_num b) {
  s.hh = fx_mad(a.h, b.h, s.hh);
  s.x = fx_mad(a.h, b.l, s.x);
  s.x = fx_mad(a.l, b.h, s.x);
}
GF_HD i64 fx_get(fx_sum s) { return s.hh + (s.x >> 30); }
GF_HD i64 fx_mul(fx_num a, fx_num b) {
  fx_sum s = fx_zero_sum();
  fx_mac(s, a, b);
  return fx_get(s);
}
// (re, im) += a b for complex a, b
GF_HD void fx_cmac(fx_sum& re, fx_sum& im, fx_num ar, fx_num ai, fx_num br, fx_num bi) {
  fx_mac(re, ar, br);
  fx_mac(re, fx_neg(ai), bi);
  fx_mac(im, ar, bi);
  fx_mac(im, ai, br);
}
// R / 2^d, d of either sign, rounded
GF_HD i64 fx_shift(i64 R, int d) {
  if (d <= 0) return d > -63 ? (i64)((u64)R << -d) : 0;
  return d < 62 ? (R + (1ll << (d - 1))) >> d : 0;
}

// 1 / sqrt(m) for m in [1/2, 2), from a fp32 seed y by two Newton steps
// y <- y + y (1 - m y^2) / 2, whose relative errors go 2^-23, 2^-45, 2^-59
GF_HD i64 fx_rsqrt(i64 m, float y0) {
  const fx_num n = fx_pre(m);
  i64 y = (i64)(int)(y0 * 1073741824.f) << 30;
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const fx_num py = fx_pre(y);
    const i64 e = (1ll << 60) - fx_mul(n, fx_pre(fx_mul(py, py)));
    y += fx_mul(py, fx_pre(e)) >> 1;
  }
  return y;
}

// A kernel parameter c = (h 2^30 + l) 2^(e - 60), |h 2^30 + l| < 2^60. Zero has the
// exponent GF_FX_ZERO, below any other, so that a sum with something that it
// scales is not aligned to what it scales.
#define GF_FX_ZERO (-(1 << 18))
struct fx_scalar {
  int h, l, e;
};
inline fx_scalar fx_scalar_of(double c) {
  int e = 0;
  const double m = frexp(c, &e);  // c = m 2^e, 1/2 <= |m| < 1
  if (!(m == m) || m - m != 0.0) return fx_scalar{0, 0, GF_FX_BAD};
  fx_scalar s;
  fx_split<0>((i64)ldexp(m, 60), s.h, s.l);
  s.e = m == 0.0 ? GF_FX_ZERO : e;
  return s;
}
GF_HD fx_num fx_num_of(const fx_scalar& s) { return fx_num{s.h, s.l}; }
GF_HD void fx_scale_row(fx_acc& v, const fx_scalar& c) {
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    v.re[j] = fx_mul(fx_pre(v.re[j]), fx_num_of(c));
    v.im[j] = fx_mul(fx_pre(v.im[j]), fx_num_of(c));
  }
}

// ---------------------------------------------------------------------------
// Cayley-Hamilton exponential of iX, X = 2^s q, q traceless Hermitian with
// |q| <= 1: exp(iX) = f0 + f1 q + f2 q^2, from the power series in Horner form
// with q^3 = c1 q + c0. The coefficients are real series for their real and
// imaginary parts, which two threads evaluate side by side. They are returned
// in units of 2^(guard - 60), as are their derivatives in c1 and c0 (of q).
// ---------------------------------------------------------------------------
#define GF_FX_CH_TERMS 64  // 48 would do; lanes of two scales read it 3% faster at this distance (link update, 16^4)
#define GF_FX_CH_SCALES 3

// 2^(s n) / n! in units of 2^(base - 60), rounded
GF_HD constexpr int fx_kappa_base(int s) { return s == 0 ? 0 : (s == 1 ? 1 : 3); }
struct fx_kappa {
  i64 k[GF_FX_CH_SCALES][GF_FX_CH_TERMS];
};
constexpr fx_kappa fx_make_kappa() {
  fx_kappa t{};
  for (int s = 0; s < GF_FX_CH_SCALES; ++s) {
    unsigned __int128 v = (unsigned __int128)1 << 100;
    for (int n = 0; n < GF_FX_CH_TERMS; ++n) {
      if (n > 0) v = (v << s) / (unsigned)n;
      const int d = 40 + fx_kappa_base(s);
      t.k[s][n] = (i64)((v + ((unsigned __int128)1 << (d - 1))) >> d);
    }
  }
  return t;
}

// c1 = tr(q^2)/2 and c0 = det q; d the diagonal, o12 .. the upper entries
struct fx_herm {
  i64 d[3];
  i64 re[3], im[3];  // entries (0,1), (0,2), (1,2)
};
GF_HD void fx_invariants(const fx_herm& q, i64& c0, i64& c1) {
  fx_num d[3], re[3], im[3];
  i64 n[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    d[k] = fx_pre(q.d[k]);
    re[k] = fx_pre(q.re[k]);
    im[k] = fx_pre(q.im[k]);
    fx_sum t = fx_zero_sum();
    fx_mac(t, re[k], re[k]);
    fx_mac(t, im[k], im[k]);
    n[k] = fx_get(t);
  }
  fx_sum sq = fx_zero_sum();
#pragma unroll
  for (int k = 0; k < 3; ++k) fx_mac(sq, d[k], d[k]);
  c1 = (fx_get(sq) >> 1) + n[0] + n[1] + n[2];
  // det = d0 d1 d2 + 2 Re(q01 q12 conj(q02)) - d0 |q12|^2 - d1 |q02|^2 - d2 |q01|^2
  fx_sum tr = fx_zero_sum(), ti = fx_zero_sum();
  fx_cmac(tr, ti, re[0], im[0], re[2], im[2]);
  const fx_num t0 = fx_pre(fx_get(tr)), t1 = fx_pre(fx_get(ti));
  fx_sum r = fx_zero_sum();
  fx_mac(r, t0, re[1]);
  fx_mac(r, t1, im[1]);
  fx_sum det = fx_zero_sum();
  fx_mac(det, fx_pre(fx_mul(d[0], d[1])), d[2]);
  fx_mac(det, fx_neg(d[0]), fx_pre(n[2]));
  fx_mac(det, fx_neg(d[1]), fx_pre(n[1]));
  fx_mac(det, fx_neg(d[2]), fx_pre(n[0]));
  c0 = fx_get(det) + 2 * fx_get(r);
}

// Beyond |X| = 2^53 the phases of exp(iX) are lost in the rounding of X, in any
// arithmetic of this size: the result is a NaN.
#define GF_FX_MAX_POW2 53
// How to sum the series for a norm bound lam of X (real).
struct fx_plan {
  int pow2;     // q = X / 2^pow2
  int series;   // power of two of the series, <= pow2
  int squares;  // squarings of the result, pow2 - series
  int guard;
  int terms;
  bool beyond;  // with derivatives: |X| may exceed 4, which the series does not serve
};
// Terms: lam^n / n! < 2^-62 from n = terms - 4 on; the derivatives of the n-th
// power's coefficients go as n lam^(n - 4), so they need the four more.
// Without derivatives the series runs to |X| <= 2 and larger exponentials are
// squared from it. With them it serves |X| <= 4, the guard bits following the
// largest coefficient, a derivative of at most lam e^lam / 2 (1 / |q|)^4, half of
// it in each part: six bits at |X| = 4. (Sixteen would take 25 of the 60 bits:
// exp(iX) was off by 5e-14 at |X| = 6 and 3e-8 at 16.) Larger X: the caller's.
template <bool DERIV>
GF_HD fx_plan fx_series(float lam) {
  fx_plan p;
  p.pow2 = 0;
  for (float x = lam; x > 1.f && p.pow2 < 60; x *= 0.5f) ++p.pow2;
  p.beyond = DERIV && p.pow2 > GF_FX_CH_SCALES - 1;
  if (p.beyond) {
    p.pow2 = GF_FX_CH_SCALES - 1;
    lam = 4.f;
  }
  p.series = DERIV || p.pow2 < 1 ? p.pow2 : 1;
  p.squares = p.pow2 - p.series;
  for (int k = 0; k < p.squares; ++k) lam *= 0.5f;
  p.guard = DERIV ? 1 : 0;
  if (DERIV && p.series > 0) {
    const float w = (float)(1 << p.series) / lam, b = 0.25f * lam * expf(lam) * (w * w) * (w * w);
    for (float x = b; x > 1.f && p.guard < 40; x *= 0.5f) ++p.guard;
  }
  if (p.guard < fx_kappa_base(p.series)) p.guard = fx_kappa_base(p.series);
  if (p.guard < 1) p.guard = 1;
  float t = 1.f;
  int n = 1;
  for (; n < GF_FX_CH_TERMS - 5; ++n) {
    t *= lam / (float)n;
    if (t < 2.2e-19f) break;
  }
  p.terms = DERIV ? n + 4 : n;
  return p;
}

// Real (im = 0) or imaginary (1) parts of f_j, kappa taken `down` bits down,
// and of df_j/dc1 (b1) and df_j/dc0 (b2) when DERIV. Only the c0 derivatives
// are summed: with C_n the q^2 coefficient of q^n, dC_n/dc0 = dC_(n-1)/dc1, so
// b1_0 = c0 b2_2, b1_1 = b2_0 + c1 b2_2 and b1_2 = b2_1, term by term.
template <bool DERIV>
GF_HD void fx_ch(const i64* kappa, int down, int terms, int im, i64 c0, i64 c1, i64 f[3], i64 b1[3], i64 b2[3]) {
  const fx_num n0 = fx_pre(c0), n1 = fx_pre(c1);
  i64 a = 0, b = 0, c = 0;
  i64 a0 = 0, b0 = 0, g0 = 0;
#pragma unroll 1
  for (int n = terms; n >= 0; --n) {
    const fx_num pc = fx_pre(c);
    i64 k = ((n & 1) == im) ? kappa[n] >> down : 0;
    if (n & 2) k = -k;
    const i64 na = fx_mul(pc, n0) + k, nb = a + fx_mul(pc, n1);
    if (DERIV) {
      const fx_num p0 = fx_pre(g0);
      const i64 na0 = c + fx_mul(p0, n0), nb0 = a0 + fx_mul(p0, n1);
      g0 = b0;
      a0 = na0;
      b0 = nb0;
    }
    c = b;
    a = na;
    b = nb;
  }
  f[0] = a;
  f[1] = b;
  f[2] = c;
  if (DERIV) {
    const fx_num g = fx_pre(g0);
    b2[0] = a0;
    b2[1] = b0;
    b2[2] = g0;
    b1[0] = fx_mul(g, n0);
    b1[1] = a0 + fx_mul(g, n1);
    b1[2] = b0;
  }
}

// ---------------------------------------------------------------------------
// fp64 <-> fixed
// ---------------------------------------------------------------------------
GF_HD u64 fx_bits(double d) {
#ifdef __CUDA_ARCH__
  return (u64)__double_as_longlong(d);
#else
  u64 u;
  memcpy(&u, &d, 8);
  return u;
#endif
}
GF_HD double fx_from_bits(u64 u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((i64)u);
#else
  double d;
  memcpy(&d, &u, 8);
  return d;
#endif
}
GF_HD float fx_float_bits(unsigned int u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f;
  memcpy(&f, &u, 4);
  return f;
#endif
}

GF_HD int fx_exponent_field(double d) { return (int)((fx_bits(d) >> 52) & 0x7FF); }
// d / 2^(emax - 1083 + up), rounded; emax at least d's exponent field, so that
// |result| < 2^(61 - up)
GF_HD i64 fx_mantissa(double d, int emax, int up) {
  const u64 b = fx_bits(d);
  int e = (int)((b >> 52) & 0x7FF);
  i64 v = (i64)(b & 0xFFFFFFFFFFFFFull);
  if (e) v |= 1ll << 52;
  else e = 1;
  const int s = 8 - up - (emax - e);
  if (s >= 0) v <<= s;
  else v = s > -55 ? (v + (1ll << (-s - 1))) >> -s : 0;
  return (b >> 63) ? -v : v;
}
// d / 2^(emax - 1023) in fp32 from the leading bits (0 below 2^-126)
GF_HD float fx_leading(double d, int emax) {
  const u64 b = fx_bits(d);
  const int e = (int)((b >> 52) & 0x7FF), ef = e - emax + 127;
  const unsigned int man = (unsigned int)(b >> 29) & 0x7FFFFFu, sg = (unsigned int)(b >> 32) & 0x80000000u;
  return (e == 0 || ef <= 0) ? 0.f : fx_float_bits(sg | ((unsigned int)ef << 23) | man);
}

// Exponent emax - 1023 + up of a matrix: the smallest for which a bound on the
// spectral norm, max_i sum_j |(M^dag M)_ij| in fp32 from the leading bits, is
// at most 1 (1 + 2^-10). It is 1 for a unitary matrix. False for a matrix that
// is not finite.
// small: entries below 2^-7 of that unit.
GF_HD bool fx_exponent_of(const double* m /* 18, row-major, re im */, int& emax, int& up, int& small) {
  emax = 1;
  up = small = 0;
#pragma unroll
  for (int i = 0; i < 18; ++i) {
    const int e = fx_exponent_field(m[i]);
    emax = e > emax ? e : emax;
  }
  if (emax == 0x7FF) return false;
  float f[18];
#pragma unroll
  for (int i = 0; i < 18; ++i) f[i] = fx_leading(m[i], emax);
  float bound = 0.f;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      float re = 0.f, im = 0.f;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float xr = f[2 * (3 * k + i)], xi = f[2 * (3 * k + i) + 1];
        const float yr = f[2 * (3 * k + j)], yi = f[2 * (3 * k + j) + 1];
        re = fmaf(xr, yr, fmaf(xi, yi, re));
        im = fmaf(xr, yi, fmaf(-xi, yr, im));
      }
      s += fabsf(re) + fabsf(im);
    }
    bound = fmaxf(bound, s);
  }
  // bound < 3 * 72 < 4^4
  up = (bound > 1.0009765625f) + (bound > 4.00390625f) + (bound > 16.015625f) + (bound > 64.0625f);
  const float tiny = 0.0078125f * (float)(1 << up);
  small = 0;
#pragma unroll
  for (int i = 0; i < 18; ++i) small += fabsf(f[i]) < tiny;
  return true;
}
GF_HD bool fx_has_f64(int e) { return e >= GF_FX_F64_SUM; }

// One exponent per matrix gives every entry the same absolute error, 2^-61 of
// the norm. That is below fp64's rounding of the matrix, but an entry below
// 2^-7 of the norm had more digits of its own in fp64. Where the small entries
// are a pattern that products keep, results live off those digits: links near
// the identity (weak fields; 15 small entries), near the diagonal (12), real
// ones (9), SU(2) subgroups (8), rows or columns of another size (6). A matrix
// with such a pattern is "graded": its slot keeps fp64, and what it enters is
// computed in fp64. Exact zeros lose nothing, so entries below 2^-7 must
// include one that is not zero. A Haar-random link is graded with probability
// 8 10^-8 (8 of 10^8 drawn; an entry close to the unit circle makes the rest of
// its row and column small): one in three 32^4 configurations.
// small: bit i for entry i below 2^-7 2^(unit - 1023); returns whether they form
// a pattern (zeros included).
GF_HD bool fx_small_pattern(unsigned small) {
  unsigned n = small - ((small >> 1) & 0x55555555u);
  n = (n & 0x33333333u) + ((n >> 2) & 0x33333333u);
  n = (n + (n >> 4)) & 0x0F0F0F0Fu;
  n = (n + (n >> 8) + (n >> 16)) & 0xFFu;
  bool line = false;
#pragma unroll
  for (int k = 0; k < 3; ++k)
    line = line || (small & (0x3Fu << (6 * k))) == (0x3Fu << (6 * k)) ||
           (small & (0x30C3u << (2 * k))) == (0x30C3u << (2 * k));
  return n >= 8 || line;
}
GF_HD bool fx_is_small(double d, int unit) {
  return ((int)(fx_bits(d) >> 32) & 0x7FFFFFFF) < (int)((unsigned)(unit - 7) << 20);
}
GF_HD bool fx_small_nonzero(double d, int unit) { return fx_is_small(d, unit) && (fx_bits(d) << 1) != 0; }
#define GF_FX_PATTERN_MIN 6  // the fewest small entries of a pattern
GF_HD bool fx_graded(const double* m, int unit) {
  unsigned small = 0;
  bool any = false;
#pragma unroll
  for (int i = 0; i < 18; ++i) {
    small |= (unsigned)fx_is_small(m[i], unit) << i;
    any = any || fx_small_nonzero(m[i], unit);
  }
  return any && fx_small_pattern(small);
}
// an entry of a slot that holds fp64
GF_HD int4 fx_pack64(double re, double im) {
  const u64 a = fx_bits(re), b = fx_bits(im);
  return make_int4((int)(unsigned)a, (int)(unsigned)(a >> 32), (int)(unsigned)b, (int)(unsigned)(b >> 32));
}
GF_HD double fx_unpack64(int lo, int hi) { return fx_from_bits(((u64)(unsigned)hi << 32) | (unsigned)lo); }

// One matrix to fixed point; returns its exponent. few: it has small entries
// enough to be graded.
GF_HD int fx_from_f64(const double* m, int4 out[9], bool& few) {
  int emax, up, small;
  few = false;
  if (!fx_exponent_of(m, emax, up, small)) {
#pragma unroll
    for (int i = 0; i < 9; ++i) out[i] = make_int4(0, 0, 0, 0);
    return GF_FX_BAD;
  }
  few = small >= GF_FX_PATTERN_MIN;
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    fx_split<0>(fx_mantissa(m[2 * i], emax, up), out[i].x, out[i].y);
    fx_split<0>(fx_mantissa(m[2 * i + 1], emax, up), out[i].z, out[i].w);
  }
  return emax - 1023 + up;
}
GF_HD int fx_from_f64(const double* m, int4 out[9]) {
  bool few;
  return fx_from_f64(m, out, few);
}

// One matrix to what its slot holds: fixed point, or fp64 if it is graded.
GF_HD int fx_encode(const double* m, int4 out[9]) {
  bool few;
  int e = fx_from_f64(m, out, few);
  if (few && fx_graded(m, e + 1023)) {
    e = GF_FX_F64;
#pragma unroll
    for (int i = 0; i < 9; ++i) out[i] = fx_pack64(m[2 * i], m[2 * i + 1]);
  }
  return e;
}

// real and imaginary parts of the f_j, side by side: f at [2 j + im]
GF_HD void fx_ch_both(const i64* kappa, int down, int terms, i64 c0, i64 c1, i64 f[6]) {
  const fx_num n0 = fx_pre(c0), n1 = fx_pre(c1);
  i64 a[2] = {0, 0}, b[2] = {0, 0}, c[2] = {0, 0};
#pragma unroll 1
  for (int n = terms; n >= 0; --n) {
    i64 k = kappa[n] >> down;
    if (n & 2) k = -k;
#pragma unroll
    for (int im = 0; im < 2; ++im) {
      const fx_num pc = fx_pre(c[im]);
      const i64 na = fx_mul(pc, n0) + ((n & 1) == im ? k : 0), nb = a[im] + fx_mul(pc, n1);
      c[im] = b[im];
      a[im] = na;
      b[im] = nb;
    }
  }
#pragma unroll
  for (int im = 0; im < 2; ++im) {
    f[im] = a[im];
    f[2 + im] = b[im];
    f[4 + im] = c[im];
  }
}

// R 2^(E - 60) as fp64, rounded once to nearest (ties up in magnitude; at most
// half an ulp), by integer operations, for E above GF_FX_NORMAL, where no result
// but zero is below the normal range. Overflow gives an infinity, GF_FX_BAD a NaN.
#define GF_FX_NORMAL (-960)
GF_HD int fx_leading_zeros(u64 a) {
#ifdef __CUDA_ARCH__
  return __clzll((i64)a);
#else
  return __builtin_clzll(a);
#endif
}
GF_HD double fx_to_normal(i64 R, int E) {
  const u64 sign = R < 0 ? 1ull << 63 : 0ull;
  u64 a = R < 0 ? (u64)(-R) : (u64)R;
  if (E > GF_FX_BAD / 2) return fx_from_bits(0x7FF8000000000000ull);
  if (a == 0) return 0.0;
  const int lz = fx_leading_zeros(a);
  a <<= lz;
  const u64 man = (a >> 11) + ((a >> 10) & 1);  // 2^52 <= man <= 2^53
  const int ex = 1023 + 3 - lz + E;              // value = (a / 2^63) 2^(63 - lz + E - 60)
  if (ex >= 0x7FF) return fx_from_bits(sign | 0x7FF0000000000000ull);
  return fx_from_bits(sign | (((u64)(ex - 1) << 52) + man));
}
// the same for any E
GF_HD double fx_to_f64(i64 R, int E) {
  const u64 a = R < 0 ? (u64)(-R) : (u64)R;
  if (E <= GF_FX_NORMAL && a != 0) {
    const int lz = fx_leading_zeros(a), d = 12 - (1023 + 3 - lz + E);
    if (d >= 12) {  // below the normal range: in units of 2^-1074
      const u64 n = d > 64 ? 0 : (d < 64 ? (a << lz) >> d : 0) + (((a << lz) >> (d - 1)) & 1);
      return fx_from_bits((R < 0 ? 1ull << 63 : 0ull) | n);
    }
  }
  return fx_to_normal(R, E);
}

}  // namespace gf
