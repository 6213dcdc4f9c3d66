// Block fixed-point arithmetic on the integer pipes, for fp64-class 3x3 work.
//
// GB300 issues one fp64 multiply-add per 64 fp32 ones, but a 32 x 32 + 64 bit
// integer multiply-add (IMAD.WIDE) per four (measured: 3.95 cycles per warp
// and scheduler). A product of two 60-bit fixed-point numbers kept as limbs of
// 30 bits needs three of them (high x high and the two cross terms), so a
// real multiply-add costs 12 issue slots instead of 64, with an absolute
// error of about 2^-59 of the operands' norms, below the 2^-53 of fp64.
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
// row r of the conjugate: the imaginary part negated limb by limb
GF_HD void fx_conj(fx_row& r) {
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    r.bh[j] = -r.bh[j];
    r.bl[j] = -r.bl[j];
  }
}

// a b + c as one IMAD.WIDE. The product is written in PTX: knowing that a limb
// is not negative, the compiler widens it as unsigned, finds no 32 x 32 form
// for the mixed signs and emits a full 64-bit product (400 instructions for
// a row product instead of 136). mad.wide in PTX becomes two instructions.
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
GF_HD void fx_add(fx_acc& acc, int& ea, fx_acc v, int ev) {
  if (ev != ea) {
    const int d = ev > ea ? ev - ea : ea - ev;
    const int s = d < 63 ? d : 63;
    fx_acc& small = ev > ea ? acc : v;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      small.re[j] >>= s;
      small.im[j] >>= s;
    }
    if (ev > ea) ea = ev;
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    acc.re[j] += v.re[j];
    acc.im[j] += v.im[j];
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

// One matrix to fixed point; returns its exponent. A bound on the squared
// spectral norm, max_i sum_j |(M^dag M)_ij|, is formed in fp32 from the
// leading bits; it is 1 for a unitary matrix.
GF_HD int fx_from_f64(const double* m /* 18, row-major, re im */, int4 out[9]) {
  int emax = 1;
#pragma unroll
  for (int i = 0; i < 18; ++i) {
    const int e = (int)((fx_bits(m[i]) >> 52) & 0x7FF);
    emax = e > emax ? e : emax;
  }
  if (emax == 0x7FF) {
#pragma unroll
    for (int i = 0; i < 9; ++i) out[i] = make_int4(0, 0, 0, 0);
    return GF_FX_BAD;
  }
  // leading bits relative to 2^emax: |f| < 2, entries below 2^-126 of it as 0
  float f[18];
#pragma unroll
  for (int i = 0; i < 18; ++i) {
    const u64 b = fx_bits(m[i]);
    const int e = (int)((b >> 52) & 0x7FF);
    const int ef = e - emax + 127;
    const unsigned int man = (unsigned int)(b >> 29) & 0x7FFFFFu;
    const unsigned int sg = (unsigned int)(b >> 32) & 0x80000000u;
    f[i] = (e == 0 || ef <= 0) ? 0.f : fx_float_bits(sg | ((unsigned int)ef << 23) | man);
  }
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
  // smallest E2 with bound <= 4^E2 (1 + 2^-10); bound < 3 * 72 < 4^4
  const int E2 = (bound > 1.0009765625f) + (bound > 4.00390625f) + (bound > 16.015625f) + (bound > 64.0625f);
  i64 R[18];
#pragma unroll
  for (int i = 0; i < 18; ++i) {
    const u64 b = fx_bits(m[i]);
    int e = (int)((b >> 52) & 0x7FF);
    i64 v = (i64)(b & 0xFFFFFFFFFFFFFull);
    if (e) v |= 1ll << 52;
    else e = 1;
    // value = v 2^(e - 1075) = R 2^(emax - 1023 + E2 - 60)
    const int s = 8 - E2 - (emax - e);
    if (s >= 0) v <<= s;
    else v = s > -55 ? (v + (1ll << (-s - 1))) >> -s : 0;
    R[i] = (b >> 63) ? -v : v;
  }
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    fx_split<0>(R[2 * i], out[i].x, out[i].y);
    fx_split<0>(R[2 * i + 1], out[i].z, out[i].w);
  }
  return emax - 1023 + E2;
}

// R 2^(E - 60) as fp64, rounded once to nearest (ties up in magnitude; at
// most half an ulp), by integer operations. Overflow gives an infinity, a
// result below the normal range a zero, GF_FX_BAD a NaN.
GF_HD double fx_to_f64(i64 R, int E) {
  const u64 sign = R < 0 ? 1ull << 63 : 0ull;
  u64 a = R < 0 ? (u64)(-R) : (u64)R;
  if (E > GF_FX_BAD / 2) return fx_from_bits(0x7FF8000000000000ull);
  if (a == 0) return 0.0;
#ifdef __CUDA_ARCH__
  const int lz = __clzll((i64)a);
#else
  const int lz = __builtin_clzll(a);
#endif
  a <<= lz;
  const u64 man = (a >> 11) + ((a >> 10) & 1);  // 2^52 <= man <= 2^53
  const int ex = 1023 + 3 - lz + E;              // value = (a / 2^63) 2^(63 - lz + E - 60)
  if (ex <= 0) return fx_from_bits(sign);
  if (ex >= 0x7FF) return fx_from_bits(sign | 0x7FF0000000000000ull);
  return fx_from_bits(sign | (((u64)(ex - 1) << 52) + man));
}

}  // namespace gf
