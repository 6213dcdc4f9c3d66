// Device side of the fixed-point kernels: field storage, the block shape
// shared by all of them and staple chains by rows.
//
// A fixed-point link or matrix field is tiled by 32 sites: per direction and
// tile, int4 [9][32] (re.h, re.l, im.h, im.l; or two doubles, for a matrix kept
// in fp64) and the exponents int [32]. The
// elements of a matrix are then at constant distances (one address per
// matrix, immediate offsets for its nine loads) and coalesced over sites.
//
// Blocks are 96 threads = 32 links of one direction x 3 rows, thread
// t = 3 link + row: the rows of a link sit in the same warp or the next one,
// so a matrix element that all three read is one transaction.
//
// A kernel runs its fixed-point arithmetic on whatever the slots hold and sums
// the exponents beside it; a sum that shows an fp64 matrix (fx_has_f64) means that
// the link's result is formed anew in fp64 (fxrows64.cuh) before it is stored.
#pragma once
#include "fixed.cuh"

namespace gf {

#ifndef GF_FX_MINB
#define GF_FX_MINB 7
#endif
// Up to so many sites the blocks of a stencil fit on the GPU at five per SM, and
// the kernels take the registers that leaves: 8^4 trajectory 684 us, with seven
// 721; at 24^4, where the GPU is full, the force takes 711 us with seven and 753
// with six.
#define GF_FX_FEW_MAX 6144
#define GF_FX_FEW_MINB 5
#define GF_FX_LINKS 32
#define GF_FX_TILE (9 * 512 + 128)
#define GF_FX_THREADS (3 * GF_FX_LINKS)

// storage of a field, in bytes: 4 directions of ceil(V / 32) tiles
inline size_t fx_field_bytes(size_t V) { return 4 * ((V + 31) / 32) * (size_t)GF_FX_TILE; }

struct FxField {
  const char* p;
};
__device__ __forceinline__ size_t fx_offset(int mu, int s, int V) {
  return (size_t)(unsigned)(mu * ((V + 31) >> 5) + (s >> 5)) * GF_FX_TILE + (unsigned)(s & 31) * 16u;
}
// one matrix of a field
struct FxMat {
  const char* p;
  __device__ __forceinline__ int4 operator()(int el) const {
    return __ldg(reinterpret_cast<const int4*>(p + el * 512));
  }
};
__device__ __forceinline__ FxMat fx_mat(const FxField& F, int mu, int s, int V) {
  return FxMat{F.p + fx_offset(mu, s, V)};
}
__device__ __forceinline__ int fx_exp(const FxField& F, int mu, int s, int V) {
  return __ldg(reinterpret_cast<const int*>(F.p + (size_t)(unsigned)(mu * ((V + 31) >> 5) + (s >> 5)) * GF_FX_TILE +
                                            9 * 512 + (unsigned)(s & 31) * 4u));
}

// row r of a field matrix or of its dagger (column r, conjugated)
template <bool DAG>
__device__ __forceinline__ fx_row fx_load_row(const FxMat& M, int r) {
  fx_row a;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int4 v = M(DAG ? 3 * k + r : 3 * r + k);
    a.ah[k] = v.x;
    a.al[k] = v.y;
    a.bh[k] = DAG ? -v.z : v.z;
    a.bl[k] = DAG ? -v.w : v.w;
  }
  return a;
}

// writes element el of a field's matrix, and the matrix's exponent
__device__ __forceinline__ void fx_store(char* p, size_t off, int el, i64 re, i64 im) {
  int4 v;
  fx_split<0>(re, v.x, v.y);
  fx_split<0>(im, v.z, v.w);
  *reinterpret_cast<int4*>(p + off + el * 512) = v;
}
__device__ __forceinline__ void fx_store_exp(char* p, size_t off, int s, int e) {
  *reinterpret_cast<int*>(p + off + 9 * 512 - 12 * (s & 31)) = e > GF_FX_BAD / 2 ? GF_FX_BAD : e;
}
__device__ __forceinline__ void fx_store_row(char* p, size_t off, int r, const fx_acc& v) {
#pragma unroll
  for (int j = 0; j < 3; ++j) fx_store(p, off, 3 * r + j, v.re[j], v.im[j]);
}

// ---------------------------------------------------------------------------
// exchange between the rows of a link through shared memory, component-major
// over the block's links, so that a thread per link reads without conflicts
// ---------------------------------------------------------------------------
struct FxRaw {  // 64-bit matrix
  i64 v[18][GF_FX_LINKS];
};
struct FxOperand {  // matrix as limbs, a right factor
  int4 v[9][GF_FX_LINKS];
};
struct FxShMat {
  const FxOperand* m;
  int link;
  __device__ __forceinline__ int4 operator()(int el) const { return m->v[el][link]; }
};
__device__ __forceinline__ void fx_share(FxRaw& sh, int link, int r, const fx_acc& m) {
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    sh.v[2 * (3 * r + j)][link] = m.re[j];
    sh.v[2 * (3 * r + j) + 1][link] = m.im[j];
  }
}
template <int K>
__device__ __forceinline__ void fx_share(FxOperand& sh, int link, int r, const fx_acc& m) {
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    int4 v;
    fx_split<K>(m.re[j], v.x, v.y);
    fx_split<K>(m.im[j], v.z, v.w);
    sh.v[3 * r + j][link] = v;
  }
}
template <bool DAG>
__device__ __forceinline__ fx_row fx_load_row(const FxShMat& M, int r) {
  fx_row a;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int4 v = M(DAG ? 3 * k + r : 3 * r + k);
    a.ah[k] = v.x;
    a.al[k] = v.y;
    a.bh[k] = DAG ? -v.z : v.z;
    a.bl[k] = DAG ? -v.w : v.w;
  }
  return a;
}

// fp64 value of R (unit 1): the two words through exponent constants, no
// integer-to-double conversion
__device__ __forceinline__ double fx_value(i64 R) {
  const int h = (int)(R >> 32);
  const double dh = __hiloint2double(0x43300000, h ^ (int)0x80000000) - 4503601774854144.0;  // 2^52 + 2^31
  const double dl = __hiloint2double(0x43300000, (int)(unsigned)R) - 4503599627370496.0;      // 2^52
  return fma(dh, 4294967296.0, dl);
}
// c 2^(E - 60); NaN for GF_FX_BAD
__device__ __forceinline__ double fx_unit(double c, int E) {
  if (E > GF_FX_BAD / 2) return __longlong_as_double(0x7FF8000000000000ll);
  const int k = E - 60;
  if (k > -1000 && k < 1000) return c * __hiloint2double((k + 1023) << 20, 0);
  return scalbn(c, k);
}

// P <- keep P + coef c(M), c the su(3) coefficients of TA(M) for the 32
// matrices M of a block (raw, exponents se); thread t serves link t % 32 and,
// by t / 32, the coefficients (0, 1, 2), (3, 4, 7) or (5, 6).
// Links whose products hold an fp64 matrix are left out (fx64_update_mom).
__device__ __forceinline__ void fx_update_mom(const FxRaw& sh, const int* se, double* __restrict__ P, int mu, int s0,
                                              int V, double coef, double keep) {
  const int link = threadIdx.x & 31, part = threadIdx.x >> 5, s = s0 + link;
  if (s >= V || fx_has_f64(se[link])) return;
  const int i = part == 2 ? 1 : 0, j = part == 0 ? 1 : 2;
  const int ij = 2 * (3 * i + j), ji = 2 * (3 * j + i);
  const i64 d1 = sh.v[1][link], d2 = sh.v[9][link], d3 = sh.v[17][link];
  const i64 c[3] = {sh.v[ij + 1][link] + sh.v[ji + 1][link], sh.v[ij][link] - sh.v[ji][link],
                    part == 0 ? d1 - d2 : d1 + d2 - 2 * d3};
  const int a0 = part == 0 ? 0 : (part == 1 ? 3 : 5);
  const int a[3] = {a0, a0 + 1, part == 0 ? 2 : 7};
  const double sc = fx_unit(coef, se[link]);
  double* p = P + (size_t)mu * 8 * V + s;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    if (q == 2 && part == 2) break;
    const double f = (q == 2 && part == 1) ? sc * 0.57735026918962576451 : sc;
    double* d = p + (size_t)a[q] * V;
    const double old = keep != 0.0 ? keep * *d : 0.0;
    *d = fma(f, fx_value(c[q]), old);
  }
}

// lexicographic offset of a unit step from a site (periodic), along mu
__device__ __forceinline__ int fx_up(const Geom& g, const Site& st, int mu) {
  const int str = g.stride[mu];
  return coord(st, mu) == g.L[mu] - 1 ? str - g.L[mu] * str : str;
}
__device__ __forceinline__ int fx_down(const Geom& g, const Site& st, int mu) {
  const int str = g.stride[mu];
  return coord(st, mu) == 0 ? g.L[mu] * str - str : -str;
}

// acc += row r of the two staples of U_mu(x) in the mu-nu plane, in the
// orientation of construct_double_staple! (V = S^dag):
//   U_nu(x) U_mu(x+nu) U_nu(x+mu)^dag + U_nu(x-nu)^dag U_mu(x-nu) U_nu(x-nu+mu)
__device__ __forceinline__ void fx_add_staples(fx_acc& acc, int& ea, const FxField& U, const Geom& g, const Site& st,
                                               int s, int mu, int nu, int mu_up, int r) {
  const int V = g.vol;
  const int xpm = eo_of_lex(g, st.lex + mu_up, st.par ^ 1);
  {
    const int xpn = eo_of_lex(g, st.lex + fx_up(g, st, nu), st.par ^ 1);
    const int e = fx_exp(U, nu, s, V) + fx_exp(U, mu, xpn, V) + fx_exp(U, nu, xpm, V);
    const fx_row a = fx_load_row<false>(fx_mat(U, nu, s, V), r);
    const fx_acc t = fx_row_mul<false>(a, fx_mat(U, mu, xpn, V));
    fx_add(acc, ea, fx_row_mul<true>(fx_operand<0>(t), fx_mat(U, nu, xpm, V)), e);
  }
  {
    const int dn = fx_down(g, st, nu);
    const int xmn = eo_of_lex(g, st.lex + dn, st.par ^ 1);
    const int xpm_mn = eo_of_lex(g, st.lex + mu_up + dn, st.par);
    const int e = fx_exp(U, nu, xmn, V) + fx_exp(U, mu, xmn, V) + fx_exp(U, nu, xpm_mn, V);
    const fx_row a = fx_load_row<true>(fx_mat(U, nu, xmn, V), r);
    const fx_acc t = fx_row_mul<false>(a, fx_mat(U, mu, xmn, V));
    fx_add(acc, ea, fx_row_mul<false>(fx_operand<0>(t), fx_mat(U, nu, xpm_mn, V)), e);
  }
}

// Small lattices do not fill the GPU with three threads per link, and a call
// takes as long as one thread's chain of products. The stencil kernels then
// run three times as many, one group of 96 per axis nu != mu (thread t: axis
// t / 96), and sum the groups' rows through shared memory. 20-step Wilson
// trajectories and two-level stout forces, one group against three: 4^4 629
// and 105 us against 506 and 88, 6^4 653 and 120 against 570 and 112, 8^4 718
// and 158 against 759 and 175 (the GPU is full, and the exchange costs).
#ifndef GF_FX_SPLIT_MAX
#define GF_FX_SPLIT_MAX 2048
#endif
template <int AXES>
struct FxAxes {  // rows of the axes 1 .. AXES - 1
  FxRaw v[AXES > 1 ? AXES - 1 : 1];
  int e[AXES > 1 ? AXES - 1 : 1][GF_FX_LINKS];
};
template <>
struct FxAxes<1> {};
// acc of the other axes added to the first one's; every thread of the block
// calls it, those of axis 0 return the sum
template <int AXES>
__device__ __forceinline__ void fx_sum_axes(FxAxes<AXES>& sh, int axis, int link, int r, fx_acc& acc, int& ea) {
  if constexpr (AXES > 1) {
    if (axis > 0) {
      fx_share(sh.v[axis - 1], link, r, acc);
      if (r == 0) sh.e[axis - 1][link] = ea;
    }
    __syncthreads();
    if (axis == 0) {
#pragma unroll
      for (int a = 0; a < AXES - 1; ++a) {
        fx_acc o;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          o.re[j] = sh.v[a].v[2 * (3 * r + j)][link];
          o.im[j] = sh.v[a].v[2 * (3 * r + j) + 1][link];
        }
        fx_add(acc, ea, o, sh.e[a][link]);
      }
    }
  }
}
// rows of V = S^dag of a field at s: the staple sum, |V| <= 6 2^ea (axis 0's
// threads when AXES = 3)
template <int AXES>
__device__ __forceinline__ fx_acc fx_staple_row(FxAxes<AXES>& sh, const FxField& U, const Geom& g, const Site& st,
                                                int s, int mu, int axis, int link, int r, int& ea) {
  fx_acc acc = {{0, 0, 0}, {0, 0, 0}};
  ea = -GF_FX_BAD;
  const int mu_up = fx_up(g, st, mu);
  if (AXES > 1) {
    fx_add_staples(acc, ea, U, g, st, s, mu, (mu + 1 + axis) & 3, mu_up, r);
  } else {
#pragma unroll 1
    for (int k = 1; k < 4; ++k) fx_add_staples(acc, ea, U, g, st, s, mu, (mu + k) & 3, mu_up, r);
  }
  fx_sum_axes<AXES>(sh, axis, link, r, acc, ea);
  return acc;
}

// ---------------------------------------------------------------------------
// exp(iX) of the block's links
// ---------------------------------------------------------------------------
static __constant__ fx_kappa c_fx_kappa = fx_make_kappa();

struct FxExp {      // exp(iX) of the block's links
  FxRaw m;          // in: the matrix whose TA gives q
  FxOperand q;      // X / 2^scale as operand
  i64 f[6][GF_FX_LINKS];   // f_j at [2 j + im], units 2^(guard - 60)
  int e[GF_FX_LINKS];      // in: exponent of m
  int s[GF_FX_LINKS];      // scale
  int g[GF_FX_LINKS];      // guard
  int sq[GF_FX_LINKS];     // squarings
  int most;                // most squarings of a link of the block
};

// Plan of exp(iX), X = q 2^(e - 60) Hermitian and traceless; q becomes
// X / 2^pow2 in units of 2^-60. q = 0 for a non-finite X.
template <bool DERIV>
__device__ __forceinline__ fx_plan fx_exp_plan(fx_herm& q, int e) {
  // |X|^2 <= (2/3) tr X^2 for a traceless Hermitian X
  float n2 = 0.f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float u = (float)(int)(q.d[k] >> 32), v = (float)(int)(q.re[k] >> 32), w = (float)(int)(q.im[k] >> 32);
    n2 = fmaf(u, u, fmaf(2.f * v, v, fmaf(2.f * w, w, n2)));
  }
  const bool bad = e > GF_FX_BAD / 2;
  const int ee = e < -90 ? -90 : (e > 90 ? 90 : e);
  const float lam = bad ? 0.f : sqrtf(0.66667f * n2) * 1.00001f * exp2f((float)(ee - 28));
  const fx_plan plan = fx_series<DERIV>(lam);
  const int d = plan.pow2 - e;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    q.d[k] = bad ? 0 : fx_shift(q.d[k], d);
    q.re[k] = bad ? 0 : fx_shift(q.re[k], d);
    q.im[k] = bad ? 0 : fx_shift(q.im[k], d);
  }
  q.d[2] = -q.d[0] - q.d[1];
  return plan;
}
// element (i, j) of q as an operand
__device__ __forceinline__ int4 fx_herm_element(const fx_herm& q, int i, int j) {
  if (i == j) {
    const fx_num x = fx_pre(q.d[i]);
    return make_int4(x.h, x.l, 0, 0);
  }
  const int k = i + j - 1;
  const fx_num u = fx_pre(q.re[k]), v = fx_pre(q.im[k]);
  return i < j ? make_int4(u.h, u.l, v.h, v.l) : make_int4(u.h, u.l, -v.h, -v.l);
}

// Plan, operand and coefficients of exp(iX) for a block's links; thread per
// link, im = 0 or 1. b: derivatives, df_j/dc1 at [2 j + im] and df_j/dc0 at
// [6 + 2 j + im]. True if X is beyond the derivatives' series.
template <bool DERIV>
__device__ __forceinline__ bool fx_exp_coefficients(FxExp& sh, i64 (*b)[GF_FX_LINKS], int link, int im, fx_herm q,
                                                    int e) {
  const fx_plan plan = fx_exp_plan<DERIV>(q, e);
  i64 c0, c1, f[3], b1[3], b2[3];
  fx_invariants(q, c0, c1);
  const int terms = __reduce_max_sync(0xffffffffu, plan.terms);
  fx_ch<DERIV>(c_fx_kappa.k[plan.series], plan.guard - fx_kappa_base(plan.series), terms, im, c0, c1, f, b1, b2);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    sh.f[2 * j + im][link] = f[j];
    if (DERIV) {
      b[2 * j + im][link] = b1[j];
      b[6 + 2 * j + im][link] = b2[j];
    }
  }
  if (im == 0) {
#pragma unroll
    for (int el = 0; el < 9; ++el) sh.q.v[el][link] = fx_herm_element(q, el / 3, el % 3);
    sh.s[link] = plan.pow2;
    sh.g[link] = plan.guard;
    sh.sq[link] = plan.squares;
    const int most = __reduce_max_sync(0xffffffffu, plan.squares);
    if (link == 0) sh.most = most;
  }
  return plan.beyond;
}
// X = -i TA(rho m) of the block's matrices m as entries and exponent
__device__ __forceinline__ fx_herm fx_ta_herm(const FxExp& sh, int link, const fx_scalar rho, const fx_scalar rho3,
                                              int& e) {
  e = sh.e[link] + rho.e + 1;  // of the entries below
  fx_herm q;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int i = k == 2 ? 1 : 0, j = k == 0 ? 1 : 2, ij = 2 * (3 * i + j), ji = 2 * (3 * j + i);
    const i64 xr = sh.m.v[ij][link] - sh.m.v[ji][link], xi = sh.m.v[ij + 1][link] + sh.m.v[ji + 1][link];
    q.re[k] = fx_mul(fx_pre(xi >> 2), fx_num_of(rho));
    q.im[k] = -fx_mul(fx_pre(xr >> 2), fx_num_of(rho));
  }
  const i64 d0 = sh.m.v[1][link], d1 = sh.m.v[9][link], d2 = sh.m.v[17][link];
  q.d[0] = fx_mul(fx_pre((2 * d0 - d1 - d2) >> 1), fx_num_of(rho3));
  q.d[1] = fx_mul(fx_pre((2 * d1 - d0 - d2) >> 1), fx_num_of(rho3));
  q.d[2] = -q.d[0] - q.d[1];
  return q;
}

// row r of exp(iX), exponent 0: f0 + (f1 + f2 q) q; qrow is row r of q, f the
// coefficients (re, im) in units of 2^(g - 60)
template <class MAT>
__device__ __forceinline__ fx_acc fx_exp_row(const i64 f[6], int g, const fx_row& qrow, const MAT& q, int r) {
  const fx_num f2r = fx_pre(f[4]), f2i = fx_pre(f[5]);
  fx_acc G;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    fx_sum re = fx_zero_sum(), im = fx_zero_sum();
    fx_cmac(re, im, f2r, f2i, fx_num{qrow.ah[j], qrow.al[j]}, fx_num{qrow.bh[j], qrow.bl[j]});
    G.re[j] = fx_get(re) + (j == r ? f[2] : 0);
    G.im[j] = fx_get(im) + (j == r ? f[3] : 0);
  }
  fx_acc E = fx_row_mul<false>(fx_operand<1>(G), q);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    E.re[j] = (E.re[j] + (j == r ? f[0] >> 1 : 0)) << (g + 1);
    E.im[j] = (E.im[j] + (j == r ? f[1] >> 1 : 0)) << (g + 1);
  }
  return E;
}
__device__ __forceinline__ fx_acc fx_exp_row(const FxExp& sh, int link, int r) {
  i64 f[6];
#pragma unroll
  for (int j = 0; j < 6; ++j) f[j] = sh.f[j][link];
  const FxShMat q{&sh.q, link};
  return fx_exp_row(f, sh.g[link], fx_load_row<false>(q, r), q, r);
}

// the same after the squarings that |X| > 2 takes; every thread of the block
// calls it. sh.m is overwritten by those.
__device__ __forceinline__ fx_acc fx_exp_row_squared(FxExp& sh, int link, int r) {
  fx_acc E = fx_exp_row(sh, link, r);
  const int most = sh.most, mine = sh.sq[link];
  FxOperand& em = reinterpret_cast<FxOperand&>(sh.m);
#pragma unroll 1
  for (int k = 0; k < most; ++k) {
    fx_share<0>(em, link, r, E);
    __syncthreads();
    if (k < mine) E = fx_row_mul<false>(fx_operand<0>(E), FxShMat{&em, link});
    __syncthreads();
  }
  return E;
}

// (R / 2^20)^2 in fp32
__device__ __forceinline__ float fx_square(i64 R) {
  const float v = fmaf((float)(int)(R >> 32), 4096.f, (float)(unsigned)R * 9.5367431640625e-7f);
  return v * v;
}
__device__ __forceinline__ float fx_square(const fx_acc& v) {
  float n = 0.f;
#pragma unroll
  for (int j = 0; j < 3; ++j) n += fx_square(v.re[j]) + fx_square(v.im[j]);
  return n;
}
// shift d for which a matrix of raw norm^2 n (units of fx_square) has
// norm <= 2^60 after R >> d, and > 2^58 (0 for a zero or non-finite matrix)
__device__ __forceinline__ int fx_norm_shift(float n, int e) {
  if (n == 0.f || e > GF_FX_BAD / 2) return 0;
  // n (1 + 2^-10) < 2^k4, norm < 2^(20 + k4 / 2)
  const int k4 = (int)(__float_as_uint(n * 1.0009765625f) >> 23) - 126;
  return ((k4 + 1) >> 1) - 40;
}

// an element of a slot as fp64. Out of line where it is not fp64 already: by
// integer operations, for the fp64 pipe is what its callers wait for, and inlined
// nine times a matrix they took registers from the fixed-point kernels around
// (24^4 force 736 us, out of line 715).
static __device__ __noinline__ double2 fx_convert64(int4 v, int e) {
  return make_double2(fx_to_f64(fx_join(v.x, v.y), e), fx_to_f64(fx_join(v.z, v.w), e));
}
__device__ __forceinline__ double2 fx_element64(int4 v, int e) {
  if (e == GF_FX_F64) return make_double2(fx_unpack64(v.x, v.y), fx_unpack64(v.z, v.w));
  return fx_convert64(v, e);
}
// fp64 view of a fixed-point field: element by element, and whole matrices (fp64
// kernels)
struct FxMat64 {
  FxMat m;
  int e;
  __device__ __forceinline__ double2 operator()(int el) const { return fx_element64(m(el), e); }
};
__device__ __forceinline__ FxMat64 fx_mat64(const FxField& F, int mu, int s, int V) {
  return FxMat64{fx_mat(F, mu, s, V), fx_exp(F, mu, s, V)};
}
struct LinkSrcFx64 {
  FxField F;
  __device__ __forceinline__ mat3<double> operator()(int mu, int s, int V) const {
    mat3<double> m;
    const FxMat64 M = fx_mat64(F, mu, s, V);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const double2 v = M(k);
      m.e[k / 3][k % 3] = mk(v.x, v.y);
    }
    return m;
  }
};
__device__ __forceinline__ double2 fx_complex64(double2 v) { return v; }
__device__ __forceinline__ double2 fx_complex64(float4 v) {
  return make_double2(df_to_double(dfl(v.x, v.y)), df_to_double(dfl(v.z, v.w)));
}
// The slot of a matrix that was stored in fixed point at exponent e, if it proves
// to be graded: its fp64 entries, from the field `m` that holds it. Out of line,
// for the few matrices with enough small entries: link update with the copy at
// 16^4 80.9 us with the test of the pattern in line, 78.4 so, 71.7 without.
template <typename E>
static __device__ __noinline__ void fx_regrade(const E* m, char* fx, int mu, int s, int V, int e) {
  const E* b = m + (size_t)mu * 9 * V + s;
  double d[18];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const double2 v = fx_complex64(b[(size_t)k * V]);
    d[2 * k] = v.x;
    d[2 * k + 1] = v.y;
  }
  if (!fx_graded(d, e + 1023)) return;
  char* o = fx + fx_offset(mu, s, V);
#pragma unroll
  for (int k = 0; k < 9; ++k) *reinterpret_cast<int4*>(o + 512 * k) = fx_pack64(d[2 * k], d[2 * k + 1]);
  *reinterpret_cast<int*>(o + 9 * 512 - 12 * (s & 31)) = GF_FX_F64;
}
// one matrix into a field, in the form that it takes (fx_encode)
__device__ __forceinline__ void fx_store64(char* p, int mu, int s, int V, const double* m) {
  int4 f[9];
  const int e = fx_encode(m, f);
  char* o = p + fx_offset(mu, s, V);
#pragma unroll
  for (int k = 0; k < 9; ++k) *reinterpret_cast<int4*>(o + 512 * k) = f[k];
  *reinterpret_cast<int*>(o + 9 * 512 - 12 * (s & 31)) = e;
}

}  // namespace gf
