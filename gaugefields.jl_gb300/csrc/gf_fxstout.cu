// Stout forward and adjoint (the formulas of gf_stout.cu) in block fixed point
// by rows: fp64-class results at integer-pipe rates. A block serves 32 links;
// thread 3 link + row carries a row of each matrix through the products, and
// two warps evaluate the Cayley-Hamilton series with a thread per link (real
// and imaginary parts), exchanging through shared memory. The kernels
// are bound by integer multiply-add issue. A two-level smearing with its
// adjoint at 16^4: 9.65 ms in fp64 arithmetic, 1.69 ms here (1.4 ms of it in
// these kernels), at no larger an error (gradient 4.3e-16 against 4.8e-16 of
// the largest entry).
#include "gf_internal.h"
#include "fxrows64.cuh"
#include <cstddef>

namespace gf {

// a raw row from an operand row of a field
__device__ __forceinline__ fx_acc fx_raw_row(const fx_row& a) {
  fx_acc v;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    v.re[j] = fx_join(a.ah[j], a.al[j]);
    v.im[j] = fx_join(a.bh[j], a.bl[j]);
  }
  return v;
}
template <int K>
__device__ __forceinline__ void fx_down_row(fx_acc& v) {
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    v.re[j] >>= K;
    v.im[j] >>= K;
  }
}

// Ubar = exp(TA(C U^dag)) U, C = rho V stored when Cout is given
// Blocks per SM, by 32^4 launches: gather 5.20 ms with four (168 registers),
// 5.12 with five, 5.82 with six (spills); local adjoint 3.74 with four, 3.71
// with five, 3.96 with six; forward 2.84 with seven, 2.93 with eight, 3.1 with
// five or six.
#ifndef GF_FX_GATHER_MINB
#define GF_FX_GATHER_MINB 5
#endif
#ifndef GF_FX_LOCAL_MINB
#define GF_FX_LOCAL_MINB 5
#endif
#ifndef GF_FX_FWD_MINB
#define GF_FX_FWD_MINB 7
#endif
// row r of f0 + f1 q + f2 q^2 in fp64
__device__ __forceinline__ row64 exp_row64(const double (*f)[GF_FX_LINKS], int link, int r, const row64& q,
                                           const row64& q2) {
  row64 e = zero64();
  cadd64(e, f[4][link], f[5][link], q2);
  cadd64(e, f[2][link], f[3][link], q);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    e.re[j] += j == r ? f[0][link] : 0.0;
    e.im[j] += j == r ? f[1][link] : 0.0;
  }
  return e;
}
__device__ __forceinline__ void share_herm64(const Sh64& sh, const mat3<double>& q) {
#pragma unroll
  for (int k = 0; k < 9; ++k) sh.v[k][sh.link] = make_double2(q.e[k / 3][k % 3].re, q.e[k / 3][k % 3].im);
}

// The level in fp64 for the block's links whose staples hold an fp64 slot (by
// x.e); the first 96 threads work.
__device__ __noinline__ void fwd_rows64(const FxField U, char* Uout, char* Cout, const Geom& g, double rho, int mu,
                                        int s0, FxExp& x) {
  const int t = threadIdx.x, link = t / 3, r = t - 3 * link, V = g.vol;
  const bool mine = t < GF_FX_THREADS && fx_has_f64(x.e[link]);
  const int s = min(s0 + link, V - 1);
  double(*f)[GF_FX_LINKS] = reinterpret_cast<double(*)[GF_FX_LINKS]>(x.f);
  row64 v = zero64(), E = zero64();
  __syncthreads();  // x has been read
  if (mine) {
    v = staple_row64(U, g, site_of(g, s), s, mu, r);
    share64(sh64(x.m, link), r, mul64<true>(v, fx_mat64(U, mu, s, V)));
  }
  __syncthreads();
  if (t < GF_FX_LINKS) {
    int halvings = 0;
    if (fx_has_f64(x.e[t])) {
      const mat3<double> q = ta_herm64(sh64(x.m, t), rho, halvings);
      double c0, c1;
      herm_invariants(q, c0, c1);
      ch_coef<double> cc;
      ch_coefficients<double, false>(c0, c1, cc);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        f[2 * j][t] = cc.f[j].re;
        f[2 * j + 1][t] = cc.f[j].im;
      }
      share_herm64(sh64(x.q, t), q);
    }
    x.sq[t] = halvings;
    const int most = __reduce_max_sync(0xffffffffu, halvings);
    if (t == 0) x.most = most;
  }
  __syncthreads();
  if (mine) {
    const row64 q = load_row64<false>(sh64(x.q, link), r);
    E = exp_row64(f, link, r, q, mul64<false>(q, sh64(x.q, link)));
  }
  const int most = x.most;
#pragma unroll 1
  for (int k = 0; k < most; ++k) {
    if (mine) share64(sh64(x.m, link), r, E);
    __syncthreads();
    if (mine && k < x.sq[link]) E = mul64<false>(E, sh64(x.m, link));
    __syncthreads();
  }
  __syncthreads();
  if (mine) {
    share64(sh64(x.m, link), r, mul64<false>(E, fx_mat64(U, mu, s, V)));
    E = zero64();
    add64(E, v, rho);
    share64(sh64(x.q, link), r, E);
  }
  __syncthreads();
  if (t < 2 * GF_FX_LINKS && s0 + (t & 31) < V && fx_has_f64(x.e[t & 31])) {
    if (t < GF_FX_LINKS) store_field64(sh64(x.m, t), Uout, mu, s0 + t, V);
    else if (Cout) store_field64(sh64(x.q, t & 31), Cout, mu, s0 + (t & 31), V);
  }
}

template <int AXES, int MINB>
__global__ void __launch_bounds__(GF_FX_THREADS * AXES, MINB)
    k_stout_fwd_fx(FxField U, char* __restrict__ Uout, char* __restrict__ Cout, const __grid_constant__ Geom g,
                   fx_scalar rho, fx_scalar rho3, double rho64) {
  __shared__ FxExp sh;
  __shared__ FxAxes<AXES> ax;
  const int axis = AXES > 1 ? threadIdx.x / GF_FX_THREADS : 0, t = threadIdx.x - axis * GF_FX_THREADS;
  const int mu = blockIdx.x & 3, V = g.vol;
  const int link = t / 3, r = t - 3 * link;
  const int sx = (blockIdx.x >> 2) * GF_FX_LINKS + link, s = min(sx, V - 1);
  const size_t off = fx_offset(mu, s, V);
  bool f64 = false;
  {
    const Site st = site_of(g, s);
    int ev;
    fx_acc v = fx_staple_row<AXES>(ax, U, g, st, s, mu, axis, link, r, ev);
    if (axis == 0) {
      const fx_row vr = fx_operand<3>(v);
      fx_share(sh.m, link, r, fx_row_mul<true>(vr, fx_mat(U, mu, s, V)));
      const int e = ev + 3 + fx_exp(U, mu, s, V);
      f64 = fx_has_f64(e);
      if (r == 0) sh.e[link] = e;
      if (Cout && sx < V && !f64) {
        fx_down_row<3>(v);
        fx_scale_row(v, rho);
        fx_store_row(Cout, off, r, v);
        if (r == 0) fx_store_exp(Cout, off, s, ev + 3 + rho.e);
      }
    }
  }
  const bool any64 = __syncthreads_or(f64);
  if (threadIdx.x < 64) {
    int e;
    const fx_herm q = fx_ta_herm(sh, t & 31, rho, rho3, e);
    fx_exp_coefficients<false>(sh, nullptr, t & 31, t >> 5, q, e);
  }
  __syncthreads();
  const int E0 = sh.s[link] > GF_FX_MAX_POW2 ? GF_FX_BAD : sh.e[link];
  if (AXES > 1 && axis > 0) {
    // the other axes' threads only keep step with the squarings' barriers
    for (int k = 0; k < 2 * sh.most; ++k) __syncthreads();
  } else {
    const fx_acc E = fx_exp_row_squared(sh, link, r);
    const fx_acc W = fx_row_mul<false>(fx_operand<0>(E), fx_mat(U, mu, s, V));
    if (sx < V && !f64) {
      fx_store_row(Uout, off, r, W);
      if (r == 0) fx_store_exp(Uout, off, s, E0 + rho.e > GF_FX_BAD / 2 ? GF_FX_BAD : fx_exp(U, mu, s, V));
    }
  }
  if (any64) fwd_rows64(U, Uout, Cout, g, rho64, mu, (blockIdx.x >> 2) * GF_FX_LINKS, sh);
}

// D = halfbeta S of the smeared links: dS/dUbar of the Wilson action, the top
// level's input. The local adjoint can form it itself (TOP), and does where a
// launch counts; on larger lattices its products are faster in a kernel of
// their own, at the force's 70% of the multiply pipe instead of 61% beside 70
// KB of other code. Two-level force, inside against apart: 8^4 159 / 166 us,
// 12^4 537 / 540, 16^4 1547 / 1529, 32^4 23.9 / 23.5 ms.
#ifndef GF_FX_DSDU_MIN
#define GF_FX_DSDU_MIN 40000
#endif
__device__ __noinline__ void dsdu_rows64(const FxField U, char* D, const Geom& g, double halfbeta, int mu, int s0,
                                         FxRaw& m, const int* se) {
  const int t = threadIdx.x, link = t / 3, r = t - 3 * link, V = g.vol, s = min(s0 + link, V - 1);
  if (fx_has_f64(se[link])) {
    row64 v = zero64();
    add64(v, staple_row64(U, g, site_of(g, s), s, mu, r), halfbeta);
    share64(sh64(m, link), r, v);
  }
  __syncthreads();
  if (t < GF_FX_LINKS && s0 + t < V && fx_has_f64(se[t])) store_field64(sh64(m, t), D, mu, s0 + t, V, true);
}
__global__ void __launch_bounds__(GF_FX_THREADS, GF_FX_FWD_MINB)
    k_dsdu_fx(FxField U, char* __restrict__ D, const __grid_constant__ Geom g, fx_scalar halfbeta, double halfbeta64) {
  __shared__ float n[3][GF_FX_LINKS];
  __shared__ FxRaw m;
  __shared__ int se[GF_FX_LINKS];
  FxAxes<1> none;
  const int t = threadIdx.x, mu = blockIdx.x & 3, V = g.vol;
  const int link = t / 3, r = t - 3 * link;
  const int sx = (blockIdx.x >> 2) * GF_FX_LINKS + link, s = min(sx, V - 1);
  int e;
  fx_acc v = fx_staple_row<1>(none, U, g, site_of(g, s), s, mu, 0, link, r, e);
  fx_down_row<3>(v);
  fx_scale_row(v, halfbeta);
  e += 3 + halfbeta.e;
  n[r][link] = fx_square(v);
  if (r == 0) se[link] = e;
  const bool f64 = fx_has_f64(e), any64 = __syncthreads_or(f64);
  if (sx < V && !f64) {
    // V = S^dag: stored as its dagger
    const int k = fx_norm_shift(n[0][link] + n[1][link] + n[2][link], e);
    const size_t off = fx_offset(mu, s, V);
#pragma unroll
    for (int j = 0; j < 3; ++j) fx_store(D, off, 3 * j + r, fx_shift(v.re[j], k), -fx_shift(v.im[j], k));
    if (r == 0) fx_store_exp(D, off, s, e + k);
  }
  if (any64) dsdu_rows64(U, D, g, halfbeta64, mu, (blockIdx.x >> 2) * GF_FX_LINKS, m, se);
}

// The local adjoint. F1 = Dbar, or (TOP) the smeared links, whose staples give
// Dbar = halfbeta S; C = Cst, or rebuilt from U.
struct FxLocal {
  FxExp x;                     // x.m: C U^dag, then the trace partials, then Gamma
  FxOperand lam;               // Lambda, then Y
  FxOperand em;                // e^Q
  i64 b[12][GF_FX_LINKS];      // derivatives of the f_j, then trB_k at [2 k + im]
  int ey[GF_FX_LINKS];
  int f64[GF_FX_LINKS];        // the link is formed in fp64: a slot among its operands, or a large X
  FxOperand db;                // TOP: halfbeta V of the smeared links
  FxOperand cm;                // recompute: C
};
static size_t fx_local_bytes(bool top, bool recompute) {
  return offsetof(FxLocal, db) + (recompute ? 2 : (top ? 1 : 0)) * sizeof(FxOperand);
}

// The same in fp64 for the block's links that f64 marks; exp(Q) from Q halved to
// |Q| <= 1, so that it serves any Q.
template <bool TOP, bool RECOMPUTE>
__device__ __noinline__ void local_rows64(const FxField U, const FxField F1, const FxField Cst, char* Zout, char* Dpout,
                                          const Geom& g, double rho, double halfbeta, int mu, int s0, FxLocal& sh) {
  const int t = threadIdx.x, link = t / 3, r = t - 3 * link, V = g.vol, s = min(s0 + link, V - 1);
  const bool mine = sh.f64[link];
  double(*f)[GF_FX_LINKS] = reinterpret_cast<double(*)[GF_FX_LINKS]>(sh.x.f);
  double(*b)[GF_FX_LINKS] = reinterpret_cast<double(*)[GF_FX_LINKS]>(sh.b);
  double(*tr)[GF_FX_LINKS] = reinterpret_cast<double(*)[GF_FX_LINKS]>(sh.x.m.v);
  const Sh64 M = sh64(sh.x.m, link), Q = sh64(sh.x.q, link), L = sh64(sh.lam, link), E = sh64(sh.em, link);
  __syncthreads();  // sh has been read
  // C U^dag
  if (mine) {
    row64 c;
    if (RECOMPUTE) {
      c = zero64();
      add64(c, staple_row64(U, g, site_of(g, s), s, mu, r), rho);
      share64(sh64(sh.cm, link), r, c);
    } else {
      c = load_row64<false>(fx_mat64(Cst, mu, s, V), r);
    }
    share64(M, r, mul64<true>(c, fx_mat64(U, mu, s, V)));
    if (TOP) {
      row64 v = zero64();
      add64(v, staple_row64(F1, g, site_of(g, s), s, mu, r), halfbeta);
      share64(sh64(sh.db, link), r, v);
    }
  }
  __syncthreads();
  // Lambda = U Dbar; the exponential of Q and its derivatives
  row64 lam = zero64();
  if (mine) {
    const row64 u = load_row64<false>(fx_mat64(U, mu, s, V), r);
    lam = TOP ? mul64<true>(u, sh64(sh.db, link)) : mul64<false>(u, fx_mat64(F1, mu, s, V));
    share64(L, r, lam);
  }
  if (t < GF_FX_LINKS) {
    int halvings = 0;
    if (sh.f64[t]) {
      const mat3<double> q = ta_herm64(sh64(sh.x.m, t), 1.0, halvings);
      double c0, c1;
      herm_invariants(q, c0, c1);
      ch_coef<double> cc;
      ch_coefficients<double, true>(c0, c1, cc);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        f[2 * j][t] = cc.f[j].re;
        f[2 * j + 1][t] = cc.f[j].im;
        b[2 * j][t] = cc.b1[j].re;
        b[2 * j + 1][t] = cc.b1[j].im;
        b[6 + 2 * j][t] = cc.b2[j].re;
        b[7 + 2 * j][t] = cc.b2[j].im;
      }
      share_herm64(sh64(sh.x.q, t), q);
    }
    sh.x.sq[t] = halvings;
    const int most = __reduce_max_sync(0xffffffffu, halvings);
    if (t == 0) sh.x.most = most;
  }
  __syncthreads();
  row64 q = zero64(), q2 = zero64(), w = zero64(), e = zero64();
  if (mine) {
    q = load_row64<false>(Q, r);
    q2 = mul64<false>(q, Q);
    e = exp_row64(f, link, r, q, q2);
    share64(E, r, e);
  }
  // e^Q = F^n, n = 2^s, F = exp(Q / n): tr(Lambda de^Q) = tr(Lambda' dF) with
  // Lambda' = sum_k F^k Lambda F^(n - 1 - k), which doubles its terms by
  // Lambda' <- F Lambda' + Lambda' F, F <- F F
  const int most = sh.x.most, halvings = sh.x.sq[link];
#pragma unroll 1
  for (int k = 0; k < most; ++k) {
    const bool now = mine && k < halvings;
    __syncthreads();
    if (now) {
      row64 l = mul64<false>(e, L);
      add64(l, mul64<false>(lam, E));
      lam = l;
      e = mul64<false>(e, E);
    }
    __syncthreads();
    if (now) {
      share64(L, r, lam);
      share64(E, r, e);
    }
  }
  __syncthreads();
  // Lambda Q, Q Lambda; the traces' parts (Lambda and Q the halved ones)
  if (mine) {
    w = mul64<false>(lam, Q);
    double re = 0.0, im = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double2 v = Q(3 * k + r);
      re = fma(w.re[k], v.x, fma(-w.im[k], v.y, re));
      im = fma(w.re[k], v.y, fma(w.im[k], v.x, im));
    }
    tr[6 * r][link] = pick64(lam.re[0], lam.re[1], lam.re[2], r);
    tr[6 * r + 1][link] = pick64(lam.im[0], lam.im[1], lam.im[2], r);
    tr[6 * r + 2][link] = pick64(w.re[0], w.re[1], w.re[2], r);
    tr[6 * r + 3][link] = pick64(w.im[0], w.im[1], w.im[2], r);
    tr[6 * r + 4][link] = re;
    tr[6 * r + 5][link] = im;
    add64(w, mul64<false>(q, L));
  }
  __syncthreads();
  // trB_k = sum_j b_k[j] tr(Lambda Q^j)
  if (t < 2 * GF_FX_LINKS && sh.f64[t & 31]) {
    const int l = t & 31, k = t >> 5;
    double re = 0.0, im = 0.0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double x = tr[2 * j][l] + tr[6 + 2 * j][l] + tr[12 + 2 * j][l];
      const double y = tr[2 * j + 1][l] + tr[7 + 2 * j][l] + tr[13 + 2 * j][l];
      const double br = b[6 * k + 2 * j][l], bi = b[6 * k + 2 * j + 1][l];
      re = fma(br, x, fma(-bi, y, re));
      im = fma(br, y, fma(bi, x, im));
    }
    b[6 * k][l] = re;
    b[6 * k + 1][l] = im;
  }
  __syncthreads();
  // Gamma, of the whole Q
  if (mine) {
    row64 G = zero64(), h = zero64();
    cadd64(G, f[4][link], f[5][link], w);
    cadd64(G, f[2][link], f[3][link], lam);
    cadd64(G, b[0][link], b[1][link], q);
    cadd64(G, b[6][link], b[7][link], q2);
    add64(h, G, scalbn(1.0, -halvings));
    share64(M, r, h);
  }
  __syncthreads();
  // Y = TA(-i Gamma)
  if (mine) {
    row64 y;
    const double tr3 = (M(0).x + M(4).x + M(8).x) * (1.0 / 3.0);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double2 a = M(3 * r + j), c = M(3 * j + r);
      y.re[j] = j == r ? 0.0 : 0.5 * (a.y - c.y);
      y.im[j] = j == r ? tr3 - a.x : -0.5 * (a.x + c.x);
    }
    share64(L, r, y);
  }
  __syncthreads();
  // Z = U^dag Y, Dp = Dbar e^Q + C^dag Y^dag
  if (mine) {
    share64(M, r, mul64<false>(load_row64<true>(fx_mat64(U, mu, s, V), r), L));
    row64 d = TOP ? load_row64<true>(sh64(sh.db, link), r) : load_row64<false>(fx_mat64(F1, mu, s, V), r);
    d = mul64<false>(d, E);
    const row64 c = RECOMPUTE ? load_row64<true>(sh64(sh.cm, link), r) : load_row64<true>(fx_mat64(Cst, mu, s, V), r);
    add64(d, mul64<true>(c, L));
    share64(Q, r, d);
  }
  __syncthreads();
  if (t < 2 * GF_FX_LINKS && s0 + (t & 31) < V && sh.f64[t & 31]) {
    if (t < GF_FX_LINKS) store_field64(sh64(sh.x.m, t), Zout, mu, s0 + t, V);
    else store_field64(sh64(sh.x.q, t & 31), Dpout, mu, s0 + (t & 31), V);
  }
}

template <bool TOP, bool RECOMPUTE>
__global__ void __launch_bounds__(GF_FX_THREADS, GF_FX_LOCAL_MINB)
    k_bwd_local_fx(FxField U, FxField F1, FxField Cst, char* __restrict__ Zout, char* __restrict__ Dpout,
                   const __grid_constant__ Geom g, fx_scalar rho, fx_scalar one, fx_scalar one3, fx_scalar halfbeta,
                   double rho64, double halfbeta64) {
  extern __shared__ __align__(16) char smem[];
  FxLocal& sh = *reinterpret_cast<FxLocal*>(smem);
  const int t = threadIdx.x, mu = blockIdx.x & 3, V = g.vol;
  const int link = t / 3, r = t - 3 * link;
  const int sx = (blockIdx.x >> 2) * GF_FX_LINKS + link, s = min(sx, V - 1);
  const size_t off = fx_offset(mu, s, V);
  const Site st = site_of(g, s);
  const int eu = fx_exp(U, mu, s, V);
  int ec, ed;
  // C U^dag
  if (RECOMPUTE) {
    FxAxes<1> none;
    fx_acc c = fx_staple_row<1>(none, U, g, st, s, mu, 0, link, r, ec);
    fx_down_row<3>(c);
    fx_scale_row(c, rho);
    ec += 3 + rho.e;
    fx_share<0>(sh.cm, link, r, c);
    fx_share(sh.x.m, link, r, fx_row_mul<true>(fx_operand<0>(c), fx_mat(U, mu, s, V)));
  } else {
    ec = fx_exp(Cst, mu, s, V);
    fx_share(sh.x.m, link, r, fx_row_mul<true>(fx_load_row<false>(fx_mat(Cst, mu, s, V), r), fx_mat(U, mu, s, V)));
  }
  if (r == 0) sh.x.e[link] = ec + eu;
  if (TOP) {
    FxAxes<1> none;
    fx_acc v = fx_staple_row<1>(none, F1, g, st, s, mu, 0, link, r, ed);
    fx_down_row<3>(v);
    fx_scale_row(v, halfbeta);
    ed += 3 + halfbeta.e;
    fx_share<0>(sh.db, link, r, v);
  } else {
    ed = fx_exp(F1, mu, s, V);
  }
  const bool slot64 = fx_has_f64(ec + eu) || fx_has_f64(ed);
  if (r == 0) sh.f64[link] = slot64;
  __syncthreads();
  // Lambda = U Dbar; the exponential of Q and its derivatives
  fx_acc lam;
  {
    const fx_row u = fx_load_row<false>(fx_mat(U, mu, s, V), r);
    if (TOP) lam = fx_row_mul<true>(u, FxShMat{&sh.db, link});
    else lam = fx_row_mul<false>(u, fx_mat(F1, mu, s, V));
    fx_share<0>(sh.lam, link, r, lam);
  }
  const int el = eu + ed;
  bool beyond = false;
  if (t < 64) {
    int e;
    const fx_herm q = fx_ta_herm(sh.x, t & 31, one, one3, e);
    beyond = fx_exp_coefficients<true>(sh.x, sh.b, t & 31, t >> 5, q, e);
    if (beyond) sh.f64[t & 31] = 1;
  }
  const bool any64 = __syncthreads_or(beyond || slot64);
  // Lambda Q, Q Lambda, Q^2, e^Q by rows; partial traces
  fx_acc W, X, Q2;
  const fx_row qr = fx_load_row<false>(FxShMat{&sh.x.q, link}, r);
  W = fx_row_mul<false>(fx_operand<0>(lam), FxShMat{&sh.x.q, link});
  X = fx_row_mul<false>(qr, FxShMat{&sh.lam, link});
  Q2 = fx_row_mul<false>(qr, FxShMat{&sh.x.q, link});
  {
    // row r of e^Q = f0 + f1 q + f2 q^2, q^2 being at hand
    const int g = sh.x.g[link];
    const fx_num f1r = fx_pre(sh.x.f[2][link]), f1i = fx_pre(sh.x.f[3][link]);
    const fx_num f2r = fx_pre(sh.x.f[4][link]), f2i = fx_pre(sh.x.f[5][link]);
    fx_acc E;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      fx_sum re = fx_zero_sum(), im = fx_zero_sum();
      fx_cmac(re, im, f1r, f1i, fx_num{qr.ah[j], qr.al[j]}, fx_num{qr.bh[j], qr.bl[j]});
      fx_cmac(re, im, f2r, f2i, fx_pre(Q2.re[j]), fx_pre(Q2.im[j]));
      E.re[j] = (fx_get(re) + (j == r ? sh.x.f[0][link] : 0)) << g;
      E.im[j] = (fx_get(im) + (j == r ? sh.x.f[1][link] : 0)) << g;
    }
    fx_share<0>(sh.em, link, r, E);
  }
  {
    fx_sum re = fx_zero_sum(), im = fx_zero_sum();
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int4 v = sh.x.q.v[3 * k + r][link];
      fx_cmac(re, im, fx_pre(W.re[k]), fx_pre(W.im[k]), fx_num{v.x, v.y}, fx_num{v.z, v.w});
    }
    i64(*tr)[GF_FX_LINKS] = sh.x.m.v + 6 * r;
    tr[0][link] = r == 0 ? lam.re[0] : (r == 1 ? lam.re[1] : lam.re[2]);
    tr[1][link] = r == 0 ? lam.im[0] : (r == 1 ? lam.im[1] : lam.im[2]);
    tr[2][link] = r == 0 ? W.re[0] : (r == 1 ? W.re[1] : W.re[2]);
    tr[3][link] = r == 0 ? W.im[0] : (r == 1 ? W.im[1] : W.im[2]);
    tr[4][link] = fx_get(re);
    tr[5][link] = fx_get(im);
  }
  __syncthreads();
  // trB_k = sum_j b_k[j] tr(Lambda Q^j), traces two bits down
  if (t < 64) {
    const int l = t & 31, k = t >> 5;
    fx_sum re = fx_zero_sum(), im = fx_zero_sum();
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      i64 T[2];
#pragma unroll
      for (int c = 0; c < 2; ++c)
        T[c] = (sh.x.m.v[2 * j + c][l] + sh.x.m.v[6 + 2 * j + c][l] + sh.x.m.v[12 + 2 * j + c][l]) >> 2;
      fx_cmac(re, im, fx_pre(sh.b[6 * k + 2 * j][l]), fx_pre(sh.b[6 * k + 2 * j + 1][l]), fx_pre(T[0]), fx_pre(T[1]));
    }
    __syncwarp();
    sh.b[6 * k][l] = fx_get(re);
    sh.b[6 * k + 1][l] = fx_get(im);
  }
  __syncthreads();
  // Gamma, in units of 2^(el + guard - scale). As a derivative of a unitary
  // exponential it is no larger than 2^scale Lambda; its parts wrap harmlessly.
  const int eg = el + sh.x.g[link] - sh.x.s[link] + (sh.x.e[link] > GF_FX_BAD / 2 ? GF_FX_BAD : 0);
  {
    const fx_num b1r = fx_pre(sh.b[0][link]), b1i = fx_pre(sh.b[1][link]);
    const fx_num b2r = fx_pre(sh.b[6][link]), b2i = fx_pre(sh.b[7][link]);
    const fx_num f1r = fx_pre(sh.x.f[2][link]), f1i = fx_pre(sh.x.f[3][link]);
    const fx_num f2r = fx_pre(sh.x.f[4][link]), f2i = fx_pre(sh.x.f[5][link]);
    fx_acc G;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      fx_sum re = fx_zero_sum(), im = fx_zero_sum();
      fx_cmac(re, im, b1r, b1i, fx_num{qr.ah[j], qr.al[j]}, fx_num{qr.bh[j], qr.bl[j]});
      fx_cmac(re, im, b2r, b2i, fx_pre(Q2.re[j]), fx_pre(Q2.im[j]));
      G.re[j] = fx_get(re) << 2;
      G.im[j] = fx_get(im) << 2;
      re = im = fx_zero_sum();
      fx_cmac(re, im, f2r, f2i, fx_pre((X.re[j] + W.re[j]) >> 1), fx_pre((X.im[j] + W.im[j]) >> 1));
      G.re[j] += fx_get(re) << 1;
      G.im[j] += fx_get(im) << 1;
      re = im = fx_zero_sum();
      fx_cmac(re, im, f1r, f1i, fx_pre(lam.re[j]), fx_pre(lam.im[j]));
      G.re[j] += fx_get(re);
      G.im[j] += fx_get(im);
    }
    fx_share(sh.x.m, link, r, G);
    if (r == 0) sh.ey[link] = eg;
  }
  __syncthreads();
  // Y = TA(-i Gamma), normalised; row p of link l
  {
    const int l = t & 31, p = t >> 5;
    // entries of Y (raw): off-diagonal (0,1), (0,2), (1,2) and the imaginary diagonal
    i64 yr[3], yi[3], yd[3];
    float n2 = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int i = k == 2 ? 1 : 0, j = k == 0 ? 1 : 2, ij = 2 * (3 * i + j), ji = 2 * (3 * j + i);
      yr[k] = (sh.x.m.v[ij + 1][l] - sh.x.m.v[ji + 1][l]) >> 1;
      yi[k] = -(sh.x.m.v[ij][l] + sh.x.m.v[ji][l]) >> 1;
      const i64 y = (sh.x.m.v[8 * (k == 0)][l] >> 2) + (sh.x.m.v[16 - 8 * (k == 2)][l] >> 2) -
                    (sh.x.m.v[8 * k][l] >> 1);
      yd[k] = fx_mul(fx_pre(y), fx_pre(0x555555555555555ll)) << 2;  // 2^60 / 3
      n2 += 2.f * (fx_square(yr[k]) + fx_square(yi[k])) + fx_square(yd[k]);
    }
    // |Y|^2 <= (2/3) tr Y^dag Y for a traceless anti-Hermitian Y
    const int e = sh.ey[l], d = fx_norm_shift(0.66667f * n2, e);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int k = p + j - 1;  // off-diagonal index of (p, j), p != j
      const i64 sr = k == 0 ? yr[0] : (k == 1 ? yr[1] : yr[2]), si = k == 0 ? yi[0] : (k == 1 ? yi[1] : yi[2]);
      const i64 sd = p == 0 ? yd[0] : (p == 1 ? yd[1] : yd[2]);
      const i64 re = j == p ? 0 : fx_shift(j > p ? sr : -sr, d), im = fx_shift(j == p ? sd : si, d);
      int4 v;
      fx_split<0>(re, v.x, v.y);
      fx_split<0>(im, v.z, v.w);
      sh.lam.v[3 * p + j][l] = v;
    }
    __syncthreads();
    if (p == 0) sh.ey[l] = e + d;
  }
  __syncthreads();
  // Z = U^dag Y, Dp = Dbar e^Q + C^dag Y^dag
  const FxShMat Y{&sh.lam, link};
  const int ey = sh.ey[link];
  const fx_acc z = fx_row_mul<false>(fx_load_row<true>(fx_mat(U, mu, s, V), r), Y);
  fx_acc dp;
  if (TOP) dp = fx_row_mul<false>(fx_load_row<true>(FxShMat{&sh.db, link}, r), FxShMat{&sh.em, link});
  else dp = fx_row_mul<false>(fx_load_row<false>(fx_mat(F1, mu, s, V), r), FxShMat{&sh.em, link});
  fx_row cr;
  if (RECOMPUTE) cr = fx_load_row<true>(FxShMat{&sh.cm, link}, r);
  else cr = fx_load_row<true>(fx_mat(Cst, mu, s, V), r);
  fx_add(dp, ed, fx_row_mul<true>(cr, Y), ec + ey);
  fx_down_row<1>(dp);
  if (sx < V && !sh.f64[link]) {
    fx_store_row(Zout, off, r, z);
    fx_store_row(Dpout, off, r, dp);
    if (r == 0) {
      fx_store_exp(Zout, off, s, eu + ey);
      fx_store_exp(Dpout, off, s, ed + 1);
    }
  }
  if (any64)
    local_rows64<TOP, RECOMPUTE>(U, F1, Cst, Zout, Dpout, g, rho64, halfbeta64, mu, (blockIdx.x >> 2) * GF_FX_LINKS,
                                 sh);
}

// The pull-back of Z through C: the terms (a)-(f) of gather_axis, grouped so
// that every product is a row times a matrix (ten per axis):
//   (a) U_K(x+nu) U_nu(x+K)^dag Z_K(x)
//   (c) + (f) [Z_K(x+nu)^dag U_nu(x+K)^dag + U_K(x+nu) Z_nu(x+K)] U_K(x)^dag
//   (b) U_K(x-K+nu)^dag U_nu(x-K)^dag Z_K(x-K)^dag
//   (d) + (e) [Z_K(x-K+nu) U_nu(x-K)^dag + U_K(x-K+nu)^dag Z_nu(x-K)] U_K(x-K)
// The two products with U_nu(x+-K)^dag stand side by side, so that its nine
// elements are in registers once and not across an axis (5.69 -> 5.12 ms).
// The last left factor is taken one bit down (the bracketed sums reach two
// units), and the six terms of an axis sum to at most three units.
__device__ __forceinline__ void fx_gather_axis(fx_acc& acc, int& ea, const FxField& U, const FxField& Z, const Geom& g,
                                               const Site& st, int s, int nu, int nu_up, int K, int r) {
  const int V = g.vol;
  const int xpn = eo_of_lex(g, st.lex + nu_up, st.par ^ 1);
  {
    const int xpk = eo_of_lex(g, st.lex + fx_up(g, st, K), st.par ^ 1);
    const int eun = fx_exp(U, nu, xpk, V), euk = fx_exp(U, K, xpn, V);
    const FxMat un = fx_mat(U, nu, xpk, V);
    const fx_row uk = fx_load_row<false>(fx_mat(U, K, xpn, V), r);
    fx_acc r1 = fx_row_mul<true>(uk, un);
    fx_acc t = fx_row_mul<true>(fx_load_row<true>(fx_mat(Z, K, xpn, V), r), un);
    int et = fx_exp(Z, K, xpn, V) + eun;
    fx_add(acc, ea, fx_row_mul<false>(fx_operand<1>(r1), fx_mat(Z, K, s, V)), euk + eun + fx_exp(Z, K, s, V) + 1);
    fx_add(t, et, fx_row_mul<false>(uk, fx_mat(Z, nu, xpk, V)), euk + fx_exp(Z, nu, xpk, V));
    fx_add(acc, ea, fx_row_mul<true>(fx_operand<1>(t), fx_mat(U, K, s, V)), et + fx_exp(U, K, s, V) + 1);
  }
  {
    const int dn = fx_down(g, st, K);
    const int xmk = eo_of_lex(g, st.lex + dn, st.par ^ 1);
    const int xmkn = eo_of_lex(g, st.lex + dn + nu_up, st.par);
    const int eun = fx_exp(U, nu, xmk, V), euk = fx_exp(U, K, xmkn, V);
    const FxMat un = fx_mat(U, nu, xmk, V);
    const fx_row uk = fx_load_row<true>(fx_mat(U, K, xmkn, V), r);
    fx_acc r1 = fx_row_mul<true>(uk, un);
    fx_acc t = fx_row_mul<true>(fx_load_row<false>(fx_mat(Z, K, xmkn, V), r), un);
    int et = fx_exp(Z, K, xmkn, V) + eun;
    fx_add(acc, ea, fx_row_mul<true>(fx_operand<1>(r1), fx_mat(Z, K, xmk, V)), euk + eun + fx_exp(Z, K, xmk, V) + 1);
    fx_add(t, et, fx_row_mul<false>(uk, fx_mat(Z, nu, xmk, V)), euk + fx_exp(Z, nu, xmk, V));
    fx_add(acc, ea, fx_row_mul<false>(fx_operand<1>(t), fx_mat(U, K, xmk, V)), et + fx_exp(U, K, xmk, V) + 1);
  }
}

__device__ __forceinline__ void gather_axis64(row64& acc, const FxField& U, const FxField& Z, const Geom& g,
                                              const Site& st, int s, int nu, int nu_up, int K, int r) {
  const int V = g.vol;
  const int xpn = eo_of_lex(g, st.lex + nu_up, st.par ^ 1);
  {
    const int xpk = eo_of_lex(g, st.lex + fx_up(g, st, K), st.par ^ 1);
    const FxMat64 un = fx_mat64(U, nu, xpk, V);
    const row64 uk = load_row64<false>(fx_mat64(U, K, xpn, V), r);
    add64(acc, mul64<false>(mul64<true>(uk, un), fx_mat64(Z, K, s, V)));
    row64 t = mul64<true>(load_row64<true>(fx_mat64(Z, K, xpn, V), r), un);
    add64(t, mul64<false>(uk, fx_mat64(Z, nu, xpk, V)));
    add64(acc, mul64<true>(t, fx_mat64(U, K, s, V)));
  }
  {
    const int dn = fx_down(g, st, K);
    const int xmk = eo_of_lex(g, st.lex + dn, st.par ^ 1);
    const int xmkn = eo_of_lex(g, st.lex + dn + nu_up, st.par);
    const FxMat64 un = fx_mat64(U, nu, xmk, V);
    const row64 uk = load_row64<true>(fx_mat64(U, K, xmkn, V), r);
    add64(acc, mul64<true>(mul64<true>(uk, un), fx_mat64(Z, K, xmk, V)));
    row64 t = mul64<true>(load_row64<false>(fx_mat64(Z, K, xmkn, V), r), un);
    add64(t, mul64<false>(uk, fx_mat64(Z, nu, xmk, V)));
    add64(acc, mul64<false>(t, fx_mat64(U, K, xmk, V)));
  }
}
// The gather in fp64 for the block's links that se marks; the first 96 threads.
template <int OUT>
__device__ __noinline__ void gather_rows64(const FxField U, const FxField Z, const FxField Dp, char* Dout, double* P,
                                           const Geom& g, double rho, double coef, int nu, int s0, FxRaw& m,
                                           const int* se) {
  const int t = threadIdx.x, link = t / 3, r = t - 3 * link, V = g.vol;
  const bool mine = t < GF_FX_THREADS && fx_has_f64(se[link]);
  const int s = min(s0 + link, V - 1);
  const Sh64 M = sh64(m, link);
  row64 d = zero64();
  if (mine) {
    const Site st = site_of(g, s);
    const int nu_up = fx_up(g, st, nu);
    row64 acc = zero64();
#pragma unroll 1
    for (int k = 1; k < 4; ++k) gather_axis64(acc, U, Z, g, st, s, nu, nu_up, (nu + k) & 3, r);
    d = load_row64<false>(fx_mat64(Dp, nu, s, V), r);
    add64(d, acc, rho);
  }
  if (OUT == 1) {
    if (mine && s0 + link < V) {
      double2* o = reinterpret_cast<double2*>(Dout) + (size_t)nu * 9 * V + s;
#pragma unroll
      for (int j = 0; j < 3; ++j) o[(size_t)(3 * r + j) * V] = make_double2(d.re[j], d.im[j]);
    }
    return;
  }
  __syncthreads();  // m has been read
  if (mine) share64(M, r, d);
  __syncthreads();
  if (OUT == 0) {
    if (t < GF_FX_LINKS && s0 + t < V && fx_has_f64(se[t])) store_field64(sh64(m, t), Dout, nu, s0 + t, V);
    return;
  }
  if (mine) d = mul64<false>(load_row64<false>(fx_mat64(U, nu, s, V), r), M);
  __syncthreads();
  if (mine) share64(M, r, d);
  __syncthreads();
  if (t < GF_FX_THREADS) update_mom64(sh64(m, t & 31), se, P, nu, s0, V, coef, 1.0);
}

// D = Dp + rho (pull-back). OUT 0: fixed-point Dout; 1: fp64 Dout (MAT64);
// 2: the thin-link momentum update P += coef c(U D) instead.
template <int OUT, int AXES>
__global__ void __launch_bounds__(GF_FX_THREADS * AXES, AXES > 1 ? 2 : GF_FX_GATHER_MINB)
    k_bwd_gather_fx(FxField U, FxField Z, FxField Dp, char* __restrict__ Dout, double* __restrict__ P,
                    const __grid_constant__ Geom g, fx_scalar rho, double rho64, double coef) {
  __shared__ union {
    FxOperand d;
    FxRaw m;
    float n[3][GF_FX_LINKS];
  } sh;
  __shared__ int se[GF_FX_LINKS];
  __shared__ FxAxes<AXES> ax;
  const int axis = AXES > 1 ? threadIdx.x / GF_FX_THREADS : 0, t = threadIdx.x - axis * GF_FX_THREADS;
  const int nu = blockIdx.x & 3, V = g.vol;
  const int link = t / 3, r = t - 3 * link, s0 = (blockIdx.x >> 2) * GF_FX_LINKS;
  const int sx = s0 + link, s = min(sx, V - 1);
  const Site st = site_of(g, s);
  const int nu_up = fx_up(g, st, nu);
  fx_acc d = {{0, 0, 0}, {0, 0, 0}};
  int ed = -GF_FX_BAD;
  if (axis == 0) {
    d = fx_raw_row(fx_load_row<false>(fx_mat(Dp, nu, s, V), r));
    ed = fx_exp(Dp, nu, s, V);
  }
#pragma unroll 1
  for (int k = 1 + axis; k < 4; k += AXES) {
    fx_acc acc = {{0, 0, 0}, {0, 0, 0}};
    int ea = -GF_FX_BAD;
    fx_gather_axis(acc, ea, U, Z, g, st, s, nu, nu_up, (nu + k) & 3, r);
    fx_down_row<1>(acc);
    fx_scale_row(acc, rho);
    fx_add(d, ed, acc, ea + 1 + rho.e);  // |d| <= 1 + 3 * 1.5
  }
  fx_sum_axes<AXES>(ax, axis, link, r, d, ed);
  const int e = OUT == 2 ? ed + 3 + fx_exp(U, nu, s, V) : ed;
  const bool f64 = axis == 0 && fx_has_f64(e);
  if (axis == 0 && r == 0) se[link] = e;
  bool any64;
  if (OUT == 2) {
    if (axis == 0) fx_share<3>(sh.d, link, r, d);
    any64 = __syncthreads_or(f64);
    fx_acc m;
    if (axis == 0) m = fx_row_mul<false>(fx_load_row<false>(fx_mat(U, nu, s, V), r), FxShMat{&sh.d, link});
    __syncthreads();
    if (axis == 0) fx_share(sh.m, link, r, m);
    __syncthreads();
    if (axis == 0) fx_update_mom(sh.m, se, P, nu, s0, V, coef, 1.0);
  } else if (OUT == 1) {
    any64 = __syncthreads_or(f64);
    if (sx < V && axis == 0 && !f64) {
      double2* o = reinterpret_cast<double2*>(Dout) + (size_t)nu * 9 * V + s;
#pragma unroll
      for (int j = 0; j < 3; ++j)
        o[(size_t)(3 * r + j) * V] = make_double2(fx_to_f64(d.re[j], ed), fx_to_f64(d.im[j], ed));
    }
  } else {
    if (axis == 0) sh.n[r][link] = fx_square(d);
    any64 = __syncthreads_or(f64);
    if (sx < V && axis == 0 && !f64) {
      const int k = fx_norm_shift(sh.n[0][link] + sh.n[1][link] + sh.n[2][link], ed);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        d.re[j] = fx_shift(d.re[j], k);
        d.im[j] = fx_shift(d.im[j], k);
      }
      const size_t off = fx_offset(nu, s, V);
      fx_store_row(Dout, off, r, d);
      if (r == 0) fx_store_exp(Dout, off, s, ed + k);
    }
  }
  if (any64) gather_rows64<OUT>(U, Z, Dp, Dout, P, g, rho64, coef, nu, s0, sh.m, se);
}

// --------------------------------------------------------------------------
// host side: forward and backward of a fixed-point stack (stout_forward and
// stout_backward of gf_stout.cu)
// --------------------------------------------------------------------------
static fx_scalar third_of(double c) {
  // c / 3 in the units of fx_scalar_of(c)
  const fx_scalar s = fx_scalar_of(c);
  fx_scalar r = s;
  fx_split<0>(fx_join(s.h, s.l) / 3, r.h, r.l);
  return r;
}

static int axes_of(const gf_ctx* ctx) { return ctx->geom.vol <= GF_FX_SPLIT_MAX ? 3 : 1; }

void stout_forward_fx(gf_ctx* ctx, gf_stout* st) {
  const int nb = 4 * blocks_for(ctx->geom.vol, GF_FX_LINKS);
  for (int l = 0; l < st->nlev; ++l) {
    ProfScope prof(ctx, GF_K_STOUT_FWD64);
    const int axes = axes_of(ctx);
    auto kern = axes == 3 ? k_stout_fwd_fx<3, 2>
                          : (ctx->geom.vol <= GF_FX_FEW_MAX ? k_stout_fwd_fx<1, GF_FX_FEW_MINB>
                                                            : k_stout_fwd_fx<1, GF_FX_FWD_MINB>);
    kern<<<nb, axes * GF_FX_THREADS, 0, ctx->stream>>>(fx_view(st->lev_in[l]), (char*)st->lev_in[l + 1]->ptr,
                                                       st->store ? (char*)st->C[l]->ptr : nullptr, ctx->geom,
                                                       fx_scalar_of(st->rho[l]), third_of(st->rho[l]), st->rho[l]);
    GF_CHECK_LAUNCH();
  }
}

void stout_backward_fx(gf_ctx* ctx, gf_stout* st, const gf_field* dSdUbar, double beta, gf_field* dSdU, gf_field* P,
                       double eps, double* dsdrho) {
  const int nb = 4 * blocks_for(ctx->geom.vol, GF_FX_LINKS);
  if (dSdUbar && dSdUbar != st->D[1]) copy_field(ctx, st->D[1], dSdUbar);
  for (int l = st->nlev - 1; l >= 0; --l) {
    bool top = (l == st->nlev - 1) && dSdUbar == nullptr;
    {
      ProfScope prof(ctx, GF_K_BWD_LOCAL64);
      if (top && ctx->geom.vol > GF_FX_DSDU_MIN) {
        k_dsdu_fx<<<nb, GF_FX_THREADS, 0, ctx->stream>>>(fx_view(st->lev_in[l + 1]), (char*)st->D[1]->ptr, ctx->geom,
                                                         fx_scalar_of(0.5 * beta), 0.5 * beta);
        GF_CHECK_LAUNCH();
        top = false;
      }
      const FxField C = st->store ? fx_view(st->C[l]) : FxField{nullptr};
      const size_t smem = fx_local_bytes(top, !st->store);
      auto kern = st->store ? (top ? k_bwd_local_fx<true, false> : k_bwd_local_fx<false, false>)
                            : (top ? k_bwd_local_fx<true, true> : k_bwd_local_fx<false, true>);
      GF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      kern<<<nb, GF_FX_THREADS, smem, ctx->stream>>>(fx_view(st->lev_in[l]),
                                                     fx_view(top ? st->lev_in[l + 1] : st->D[1]), C,
                                                     (char*)st->Z->ptr, (char*)st->Dp->ptr, ctx->geom,
                                                     fx_scalar_of(st->rho[l]), fx_scalar_of(1.0), third_of(1.0),
                                                     fx_scalar_of(0.5 * beta), st->rho[l], 0.5 * beta);
      GF_CHECK_LAUNCH();
    }
    if (dsdrho) dsdrho[l] = level_dsdrho(ctx, st, l);
    ProfScope prof(ctx, GF_K_BWD_GATHER64);
    const FxField u = fx_view(st->lev_in[l]), z = fx_view(st->Z), dp = fx_view(st->Dp);
    const fx_scalar rho = fx_scalar_of(st->rho[l]);
    const bool split = axes_of(ctx) == 3;
    const int nt = (split ? 3 : 1) * GF_FX_THREADS;
    if (l == 0 && P)
      (split ? k_bwd_gather_fx<2, 3> : k_bwd_gather_fx<2, 1>)<<<nb, nt, 0, ctx->stream>>>(
          u, z, dp, nullptr, (double*)P->ptr, ctx->geom, rho, st->rho[l], -eps / 3.0);
    else if (l == 0 && dSdU)
      (split ? k_bwd_gather_fx<1, 3> : k_bwd_gather_fx<1, 1>)<<<nb, nt, 0, ctx->stream>>>(
          u, z, dp, (char*)dSdU->ptr, nullptr, ctx->geom, rho, st->rho[l], 0.0);
    else
      (split ? k_bwd_gather_fx<0, 3> : k_bwd_gather_fx<0, 1>)<<<nb, nt, 0, ctx->stream>>>(
          u, z, dp, (char*)st->D[1]->ptr, nullptr, ctx->geom, rho, st->rho[l], 0.0);
    GF_CHECK_LAUNCH();
  }
}

}  // namespace gf
