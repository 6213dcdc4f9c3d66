// Plaquette + rectangle action (the loops of gf_rect.cu) in block fixed point
// by rows: the loop sum, the force, and dS/dUbar on a stack's top level. Bound
// by integer multiply-add issue; the force on 65,520 sites: 5.95 ms in fp64
// arithmetic, 0.66 ms here.
#include "gf_internal.h"
#include "fxrows64.cuh"
#include "stencil.cuh"
#include <algorithm>

namespace gf {

// the imaginary parts of a row negated
__device__ __forceinline__ void fx_conj(fx_row& a) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    a.bh[k] = -a.bh[k];
    a.bl[k] = -a.bl[k];
  }
}
// a matrix of a field or its transpose: distances of its rows and columns
struct FxTurned {
  const char* p;
  int row, column;
  __device__ __forceinline__ int4 operator()(int el) const {
    return __ldg(reinterpret_cast<const int4*>(p + (el / 3) * row + (el % 3) * column));
  }
};

// A running row of a product of links, with its exponent.
struct FxChain {
  const FxField& U;
  int V;
  fx_acc v;
  int e;
  template <bool DAG>
  __device__ __forceinline__ FxChain& mul(const fx_row& a, int dir, int site) {
    v = fx_row_mul<DAG>(a, fx_mat(U, dir, site, V));
    e += fx_exp(U, dir, site, V);
    return *this;
  }
  template <bool DAG>
  __device__ __forceinline__ FxChain& mul(int dir, int site) {
    return mul<DAG>(fx_operand<0>(v), dir, site);
  }
  // the same with the dagger chosen at run time, one copy of the product for
  // both: a U^dag = conj(conj(a) U^T)
  __device__ __forceinline__ FxChain& mul(fx_row a, int dir, int site, bool dag) {
    const FxTurned u{fx_mat(U, dir, site, V).p, dag ? 512 : 3 * 512, dag ? 3 * 512 : 512};
    if (dag) fx_conj(a);
    v = fx_row_mul<false>(a, u);
    if (dag) {
#pragma unroll
      for (int j = 0; j < 3; ++j) v.im[j] = -v.im[j];
    }
    e += fx_exp(U, dir, site, V);
    return *this;
  }
  __device__ __forceinline__ FxChain& mul(int dir, int site, bool dag) {
    return mul(fx_operand<0>(v), dir, site, dag);
  }
};
// row r of a link, or of its dagger, chosen at run time
__device__ __forceinline__ fx_row fx_load_row(const FxMat& M, int r, bool dag) {
  const FxTurned u{M.p, dag ? 512 : 3 * 512, dag ? 3 * 512 : 512};
  fx_row a;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int4 v = __ldg(reinterpret_cast<const int4*>(u.p + r * u.row + k * u.column));
    a.ah[k] = v.x;
    a.al[k] = v.y;
    a.bh[k] = v.z;
    a.bl[k] = v.w;
  }
  if (dag) fx_conj(a);
  return a;
}

// lexicographic offset of d steps (|d| <= 2) along mu; extents are at least 2
__device__ __forceinline__ int fx_steps(const Geom& g, const Site& st, int mu, int d) {
  const int c = coord(st, mu), L = g.L[mu];
  int n = c + d;
  n += n < 0 ? L : 0;
  n -= n >= L ? L : 0;
  return (n - c) * g.stride[mu];
}

// row r of a rectangle's product in fp64, times row r of U_nu(x)
__device__ __noinline__ double rect_row64(const FxField U, int mu, int nu, int s, int xm, int xmn, int xnn, int xn,
                                          int r, int V) {
  row64 a = mul64<false>(load_row64<false>(fx_mat64(U, mu, s, V), r), fx_mat64(U, nu, xm, V));
  a = mul64<false>(a, fx_mat64(U, nu, xmn, V));
  a = mul64<true>(mul64<true>(a, fx_mat64(U, mu, xnn, V)), fx_mat64(U, nu, xn, V));
  const row64 b = load_row64<false>(fx_mat64(U, nu, s, V), r);
  double v = 0.0;
#pragma unroll
  for (int k = 0; k < 3; ++k) v = fma(a.re[k], b.re[k], fma(a.im[k], b.im[k], v));
  return v;
}

// Sum over sites and planes of Re tr of the 1x2 and 2x1 rectangles, one
// partial per block; a work item is one plane of 32 sites.
__global__ void __launch_bounds__(GF_FX_THREADS, GF_FX_MINB)
    k_rect_sum_fx(FxField U, const __grid_constant__ Geom g, int items, SumOut to) {
  const int t = threadIdx.x, V = g.vol;
  const int link = t / 3, r = t - 3 * link;
  double v = 0.0;
#pragma unroll 1
  for (int it = blockIdx.x; it < items; it += gridDim.x) {
    const int tile = it / 12, p = (it - 12 * tile) >> 1, swap = it & 1;
    int mu = p < 3 ? 0 : (p < 5 ? 1 : 2), nu = p < 3 ? p + 1 : (p < 5 ? p - 1 : 3);
    // the 2x1 rectangle is the 1x2 one of the other orientation, reversed
    if (swap) {
      const int m = mu;
      mu = nu;
      nu = m;
    }
    const int s = tile * GF_FX_LINKS + link;
    if (s >= V) continue;
    const Site st = site_of(g, s);
    const int m1 = fx_steps(g, st, mu, 1), n1 = fx_steps(g, st, nu, 1), n2 = fx_steps(g, st, nu, 2);
    const int xm = eo_of_lex(g, st.lex + m1, st.par ^ 1), xmn = eo_of_lex(g, st.lex + m1 + n1, st.par);
    const int xnn = eo_of_lex(g, st.lex + n2, st.par), xn = eo_of_lex(g, st.lex + n1, st.par ^ 1);
    // U_mu(x) U_nu(x+mu) U_nu(x+mu+nu) U_mu(x+2nu)^+ U_nu(x+nu)^+ . U_nu(x)^+
    FxChain c{U, V, {}, fx_exp(U, mu, s, V) + fx_exp(U, nu, s, V)};
    c.mul<false>(fx_load_row<false>(fx_mat(U, mu, s, V), r), nu, xm).mul<false>(nu, xmn);
    c.mul<true>(mu, xnn).mul<true>(nu, xn);
    if (fx_has_f64(c.e)) {
      v += rect_row64(U, mu, nu, s, xm, xmn, xnn, xn, r, V);
      continue;
    }
    const fx_row b = fx_load_row<false>(fx_mat(U, nu, s, V), r);
    fx_sum d = fx_zero_sum();
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      fx_mac(d, fx_pre(c.v.re[k]), fx_num{b.ah[k], b.al[k]});
      fx_mac(d, fx_pre(c.v.im[k]), fx_num{b.bh[k], b.bl[k]});
    }
    v = fma(fx_value(fx_get(d)), fx_unit(1.0, c.e), v);
  }
  block_sum(v, to);
}

void rectangle_start_fx(gf_ctx* ctx, const gf_field* F, int slot) {
  const int items = 12 * blocks_for(ctx->geom.vol, GF_FX_LINKS);
  const int nb = std::min(std::min(items, ctx->sm_count * GF_FX_MINB * 8), ctx->partial_cap);
  const SumOut to = sum_out(ctx, nb, GF_FX_THREADS, slot);
  ProfScope prof(ctx, GF_K_RECT);
  k_rect_sum_fx<<<nb, GF_FX_THREADS, 0, ctx->stream>>>(fx_view(F), ctx->geom, items, to);
  GF_CHECK_LAUNCH();
  sum_finish(ctx, to, nb, slot);
}

// [cp p + cr t] / 4 as an operand row. Each summand is scaled before the sum
// aligns it: a small or zero coefficient of a large p leaves t its digits. |p| <= 1
// and |t| <= 2, so the sum is below 1.5 units.
__device__ __forceinline__ fx_row fx_weighted(const FxChain& p, const FxChain& t, fx_scalar cp, fx_scalar cr, int& e) {
  fx_acc a = p.v, b = t.v;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    a.re[j] = fx_mul(fx_pre(a.re[j] >> 1), fx_num_of(cp));
    a.im[j] = fx_mul(fx_pre(a.im[j] >> 1), fx_num_of(cp));
    b.re[j] = fx_mul(fx_pre(b.re[j] >> 1), fx_num_of(cr));
    b.im[j] = fx_mul(fx_pre(b.im[j] >> 1), fx_num_of(cr));
  }
  int ea = p.e + 1 + cp.e;
  fx_add(a, ea, b, t.e + 1 + cr.e);
  e = ea + 1;
  return fx_operand<1>(a);
}

__device__ __forceinline__ fx_acc fx_parked(const i64* park) {
  fx_acc v;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    v.re[j] = park[2 * j * GF_FX_THREADS];
    v.im[j] = park[(2 * j + 1) * GF_FX_THREADS];
  }
  return v;
}

// Rows of (cp S + cr R)^dag, S the six plaquette and R the eighteen rectangle
// staples of U_mu(x) (the conjugates of (a)-(f) of gf_rect.cu), by rows from
// the left. Shared factors: per plane and side the plaquette staple and (a),
// (e) (or (b), (f)) end in the same link, (c) and (d) start as the plaquette
// staples do, and all (c), (d) end in U_mu(x+mu)^dag, which is applied once:
// 61 products instead of 84. The sum is below 8 units of 2^ea. One loop body
// of ten products serves both sides: with a body for each, 96 KB of code,
// warps waited for instructions three times as long as they issued (24^4: 4.22
// ms; one body 3.71). (a), (b), (e), (f) first, so that the least stays alive:
// 3.40 ms; the sum of (c), (d) parked in shared memory (park, this thread's
// six words): 3.30 ms.
__device__ __forceinline__ fx_acc fx_loops_row(const FxField& U, const Geom& g, const Site& st, int s, int mu, int r,
                                               fx_scalar cp, fx_scalar cr, int& ea, i64* park) {
  const int V = g.vol;
  fx_acc acc = {{0, 0, 0}, {0, 0, 0}};
#pragma unroll
  for (int j = 0; j < 6; ++j) park[j * GF_FX_THREADS] = 0;
  ea = -GF_FX_BAD;
  int ef = -GF_FX_BAD;
  const int m1 = fx_steps(g, st, mu, 1), m2 = fx_steps(g, st, mu, 2), mm = fx_steps(g, st, mu, -1);
  const int xm = eo_of_lex(g, st.lex + m1, st.par ^ 1), x2m = eo_of_lex(g, st.lex + m2, st.par);
  const int xmm = eo_of_lex(g, st.lex + mm, st.par ^ 1);
#pragma unroll 1
  for (int k = 2; k < 8; ++k) {
    // above (even k) or below the link
    const int nu = (mu + (k >> 1)) & 3;
    const bool low = k & 1;
    const int n1 = fx_steps(g, st, nu, low ? -1 : 1), n2 = fx_steps(g, st, nu, low ? -2 : 2);
    const int xn = eo_of_lex(g, st.lex + n1, st.par ^ 1), x2n = eo_of_lex(g, st.lex + n2, st.par);
    const int xmn = eo_of_lex(g, st.lex + m1 + n1, st.par), xmmn = eo_of_lex(g, st.lex + mm + n1, st.par);
    const int start = low ? xn : s;
    const FxMat first = fx_mat(U, nu, start, V);
    const int e0 = fx_exp(U, nu, start, V);
    FxChain t{U, V, {}, e0};  // (a), (b)
    t.mul(fx_load_row(first, r, low), nu, low ? x2n : xn, low).mul<false>(mu, x2n);
    t.mul(nu, low ? eo_of_lex(g, st.lex + m1 + n2, st.par ^ 1) : xmn, !low);
    {
      FxChain te{U, V, {}, fx_exp(U, mu, xmm, V)};  // (e), (f)
      te.mul(fx_load_row<true>(fx_mat(U, mu, xmm, V), r), nu, low ? xmmn : xmm, low);
      te.mul<false>(mu, xmmn).mul<false>(mu, xn);
      fx_add(t.v, t.e, te.v, te.e);
    }
    FxChain p{U, V, {}, e0};
    p.mul<false>(fx_load_row(first, r, low), mu, xn);
    {
      FxChain c = p;  // (c), (d)
      c.mul<false>(mu, xmn);
      c.mul(nu, low ? eo_of_lex(g, st.lex + m2 + n1, st.par ^ 1) : x2m, !low);
      fx_acc far = fx_parked(park);
      fx_add(far, ef, c.v, c.e);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        park[2 * j * GF_FX_THREADS] = far.re[j];
        park[(2 * j + 1) * GF_FX_THREADS] = far.im[j];
      }
    }
    FxChain f{U, V, {}, 0};
    const fx_row w = fx_weighted(p, t, cp, cr, f.e);
    f.mul(w, nu, low ? xmn : xm, !low);
    fx_add(acc, ea, f.v, f.e);
  }
  fx_acc far = fx_parked(park);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    far.re[j] >>= 3;
    far.im[j] >>= 3;
  }
  fx_scale_row(far, cr);
  FxChain f{U, V, far, ef + 3 + cr.e};
  f.mul<true>(mu, xm);
  fx_add(acc, ea, f.v, f.e);
  return acc;
}

// the same row in fp64, in the chains of fx_loops_row
__device__ __forceinline__ row64 loops_row64(const FxField& U, const Geom& g, const Site& st, int s, int mu, int r,
                                             double cp, double cr) {
  const int V = g.vol;
  row64 acc = zero64(), far = zero64();
  const int m1 = fx_steps(g, st, mu, 1), m2 = fx_steps(g, st, mu, 2), mm = fx_steps(g, st, mu, -1);
  const int xm = eo_of_lex(g, st.lex + m1, st.par ^ 1), x2m = eo_of_lex(g, st.lex + m2, st.par);
  const int xmm = eo_of_lex(g, st.lex + mm, st.par ^ 1);
#pragma unroll 1
  for (int k = 2; k < 8; ++k) {
    const int nu = (mu + (k >> 1)) & 3;
    const bool low = k & 1;
    const int n1 = fx_steps(g, st, nu, low ? -1 : 1), n2 = fx_steps(g, st, nu, low ? -2 : 2);
    const int xn = eo_of_lex(g, st.lex + n1, st.par ^ 1), x2n = eo_of_lex(g, st.lex + n2, st.par);
    const int xmn = eo_of_lex(g, st.lex + m1 + n1, st.par), xmmn = eo_of_lex(g, st.lex + mm + n1, st.par);
    const int xmnn = low ? eo_of_lex(g, st.lex + m1 + n2, st.par ^ 1) : xmn;
    const int x2mn = low ? eo_of_lex(g, st.lex + m2 + n1, st.par ^ 1) : x2m;
    const FxMat64 start = fx_mat64(U, nu, low ? xn : s, V);
    const row64 first = low ? load_row64<true>(start, r) : load_row64<false>(start, r);
    row64 t = mul64(first, fx_mat64(U, nu, low ? x2n : xn, V), low);  // (a), (b)
    t = mul64(mul64<false>(t, fx_mat64(U, mu, x2n, V)), fx_mat64(U, nu, xmnn, V), !low);
    // (e), (f)
    const row64 te = mul64(load_row64<true>(fx_mat64(U, mu, xmm, V), r), fx_mat64(U, nu, low ? xmmn : xmm, V), low);
    add64(t, mul64<false>(mul64<false>(te, fx_mat64(U, mu, xmmn, V)), fx_mat64(U, mu, xn, V)));
    const row64 p = mul64<false>(first, fx_mat64(U, mu, xn, V));
    add64(far, mul64(mul64<false>(p, fx_mat64(U, mu, xmn, V)), fx_mat64(U, nu, x2mn, V), !low));  // (c), (d)
    row64 w = zero64();
    add64(w, p, cp);
    add64(w, t, cr);
    add64(acc, mul64(w, fx_mat64(U, nu, low ? xmn : xm, V), !low));
  }
  add64(acc, mul64<true>(far, fx_mat64(U, mu, xm, V)), cr);
  return acc;
}
template <bool DSDU>
__device__ __noinline__ void loops_rows64(const FxField U, double* P, char* D, const Geom& g, int mu, int s0, double cp,
                                          double cr, double keep, FxRaw& sh, const int* se) {
  const int t = threadIdx.x, link = t / 3, r = t - 3 * link, V = g.vol;
  __syncthreads();  // sh has been read
  if (fx_has_f64(se[link])) {
    const int s = min(s0 + link, V - 1);
    row64 a = loops_row64(U, g, site_of(g, s), s, mu, r, cp, cr);
    if (!DSDU) a = mul64<true>(a, fx_mat64(U, mu, s, V));
    share64(sh64(sh, link), r, a);
  }
  __syncthreads();
  if (!DSDU) {
    update_mom64(sh64(sh, t & 31), se, P, mu, s0, V, -1.0, keep);
  } else if (t < GF_FX_LINKS && s0 + t < V && fx_has_f64(se[t])) {
    store_field64(sh64(sh, t), D, mu, s0 + t, V, true);
  }
}

// P <- keep P + c(U (cp S + cr R)), or (DSDU) D = cp S + cr R. Four blocks per
// SM (168 registers): 3.30 ms at 24^4, five 3.36, six 3.81.
#ifndef GF_FX_LOOPS_MINB
#define GF_FX_LOOPS_MINB 4
#endif
template <bool DSDU>
__global__ void __launch_bounds__(GF_FX_THREADS, GF_FX_LOOPS_MINB)
    k_loops_fx(FxField U, double* __restrict__ P, char* __restrict__ D, const __grid_constant__ Geom g, fx_scalar cp,
               fx_scalar cr, double cp64, double cr64, double keep) {
  __shared__ union {
    FxRaw m;
    float n[3][GF_FX_LINKS];
  } sh;
  __shared__ i64 park[6][GF_FX_THREADS];
  __shared__ int se[GF_FX_LINKS];
  const int t = threadIdx.x, mu = blockIdx.x & 3, V = g.vol;
  const int link = t / 3, r = t - 3 * link, s0 = (blockIdx.x >> 2) * GF_FX_LINKS;
  const int sx = s0 + link, s = min(sx, V - 1);
  const Site st = site_of(g, s);
  int ea;
  fx_acc a = fx_loops_row(U, g, st, s, mu, r, cp, cr, ea, park[0] + t);
  const int e = ea + 3 + fx_exp(U, mu, s, V);
  const bool f64 = fx_has_f64(DSDU ? ea : e);
  if (r == 0) se[link] = DSDU ? ea : e;
  bool any64;
  if (DSDU) {
    sh.n[r][link] = fx_square(a);
    any64 = __syncthreads_or(f64);
    if (sx < V && !f64) {
      const int k = fx_norm_shift(sh.n[0][link] + sh.n[1][link] + sh.n[2][link], ea);
      const size_t off = fx_offset(mu, s, V);
#pragma unroll
      for (int j = 0; j < 3; ++j) fx_store(D, off, 3 * j + r, fx_shift(a.re[j], k), -fx_shift(a.im[j], k));
      if (r == 0) fx_store_exp(D, off, s, ea + k);
    }
  } else {
    fx_share(sh.m, link, r, fx_row_mul<true>(fx_operand<3>(a), fx_mat(U, mu, s, V)));
    any64 = __syncthreads_or(f64);
    fx_update_mom(sh.m, se, P, mu, s0, V, -1.0, keep);
  }
  if (any64) loops_rows64<DSDU>(U, P, D, g, mu, s0, cp64, cr64, keep, sh.m, se);
}

void loops_fx(gf_ctx* ctx, const gf_field* F, gf_field* P, gf_field* D, double cp, double cr, double keep) {
  const fx_scalar p = fx_scalar_of(cp), q = fx_scalar_of(cr);
  const int nb = 4 * blocks_for(ctx->geom.vol, GF_FX_LINKS);
  ProfScope prof(ctx, GF_K_RECT);
  if (D)
    k_loops_fx<true><<<nb, GF_FX_THREADS, 0, ctx->stream>>>(fx_view(F), nullptr, (char*)D->ptr, ctx->geom, p, q, cp,
                                                            cr, 0.0);
  else
    k_loops_fx<false><<<nb, GF_FX_THREADS, 0, ctx->stream>>>(fx_view(F), (double*)P->ptr, nullptr, ctx->geom, p, q, cp,
                                                             cr, keep);
  GF_CHECK_LAUNCH();
}

}  // namespace gf
