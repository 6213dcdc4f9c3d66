// Plaquette + rectangle action (the loops of gf_rect.cu) in block fixed point
// by rows: the loop sum, the force, and dS/dUbar on a stack's top level. Bound
// by integer multiply-add issue; the force on 65,520 sites: 5.95 ms in fp64
// arithmetic, 0.82 ms here.
#include "gf_internal.h"
#include "stencil.cuh"
#include <algorithm>

namespace gf {

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
};

// lexicographic offset of d steps (|d| <= 2) along mu; extents are at least 2
__device__ __forceinline__ int fx_steps(const Geom& g, const Site& st, int mu, int d) {
  const int c = coord(st, mu), L = g.L[mu];
  int n = c + d;
  n += n < 0 ? L : 0;
  n -= n >= L ? L : 0;
  return (n - c) * g.stride[mu];
}

// Sum over sites and planes of Re tr of the 1x2 and 2x1 rectangles, one
// partial per block; a work item is one plane of 32 sites.
__global__ void __launch_bounds__(GF_FX_THREADS, GF_FX_MINB)
    k_rect_sum_fx(FxField U, Geom g, int items, SumOut to) {
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

// acc (+)= [cp t_p + cr (t_1 + t_2)] / 4 as an operand row; cp and cr share
// one exponent (cp.e). |t| <= 1, so the bracket is below 3 units.
__device__ __forceinline__ fx_row fx_weighted(const FxChain& tp, FxChain t1, const FxChain& t2, fx_scalar cp,
                                              fx_scalar cr, int& e) {
  fx_add(t1.v, t1.e, t2.v, t2.e);
  fx_acc p = tp.v;
  int ep = tp.e;
  // one exponent for both summands
  fx_acc zero = {{0, 0, 0}, {0, 0, 0}};
  fx_add(p, ep, zero, t1.e);
  fx_add(t1.v, t1.e, zero, ep);
  fx_acc out;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    fx_sum re = fx_zero_sum(), im = fx_zero_sum();
    fx_mac(re, fx_pre(p.re[j] >> 1), fx_num_of(cp));
    fx_mac(re, fx_pre(t1.v.re[j] >> 1), fx_num_of(cr));
    fx_mac(im, fx_pre(p.im[j] >> 1), fx_num_of(cp));
    fx_mac(im, fx_pre(t1.v.im[j] >> 1), fx_num_of(cr));
    out.re[j] = fx_get(re);
    out.im[j] = fx_get(im);
  }
  e = ep + 2 + cp.e;
  return fx_operand<1>(out);
}

// Rows of (cp S + cr R)^dag, S the six plaquette and R the eighteen rectangle
// staples of U_mu(x) (the conjugates of (a)-(f) of gf_rect.cu), by rows from
// the left. Shared factors: per plane and side the plaquette staple and (a),
// (e) (or (b), (f)) end in the same link, (c) and (d) start as the plaquette
// staples do, and all (c), (d) end in U_mu(x+mu)^dag, which is applied once:
// 61 products instead of 84. The sum is below 8 units of 2^ea.
__device__ __forceinline__ fx_acc fx_loops_row(const FxField& U, const Geom& g, const Site& st, int s, int mu, int r,
                                               fx_scalar cp, fx_scalar cr, int& ea) {
  const int V = g.vol;
  fx_acc acc = {{0, 0, 0}, {0, 0, 0}}, far = {{0, 0, 0}, {0, 0, 0}};
  ea = -GF_FX_BAD;
  int ef = -GF_FX_BAD;
  const int m1 = fx_steps(g, st, mu, 1), m2 = fx_steps(g, st, mu, 2), mm = fx_steps(g, st, mu, -1);
  const int xm = eo_of_lex(g, st.lex + m1, st.par ^ 1), x2m = eo_of_lex(g, st.lex + m2, st.par);
  const int xmm = eo_of_lex(g, st.lex + mm, st.par ^ 1);
#pragma unroll 1
  for (int k = 1; k < 4; ++k) {
    const int nu = (mu + k) & 3;
    {
      const int n1 = fx_steps(g, st, nu, 1), n2 = fx_steps(g, st, nu, 2);
      const int xn = eo_of_lex(g, st.lex + n1, st.par ^ 1), x2n = eo_of_lex(g, st.lex + n2, st.par);
      const int xmn = eo_of_lex(g, st.lex + m1 + n1, st.par), xmmn = eo_of_lex(g, st.lex + mm + n1, st.par);
      const fx_row a = fx_load_row<false>(fx_mat(U, nu, s, V), r);
      const int e0 = fx_exp(U, nu, s, V);
      FxChain p{U, V, {}, e0};
      p.mul<false>(a, mu, xn);
      FxChain c = p;  // (c)
      c.mul<false>(mu, xmn).mul<true>(nu, x2m);
      fx_add(far, ef, c.v, c.e);
      FxChain ta{U, V, {}, e0};  // (a)
      ta.mul<false>(a, nu, xn).mul<false>(mu, x2n).mul<true>(nu, xmn);
      FxChain te{U, V, {}, fx_exp(U, mu, xmm, V)};  // (e)
      te.mul<false>(fx_load_row<true>(fx_mat(U, mu, xmm, V), r), nu, xmm).mul<false>(mu, xmmn).mul<false>(mu, xn);
      FxChain f{U, V, {}, 0};
      const fx_row w = fx_weighted(p, ta, te, cp, cr, f.e);
      f.mul<true>(w, nu, xm);
      fx_add(acc, ea, f.v, f.e);
    }
    {
      const int n1 = fx_steps(g, st, nu, -1), n2 = fx_steps(g, st, nu, -2);
      const int xn = eo_of_lex(g, st.lex + n1, st.par ^ 1), x2n = eo_of_lex(g, st.lex + n2, st.par);
      const int xmn = eo_of_lex(g, st.lex + m1 + n1, st.par), xmmn = eo_of_lex(g, st.lex + mm + n1, st.par);
      const int xm2n = eo_of_lex(g, st.lex + m1 + n2, st.par ^ 1), x2mn = eo_of_lex(g, st.lex + m2 + n1, st.par ^ 1);
      const fx_row a = fx_load_row<true>(fx_mat(U, nu, xn, V), r);
      const int e0 = fx_exp(U, nu, xn, V);
      FxChain p{U, V, {}, e0};
      p.mul<false>(a, mu, xn);
      FxChain c = p;  // (d)
      c.mul<false>(mu, xmn).mul<false>(nu, x2mn);
      fx_add(far, ef, c.v, c.e);
      FxChain tb{U, V, {}, e0};  // (b)
      tb.mul<true>(a, nu, x2n).mul<false>(mu, x2n).mul<false>(nu, xm2n);
      FxChain tf{U, V, {}, fx_exp(U, mu, xmm, V)};  // (f)
      tf.mul<true>(fx_load_row<true>(fx_mat(U, mu, xmm, V), r), nu, xmmn).mul<false>(mu, xmmn).mul<false>(mu, xn);
      FxChain f{U, V, {}, 0};
      const fx_row w = fx_weighted(p, tb, tf, cp, cr, f.e);
      f.mul<false>(w, nu, xmn);
      fx_add(acc, ea, f.v, f.e);
    }
  }
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

// P <- keep P + c(U (cp S + cr R)), or (DSDU) D = cp S + cr R
#ifndef GF_FX_LOOPS_MINB
#define GF_FX_LOOPS_MINB 5
#endif
template <bool DSDU>
__global__ void __launch_bounds__(GF_FX_THREADS, GF_FX_LOOPS_MINB)
    k_loops_fx(FxField U, double* __restrict__ P, char* __restrict__ D, Geom g, fx_scalar cp, fx_scalar cr,
               double keep) {
  __shared__ union {
    FxRaw m;
    float n[3][GF_FX_LINKS];
  } sh;
  __shared__ int se[GF_FX_LINKS];
  const int t = threadIdx.x, mu = blockIdx.x & 3, V = g.vol;
  const int link = t / 3, r = t - 3 * link, s0 = (blockIdx.x >> 2) * GF_FX_LINKS;
  const int sx = s0 + link, s = min(sx, V - 1);
  const Site st = site_of(g, s);
  int ea;
  fx_acc a = fx_loops_row(U, g, st, s, mu, r, cp, cr, ea);
  if (DSDU) {
    sh.n[r][link] = fx_square(a);
    __syncthreads();
    if (sx >= V) return;
    const int k = fx_norm_shift(sh.n[0][link] + sh.n[1][link] + sh.n[2][link], ea);
    const size_t off = fx_offset(mu, s, V);
#pragma unroll
    for (int j = 0; j < 3; ++j) fx_store(D, off, 3 * j + r, fx_shift(a.re[j], k), -fx_shift(a.im[j], k));
    if (r == 0) fx_store_exp(D, off, s, ea + k);
    return;
  }
  fx_share(sh.m, link, r, fx_row_mul<true>(fx_operand<3>(a), fx_mat(U, mu, s, V)));
  if (r == 0) se[link] = ea + 3 + fx_exp(U, mu, s, V);
  __syncthreads();
  fx_update_mom(sh.m, se, P, mu, s0, V, -1.0, keep);
}

void loops_fx(gf_ctx* ctx, const gf_field* F, gf_field* P, gf_field* D, double cp, double cr, double keep) {
  // both coefficients in units of one power of two
  const fx_scalar c = fx_scalar_of(std::max(std::fabs(cp), std::fabs(cr)));
  fx_scalar p = c, q = c;
  fx_split<0>((i64)ldexp(cp, 60 - c.e), p.h, p.l);
  fx_split<0>((i64)ldexp(cr, 60 - c.e), q.h, q.l);
  const int nb = 4 * blocks_for(ctx->geom.vol, GF_FX_LINKS);
  ProfScope prof(ctx, GF_K_RECT);
  if (D)
    k_loops_fx<true><<<nb, GF_FX_THREADS, 0, ctx->stream>>>(fx_view(F), nullptr, (char*)D->ptr, ctx->geom, p, q, 0.0);
  else
    k_loops_fx<false><<<nb, GF_FX_THREADS, 0, ctx->stream>>>(fx_view(F), (double*)P->ptr, nullptr, ctx->geom, p, q,
                                                             keep);
  GF_CHECK_LAUNCH();
}

}  // namespace gf
