// Link update U <- exp(i eps P) U (update_gaugefields!,
// src/molecular_dynamics.jl:513-531; exptU!, src/4D/TA_gaugefields_4D_serial.jl:760)
// with the Cayley-Hamilton exponential, optional re-unitarisation
// (normalize3!, src/AbstractGaugefields.jl:3378) and an optional fp32
// 12-real shadow copy for the mixed-precision force path. One kernel for every
// precision form: fp64 storage, fixed-point arithmetic of fp64 class.
#include "gf_internal.h"

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

// rows a, b -> orthonormal, c = conj(a x b) (normalize3!,
// src/AbstractGaugefields.jl:3378). Returns how many rows are defined.
__device__ __forceinline__ int fx_unitarise(fx_acc w[3]) {
  if (!fx_unit_row(w[0])) return 0;
  fx_num ar[3], ai[3], br[3], bi[3];
  // row 2 relative to its own size, so that the projection keeps its digits
  const int d = fx_norm_shift(fx_square(w[1]), 0);
  fx_sum pr = fx_zero_sum(), pi = fx_zero_sum();
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    w[1].re[j] = fx_shift(w[1].re[j], d);
    w[1].im[j] = fx_shift(w[1].im[j], d);
    br[j] = fx_pre(w[1].re[j]);
    bi[j] = fx_pre(w[1].im[j]);
    ar[j] = fx_pre(w[0].re[j]);
    ai[j] = fx_pre(w[0].im[j]);
    fx_cmac(pr, pi, br[j], bi[j], ar[j], fx_neg(ai[j]));
  }
  const fx_num xr = fx_pre(fx_get(pr)), xi = fx_pre(fx_get(pi));
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    fx_sum yr = fx_zero_sum(), yi = fx_zero_sum();
    fx_cmac(yr, yi, xr, xi, ar[j], ai[j]);
    w[1].re[j] -= fx_get(yr);
    w[1].im[j] -= fx_get(yi);
  }
  if (!fx_unit_row(w[1])) return 1;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    br[j] = fx_pre(w[1].re[j]);
    bi[j] = fx_pre(w[1].im[j]);
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int k = (j + 1) % 3, l = (j + 2) % 3;
    fx_sum re = fx_zero_sum(), im = fx_zero_sum();
    fx_cmac(re, im, ar[k], ai[k], br[l], bi[l]);
    fx_cmac(re, im, fx_neg(ar[l]), fx_neg(ai[l]), br[k], bi[k]);
    w[2].re[j] = fx_get(re);
    w[2].im[j] = -fx_get(im);
  }
  return 3;
}

// links of a matrix from fp64, the exponent from its Frobenius norm
__device__ __forceinline__ int fx_from_f64_fast(const double* m, int4 out[9]) {
  int emax = 1;
#pragma unroll
  for (int i = 0; i < 18; ++i) emax = max(emax, fx_exponent_field(m[i]));
  float n = 0.f;
#pragma unroll
  for (int i = 0; i < 18; ++i) {
    const float f = fx_leading(m[i], emax);
    n = fmaf(f, f, n);
  }
  const int up = (n > 0.999f) + (n > 3.996f) + (n > 15.98f) + (n > 63.9f);
  const bool bad = emax == 0x7FF;
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    fx_split<0>(bad ? 0 : fx_mantissa(m[2 * i], emax, up), out[i].x, out[i].y);
    fx_split<0>(bad ? 0 : fx_mantissa(m[2 * i + 1], emax, up), out[i].z, out[i].w);
  }
  return bad ? GF_FX_BAD : emax - 1023 + up;
}

// blocks per SM of the link update
#ifndef GF_FX_UPDATE_MINB
#define GF_FX_UPDATE_MINB 4
#endif
// W = exp(i eps P) U on fp64 links (Uin, Uout may be the same field). Bound by
// integer issue: 48^4 4.51 ms, where the double-float kernel took 7.18 ms and
// the fp64 one 20 ms; four blocks per SM (128 registers) against 4.88 ms with
// two or three, and 7.85 ms for a row of the link per thread, whose series and
// row-after-row re-unitarisation leave warps waiting at barriers. Against
// 113-bit arithmetic the result is off by 4.9e-17 (the final rounding), the
// fp64 kernel's by 1.6e-16, the double-float one's by 6.2e-15.
template <bool REUNIT>
__global__ void __launch_bounds__(128, GF_FX_UPDATE_MINB)
    k_link_update_fx(const double2* Uin, double2* Uout, const double* __restrict__ P, Geom g, fx_scalar eps,
                     float4* __restrict__ sh32, char* __restrict__ fx) {
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
  int eu;
  {
    const double2* b = Uin + (size_t)mu * 9 * V + s;
    double m[18];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const double2 v = b[(size_t)k * V];
      m[2 * k] = v.x;
      m[2 * k + 1] = v.y;
    }
    eu = fx_from_f64_fast(m, u);
  }
  if (e > GF_FX_BAD / 2) eu = GF_FX_BAD;
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
  double2* o = Uout + (size_t)mu * 9 * V + s;
  double2 v[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int ew = k / 3 < fine ? eu : GF_FX_BAD;
    v[k] = make_double2(fx_to_f64(w[k / 3].re[k % 3], ew), fx_to_f64(w[k / 3].im[k % 3], ew));
    o[(size_t)k * V] = v[k];
  }
  if (sh32) {
    float4* q4 = sh32 + (size_t)mu * 3 * V + s;
#pragma unroll
    for (int k = 0; k < 3; ++k)
      q4[(size_t)k * V] =
          make_float4((float)v[2 * k].x, (float)v[2 * k].y, (float)v[2 * k + 1].x, (float)v[2 * k + 1].y);
  }
  if (fx) {
    // the fixed-point copy of what was stored, as k_to_fx makes it
    double m[18];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      m[2 * k] = v[k].x;
      m[2 * k + 1] = v[k].y;
    }
    int4 el[9];
    const size_t off = fx_offset(mu, s, V);
    fx_store_exp(fx, off, s, fx_from_f64(m, el));
#pragma unroll
    for (int k = 0; k < 9; ++k) *reinterpret_cast<int4*>(fx + off + 512 * k) = el[k];
  }
}

// Sites up to which the update itself writes the fixed-point copy. It saves a
// launch and the copy's pass over the links (8^4 trajectory of 20 steps 784 ->
// 718 us, 24^4 of 10 steps 11.22 -> 11.13 ms), but in registers it costs the
// update more than the bandwidth-bound copy kernel once that runs at full rate
// (32^4 flow, 2 steps: 18.64 against 18.41 ms).
#ifndef GF_FX_FUSE_MAX
#define GF_FX_FUSE_MAX (1 << 19)
#endif
static void update_links(gf_ctx* ctx, gf_field* W, const gf_field* P, double eps, const gf_field* U, int reunit,
                         gf_field* shadow32, gf_field* fx) {
  dim3 grid(blocks_for(ctx->geom.vol, 128), 4);
  const bool fused = ctx->geom.vol <= GF_FX_FUSE_MAX;
  auto kern = reunit ? k_link_update_fx<true> : k_link_update_fx<false>;
  kern<<<grid, 128, 0, ctx->stream>>>((const double2*)U->ptr, (double2*)W->ptr, (const double*)P->ptr, ctx->geom,
                                      fx_scalar_of(eps), shadow32 ? (float4*)shadow32->ptr : nullptr,
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
