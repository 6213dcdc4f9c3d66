// Fixed-point (block floating, integer pipes) kernels of the fp64-class path:
// conversions and the Wilson force.
#include "gf_internal.h"
#include "fxlat.cuh"

namespace gf {

// LINK64 / MAT64 -> fixed point, one link per thread
__global__ void __launch_bounds__(128) k_f64_to_fx(const double2* __restrict__ in, char* __restrict__ out, int V) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x, mu = blockIdx.y;
  if (s >= V) return;
  const double2* b = in + (size_t)mu * 9 * V + s;
  double m[18];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const double2 v = __ldg(b + (size_t)k * V);
    m[2 * k] = v.x;
    m[2 * k + 1] = v.y;
  }
  int4 f[9];
  const int e = fx_from_f64(m, f);
  char* o = out + fx_offset(mu, s, V);
#pragma unroll
  for (int k = 0; k < 9; ++k) *reinterpret_cast<int4*>(o + 512 * k) = f[k];
  *reinterpret_cast<int*>(o + 9 * 512 - 12 * (s & 31)) = e;
}

FxField fx_view(const gf_field* f) { return FxField{(const char*)f->ptr}; }

void f64_to_fx(gf_ctx* ctx, gf_field* dst, const gf_field* src) {
  const int V = ctx->geom.vol;
  dim3 grid(blocks_for(V, 128), 4);
  k_f64_to_fx<<<grid, 128, 0, ctx->stream>>>((const double2*)src->ptr, (char*)dst->ptr, V);
  GF_CHECK_LAUNCH();
}

// the 18 reals of 32 rows-split matrices in shared memory: component-major
// over the links, so a thread per link reads without bank conflicts
struct FxShare {
  i64 v[18][GF_FX_LINKS];
};
__device__ __forceinline__ void fx_share_row(FxShare& sh, int link, int r, const fx_acc& m) {
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    sh.v[2 * (3 * r + j)][link] = m.re[j];
    sh.v[2 * (3 * r + j) + 1][link] = m.im[j];
  }
}

// R 2^(E - 60) * scale, E folded into the scale by fx_scale
__device__ __forceinline__ double fx_value(i64 R) {
  const int h = (int)(R >> 32);
  const unsigned int l = (unsigned int)R;
  const double dh = __hiloint2double(0x43300000, h ^ (int)0x80000000) - 4503601774854144.0;  // 2^52 + 2^31
  const double dl = __hiloint2double(0x43300000, (int)l) - 4503599627370496.0;               // 2^52
  return fma(dh, 4294967296.0, dl);
}
__device__ __forceinline__ double fx_scale(double c, int E) {
  if (E > GF_FX_BAD / 2) return __longlong_as_double(0x7FF8000000000000ll);
  const int k = E - 60;
  if (k > -1000 && k < 1000) return c * __hiloint2double((k + 1023) << 20, 0);
  return scalbn(c, k);
}

// P_mu(x) <- keep * P_mu(x) + coef * c(U_mu(x) S_mu(x)) as k_force_ta. The
// rows of V U_mu^dag = (U_mu S)^dag are formed (V = S^dag, the staple sum
// by rows), and TA(M^dag) = -TA(M).
// Bound by integer multiply-add issue (IMAD.WIDE holds the issue port for
// four cycles: 81 per row product, 13 products). 24^4, conversion included:
// 4.71 ms in fp64 arithmetic, 0.70 ms here. Seven blocks per SM (80
// registers) measured 0.70 ms, six 0.73, five 0.74, eight (spills) 0.72.
__global__ void __launch_bounds__(GF_FX_THREADS, GF_FX_MINB)
    k_force_fx(FxField U, double* __restrict__ P, Geom g, double coef, double keep) {
  __shared__ FxShare sh;
  __shared__ int se[GF_FX_LINKS];
  const int t = threadIdx.x, mu = blockIdx.x & 3, V = g.vol;
  const int s0 = (blockIdx.x >> 2) * GF_FX_LINKS;
  {
    const int link = t / 3, r = t - 3 * link;
    const int s = min(s0 + link, V - 1);
    const Site st = site_of(g, s);
    const int mu_up = fx_up(g, st, mu);
    fx_acc acc = {{0, 0, 0}, {0, 0, 0}};
    int ea = -GF_FX_BAD;
#pragma unroll 1
    for (int k = 1; k < 4; ++k) fx_add_staples(acc, ea, U, g, st, s, mu, (mu + k) & 3, mu_up, r);
    // |V| <= 6: three bits down to serve as an operand
    const fx_acc m = fx_row_mul<true>(fx_operand<3>(acc), fx_mat(U, mu, s, V));
    fx_share_row(sh, link, r, m);
    if (r == 0) se[link] = ea + 3 + fx_exp(U, mu, s, V);
  }
  __syncthreads();
  const int link = t & 31, part = t >> 5, s = s0 + link;
  if (s >= V) return;
  // c of TA(M^dag): x_ij(M^dag) = conj(M_ji) - M_ij
  i64 c[3];
  int a[3];
  const int i = part == 2 ? 1 : 0, j = part == 0 ? 1 : 2;
  const int ij = 2 * (3 * i + j), ji = 2 * (3 * j + i);
  c[0] = -sh.v[ji + 1][link] - sh.v[ij + 1][link];
  c[1] = sh.v[ji][link] - sh.v[ij][link];
  a[0] = part == 0 ? 0 : (part == 1 ? 3 : 5);
  const i64 d1 = -sh.v[1][link], d2 = -sh.v[9][link], d3 = -sh.v[17][link];
  c[2] = part == 0 ? d1 - d2 : d1 + d2 - 2 * d3;
  a[1] = a[0] + 1;
  a[2] = part == 0 ? 2 : 7;
  const double sc = fx_scale(coef, se[link]);
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

static gf_field* fx_links(gf_ctx* ctx, const gf_field* U) {
  if (!ctx->w_linkfx) ctx->w_linkfx = field_new(ctx, GF_LINKFX);
  f64_to_fx(ctx, ctx->w_linkfx, U);
  return ctx->w_linkfx;
}

void wilson_force_fx(gf_ctx* ctx, const gf_field* U, gf_field* P, double coef, double keep) {
  const gf_field* F = fx_links(ctx, U);
  const int nb = 4 * blocks_for(ctx->geom.vol, GF_FX_LINKS);
  k_force_fx<<<nb, GF_FX_THREADS, 0, ctx->stream>>>(fx_view(F), (double*)P->ptr, ctx->geom, coef, keep);
  GF_CHECK_LAUNCH();
}

}  // namespace gf
