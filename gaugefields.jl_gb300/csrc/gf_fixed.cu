// Fixed-point (block floating, integer pipes) kernels of the fp64-class path:
// conversions, the plaquette sum and the Wilson force.
#include "gf_internal.h"
#include <algorithm>
#include "fxrows64.cuh"
#include "stencil.cuh"

namespace gf {

// LINK64 / MAT64 (double2) or double-float pairs (float4) -> fixed point, one
// link per thread; bandwidth-bound (24^4: 57 us for 387 MB).
template <typename E>
__global__ void __launch_bounds__(128) k_to_fx(const E* __restrict__ in, char* __restrict__ out, int V) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x, mu = blockIdx.y;
  if (s >= V) return;
  const E* b = in + (size_t)mu * 9 * V + s;
  double m[18];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const double2 v = fx_complex64(__ldg(b + (size_t)k * V));
    m[2 * k] = v.x;
    m[2 * k + 1] = v.y;
  }
  int4 f[9];
  bool few;
  const int e = fx_from_f64(m, f, few);
  char* o = out + fx_offset(mu, s, V);
#pragma unroll
  for (int k = 0; k < 9; ++k) *reinterpret_cast<int4*>(o + 512 * k) = f[k];
  *reinterpret_cast<int*>(o + 9 * 512 - 12 * (s & 31)) = e;
  if (few) fx_regrade(in, out, mu, s, V, e);
}

void to_fx(gf_ctx* ctx, gf_field* dst, const gf_field* src) {
  const int V = ctx->geom.vol;
  dim3 grid(blocks_for(V, 128), 4);
  if (src->kind == GF_LINKDF || src->kind == GF_MATDF)
    k_to_fx<<<grid, 128, 0, ctx->stream>>>((const float4*)src->ptr, (char*)dst->ptr, V);
  else
    k_to_fx<<<grid, 128, 0, ctx->stream>>>((const double2*)src->ptr, (char*)dst->ptr, V);
  GF_CHECK_LAUNCH();
}

__global__ void __launch_bounds__(128) k_fx_to_f64(FxField F, double2* __restrict__ out, int V) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x, mu = blockIdx.y;
  if (s >= V) return;
  const FxMat M = fx_mat(F, mu, s, V);
  const int e = fx_exp(F, mu, s, V);
  double2* b = out + (size_t)mu * 9 * V + s;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int4 v = M(k);
    b[(size_t)k * V] = e == GF_FX_F64 ? make_double2(fx_unpack64(v.x, v.y), fx_unpack64(v.z, v.w))
                                      : make_double2(fx_to_f64(fx_join(v.x, v.y), e), fx_to_f64(fx_join(v.z, v.w), e));
  }
}

void fx_to_f64_field(gf_ctx* ctx, gf_field* dst, const gf_field* src) {
  const int V = ctx->geom.vol;
  dim3 grid(blocks_for(V, 128), 4);
  k_fx_to_f64<<<grid, 128, 0, ctx->stream>>>(fx_view(src), (double2*)dst->ptr, V);
  GF_CHECK_LAUNCH();
}

// Sum over the sites and the planes mu < nu of Re tr P_munu, one partial per
// block. A work item is one plane of 32 sites; a thread forms row r of
// U_mu(x) U_nu(x+mu) U_mu(x+nu)^dag and its product with row r of U_nu(x).
// Integer-issue-bound: 2M sites (32^3 x 64) 7.16 ms in fp64, 1.68 ms here with
// the conversion (0.4 ms, bandwidth-bound); 8^4 89 -> 25.6 us, the launches of
// the conversion and the sum and one wait.
// Links with an fp64 slot: the same row in fp64.
__device__ __noinline__ double plaquette_row64(const FxField U, int mu, int nu, int s, int xpm, int xpn, int r, int V) {
  row64 a = mul64<false>(load_row64<false>(fx_mat64(U, mu, s, V), r), fx_mat64(U, nu, xpm, V));
  a = mul64<true>(a, fx_mat64(U, mu, xpn, V));
  const row64 b = load_row64<false>(fx_mat64(U, nu, s, V), r);
  double v = 0.0;
#pragma unroll
  for (int k = 0; k < 3; ++k) v = fma(a.re[k], b.re[k], fma(a.im[k], b.im[k], v));
  return v;
}
__global__ void __launch_bounds__(GF_FX_THREADS, GF_FX_MINB)
    k_plaquette_fx(FxField U, const __grid_constant__ Geom g, int items, SumOut to) {
  const int t = threadIdx.x, V = g.vol;
  const int link = t / 3, r = t - 3 * link;
  double v = 0.0;
#pragma unroll 1
  for (int it = blockIdx.x; it < items; it += gridDim.x) {
    const int tile = it / 6, p = it - 6 * tile;
    const int mu = p < 3 ? 0 : (p < 5 ? 1 : 2), nu = p < 3 ? p + 1 : (p < 5 ? p - 1 : 3);
    const int s = tile * GF_FX_LINKS + link;
    if (s >= V) continue;
    const Site st = site_of(g, s);
    const int xpm = eo_of_lex(g, st.lex + fx_up(g, st, mu), st.par ^ 1);
    const int xpn = eo_of_lex(g, st.lex + fx_up(g, st, nu), st.par ^ 1);
    const int e = fx_exp(U, mu, s, V) + fx_exp(U, nu, xpm, V) + fx_exp(U, mu, xpn, V) + fx_exp(U, nu, s, V);
    if (fx_has_f64(e)) {
      v += plaquette_row64(U, mu, nu, s, xpm, xpn, r, V);
      continue;
    }
    fx_acc a = fx_row_mul<false>(fx_load_row<false>(fx_mat(U, mu, s, V), r), fx_mat(U, nu, xpm, V));
    a = fx_row_mul<true>(fx_operand<0>(a), fx_mat(U, mu, xpn, V));
    const fx_row b = fx_load_row<false>(fx_mat(U, nu, s, V), r);
    fx_sum d = fx_zero_sum();
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      fx_mac(d, fx_pre(a.re[k]), fx_num{b.ah[k], b.al[k]});
      fx_mac(d, fx_pre(a.im[k]), fx_num{b.bh[k], b.bl[k]});
    }
    v = fma(fx_value(fx_get(d)), fx_unit(1.0, e), v);
  }
  block_sum(v, to);
}

void plaquette_start_fx(gf_ctx* ctx, const gf_field* F, int slot) {
  const int items = 6 * blocks_for(ctx->geom.vol, GF_FX_LINKS);
  // a few waves of resident blocks, so that the second stage stays short
  const int nb = std::min(std::min(items, ctx->sm_count * GF_FX_MINB * 8), ctx->partial_cap);
  const SumOut to = sum_out(ctx, nb, GF_FX_THREADS, slot);
  k_plaquette_fx<<<nb, GF_FX_THREADS, 0, ctx->stream>>>(fx_view(F), ctx->geom, items, to);
  GF_CHECK_LAUNCH();
  sum_finish(ctx, to, nb, slot);
}

// P_mu(x) <- keep * P_mu(x) + coef * c(U_mu(x) S_mu(x)) as k_force_ta. The
// rows of V U_mu^dag = (U_mu S)^dag are formed (V = S^dag, the staple sum
// by rows), and TA(M^dag) = -TA(M).
// Bound by integer multiply-add issue (IMAD.WIDE holds the issue port for
// four cycles: 81 per row product, 13 products). 24^4, conversion included:
// 4.71 ms in fp64 arithmetic, 0.71 ms here. Seven blocks per SM (80
// registers) measured 0.71 ms, six 0.75; before links could be graded 0.70,
// 0.73, five 0.74, eight (spills) 0.72.
// Links with an fp64 slot among their staples: force_rows64, in the block's
// first 96 threads.
__device__ __noinline__ void force_rows64(const FxField U, double* P, const Geom& g, int mu, int s0, double coef,
                                          double keep, FxRaw& sh, const int* se) {
  const int t = threadIdx.x, link = t / 3, r = t - 3 * link, V = g.vol;
  __syncthreads();  // sh has been read
  if (t < GF_FX_THREADS && fx_has_f64(se[link])) {
    const int s = min(s0 + link, V - 1);
    share64(sh64(sh, link), r, mul64<true>(staple_row64(U, g, site_of(g, s), s, mu, r), fx_mat64(U, mu, s, V)));
  }
  __syncthreads();
  if (t < GF_FX_THREADS) update_mom64(sh64(sh, t & 31), se, P, mu, s0, V, coef, keep);
}
template <int AXES, int MINB>
__global__ void __launch_bounds__(GF_FX_THREADS * AXES, MINB)
    k_force_fx(FxField U, double* __restrict__ P, const __grid_constant__ Geom g, double coef, double keep) {
  __shared__ FxRaw sh;
  __shared__ FxAxes<AXES> ax;
  __shared__ int se[GF_FX_LINKS];
  const int axis = AXES > 1 ? threadIdx.x / GF_FX_THREADS : 0, t = threadIdx.x - axis * GF_FX_THREADS;
  const int mu = blockIdx.x & 3, V = g.vol, s0 = (blockIdx.x >> 2) * GF_FX_LINKS;
  bool f64 = false;
  {
    const int link = t / 3, r = t - 3 * link;
    const int s = min(s0 + link, V - 1);
    const Site st = site_of(g, s);
    int ea;
    const fx_acc acc = fx_staple_row<AXES>(ax, U, g, st, s, mu, axis, link, r, ea);
    if (axis == 0) {
      // |V| <= 6: three bits down to serve as an operand
      fx_share(sh, link, r, fx_row_mul<true>(fx_operand<3>(acc), fx_mat(U, mu, s, V)));
      const int e = ea + 3 + fx_exp(U, mu, s, V);
      if (r == 0) se[link] = e;
      f64 = fx_has_f64(e);
    }
  }
  const bool any64 = __syncthreads_or(f64);
  if (axis == 0) fx_update_mom(sh, se, P, mu, s0, V, -coef, keep);
  if (any64) force_rows64(U, P, g, mu, s0, -coef, keep, sh, se);
}

gf_field* fx_links(gf_ctx* ctx, const gf_field* U, bool for_stack) {
  // the context's own stream is not given out, so only a caller's is captured
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (!ctx->own_stream) GF_CUDA(cudaStreamIsCapturing(ctx->stream, &capture));
  if (capture != cudaStreamCaptureStatusNone) {
    // A graph may be replayed on any stream and beside any call, so a call that
    // needs no state of the context captures none: the fp64 kernels read the
    // links in place. The context's stacks are such state in any case, and
    // nothing can be allocated here; their copy is kept from then on.
    if (!for_stack || !ctx->w_linkfx) return nullptr;
    ctx->fx_graph = 1;
  }
  if (!ctx->w_linkfx) {
    try {
      ctx->w_linkfx = field_new(ctx, GF_LINKFX);
    } catch (const gf_error& e) {
      if (e.code != GF_ENOMEM) throw;
      return nullptr;
    }
  }
  to_fx(ctx, ctx->w_linkfx, U);
  return ctx->w_linkfx;
}

void wilson_force_fx(gf_ctx* ctx, const gf_field* F, gf_field* P, double coef, double keep) {
  const int nb = 4 * blocks_for(ctx->geom.vol, GF_FX_LINKS);
  const int axes = ctx->geom.vol <= GF_FX_SPLIT_MAX ? 3 : 1;
  auto kern = axes == 3 ? k_force_fx<3, 2>
                        : (ctx->geom.vol <= GF_FX_FEW_MAX ? k_force_fx<1, GF_FX_FEW_MINB> : k_force_fx<1, GF_FX_MINB>);
  kern<<<nb, axes * GF_FX_THREADS, 0, ctx->stream>>>(fx_view(F), (double*)P->ptr, ctx->geom, coef, keep);
  GF_CHECK_LAUNCH();
}

}  // namespace gf
