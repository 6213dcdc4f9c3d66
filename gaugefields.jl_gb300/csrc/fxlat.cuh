// Device side of the fixed-point kernels: field storage, the block shape
// shared by all of them and staple chains by rows.
//
// A fixed-point link or matrix field is tiled by 32 sites: per direction and
// tile, int4 [9][32] (re.h, re.l, im.h, im.l) and the exponents int [32]. The
// elements of a matrix are then at constant distances (one address per
// matrix, immediate offsets for its nine loads) and coalesced over sites.
//
// Blocks are 96 threads = 32 links of one direction x 3 rows, thread
// t = 3 link + row: the rows of a link sit in the same warp or the next one,
// so a matrix element that all three read is one transaction.
#pragma once
#include "fixed.cuh"

namespace gf {

#ifndef GF_FX_MINB
#define GF_FX_MINB 7
#endif
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

}  // namespace gf
