// staple.cuh -- row-split FP64 staple products shared by link smearing
// (links.cu) and the fermion force (force.cu).
//
// The smearing of make_imp_links is linear in the link field it starts from.
// With S_n = staple(in; mu, n) for the three directions n != mu, every path
// of 3, 5 and 7 links and the Lepage path ends in one last staple, so
//   X_n  = c3 in + cL S_n + c5 (S_r + S_s) + c7 (staple(S_r; s) + staple(S_s; r)),
//   fat(in) = c1 in + sum_n staple(X_n; n),        {n, r, s} = the directions != mu,
// takes 12 staples per direction (18 when every path is walked by itself),
// and the adjoint of a staple with respect to `in` is the same staple.
//
// One thread owns one row of one site's result (block: 32 sites x 3 rows):
// row r of a product chain needs one row of the first factor and streams the
// others, so a thread fits in 128 registers (the cap of 5 resident blocks)
// where a thread that owns the whole 3x3 result holds 140-196, and three times
// as many threads cover the latency of the loads.  The rows of a site re-read the other factors
// from L1.  The groups (directions n) of a site block are adjacent in the
// grid, group fastest, then the parity, so the fields that the groups share
// come from HBM once.
#pragma once
#include "mat3.cuh"

namespace qopb {

// 32 sites a block and 5 resident blocks (128 registers): 24^3 x 48 HISQ
// links / force 9.4 / 27.0 ms; 96 registers (6 blocks) 9.4 / 30.7, 64 sites
// and 2 blocks 10.5 / 27.7; 64-80 registers for the one-field kernels 9.1 ms
// there but 5-10 % slower at 12^4
constexpr int ST_SITES = 32;   // sites per block; the block is (ST_SITES, 3 rows)
constexpr int ST_MINB = 5;

// a site with its lexicographic index; displacements along different
// directions add up
struct StSite {
  int p, lex, x0, x1, x2, x3;
};
__device__ __forceinline__ StSite st_site(const Geom &g, int i, int p) {
  int x[4];
  site_coords(g, i, p, x);
  return {p, ((x[0] * g.L[1] + x[1]) * g.L[2] + x[2]) * g.L[3] + x[3], x[0], x[1], x[2], x[3]};
}
// lexicographic offset of a displacement d along mu, with the wrap
__device__ __forceinline__ int st_step(const Geom &g, const StSite &s, int mu, int d) {
  const int x = mu == 0 ? s.x0 : mu == 1 ? s.x1 : mu == 2 ? s.x2 : s.x3;
  const int L = mu == 0 ? g.L[0] : mu == 1 ? g.L[1] : mu == 2 ? g.L[2] : g.L[3];
  const int str = mu == 0 ? g.L[1] * g.L[2] * g.L[3] : mu == 1 ? g.L[2] * g.L[3] : mu == 2 ? g.L[3] : 1;
  const int t = x + d;   // |d| < L
  return (t >= L ? d - L : t < 0 ? d + L : d) * str;
}
// matrix field [2][9][Vh] at (parity p, lexicographic index lex)
__device__ __forceinline__ const double2 *st_at(const double2 *f, i64 Vh, int p, int lex) {
  return f + (i64)p * 9 * Vh + (lex >> 1);
}
__device__ __forceinline__ double2 *st_at(double2 *f, i64 Vh, int p, int lex) {
  return f + (i64)p * 9 * Vh + (lex >> 1);
}

// row r of a matrix, and of its adjoint
__device__ __forceinline__ void st_row(const double2 *m, i64 Vh, int r, double2 v[3]) {
#pragma unroll
  for (int k = 0; k < 3; k++) v[k] = m[(3 * r + k) * Vh];
}
__device__ __forceinline__ void st_row_dag(const double2 *m, i64 Vh, int r, double2 v[3]) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double2 t = m[(3 * k + r) * Vh];
    v[k] = make_double2(t.x, -t.y);
  }
}
// o = x M, o += x M, o += x M^+ with M streamed from memory or held
__device__ __forceinline__ void st_mul_add(const double2 x[3], const double2 *m, i64 Vh, double2 o[3]) {
#pragma unroll
  for (int k = 0; k < 3; k++)
#pragma unroll
    for (int j = 0; j < 3; j++) cfma<double>(o[j], x[k], m[(3 * k + j) * Vh]);
}
__device__ __forceinline__ void st_mul(const double2 x[3], const double2 *m, i64 Vh, double2 o[3]) {
#pragma unroll
  for (int j = 0; j < 3; j++) o[j] = make_double2(0, 0);
  st_mul_add(x, m, Vh, o);
}
__device__ __forceinline__ void st_cfma_conj(double2 &acc, double2 a, double2 b) {   // acc += a conj(b)
  acc.x += a.x * b.x + a.y * b.y;
  acc.y += a.y * b.x - a.x * b.y;
}
__device__ __forceinline__ void st_mul_dag_add(const double2 x[3], const double2 *m, i64 Vh, double2 o[3]) {
#pragma unroll
  for (int j = 0; j < 3; j++)
#pragma unroll
    for (int k = 0; k < 3; k++) st_cfma_conj(o[j], x[k], m[(3 * j + k) * Vh]);
}
__device__ __forceinline__ void st_load(const double2 *m, i64 Vh, double2 u[9]) {
#pragma unroll
  for (int e = 0; e < 9; e++) u[e] = m[e * Vh];
}
__device__ __forceinline__ void st_mul_held(const double2 x[3], const double2 u[9], double2 o[3]) {
#pragma unroll
  for (int j = 0; j < 3; j++) {
    o[j] = make_double2(0, 0);
#pragma unroll
    for (int k = 0; k < 3; k++) cfma<double>(o[j], x[k], u[3 * k + j]);
  }
}

// row r of staple(in; mu, nu) at s, added to acc, for NF fields at once (the
// four U_nu matrices are loaded once for all of them):
//   U_nu(x) in(x+nu) U_nu(x+mu)^+ + U_nu(y)^+ in(y) U_nu(y+mu),  y = x - nu
template <int NF>
__device__ __forceinline__ void st_staple(const Geom &g, const StSite &s, const double2 *const (&in)[NF],
                                          const double2 *Unu, int mu, int nu, int r, double2 (&acc)[NF][3]) {
  const i64 Vh = g.Vh;
  const int fm = st_step(g, s, mu, 1), fn = st_step(g, s, nu, 1), bn = st_step(g, s, nu, -1);
  const int p = s.p, q = 1 - s.p;
  double2 u[3], w[9], t[3];
  st_row(st_at(Unu, Vh, p, s.lex), Vh, r, u);
  if (NF > 1) st_load(st_at(Unu, Vh, q, s.lex + fm), Vh, w);
#pragma unroll
  for (int f = 0; f < NF; f++) {
    st_mul(u, st_at(in[f], Vh, q, s.lex + fn), Vh, t);
    if (NF > 1) {
#pragma unroll
      for (int j = 0; j < 3; j++)
#pragma unroll
        for (int k = 0; k < 3; k++) st_cfma_conj(acc[f][j], t[k], w[3 * j + k]);
    } else {
      st_mul_dag_add(t, st_at(Unu, Vh, q, s.lex + fm), Vh, acc[f]);
    }
  }
  st_row_dag(st_at(Unu, Vh, q, s.lex + bn), Vh, r, u);
  if (NF > 1) st_load(st_at(Unu, Vh, p, s.lex + bn + fm), Vh, w);
#pragma unroll
  for (int f = 0; f < NF; f++) {
    st_mul(u, st_at(in[f], Vh, q, s.lex + bn), Vh, t);
    if (NF > 1) {
#pragma unroll
      for (int j = 0; j < 3; j++)
#pragma unroll
        for (int k = 0; k < 3; k++) cfma<double>(acc[f][j], t[k], w[3 * k + j]);
    } else {
      st_mul_add(t, st_at(Unu, Vh, p, s.lex + bn + fm), Vh, acc[f]);
    }
  }
}

// the j-th direction (j = 0, 1, 2) other than mu
__host__ __device__ constexpr int st_dir(int mu, int j) { return j < mu ? j : j + 1; }

// block -> (group, parity, site); false outside the lattice.  NG groups from
// g0 on
template <int NG>
__device__ __forceinline__ bool st_block(const Geom &g, int g0, int &grp, int &p, int &i) {
  const int b = blockIdx.x;
  grp = g0 + b % NG;
  p = (b / NG) & 1;
  i = (b / NG >> 1) * ST_SITES + threadIdx.x;
  return i < g.Vh;
}
inline unsigned st_grid(const Geom &g, int ngrp) {
  return (unsigned)(2 * ngrp * ((g.Vh + ST_SITES - 1) / ST_SITES));
}
inline dim3 st_threads() { return dim3(ST_SITES, 3); }

// NF fields with their three staple (or X) fields
template <int NF> struct StChain {
  const double2 *in[NF];
  double2 *S[NF][3];
  double2 *X[NF][3];
  double c3[NF];       // weight of `in` in X
};
struct StCoef {
  double cL, c5, c7;
};
struct StU {
  const double2 *d[4];
};

// work fields of F elements: `most` of them, or where that allocation fails
// `least` and per = 1 (one X_n at a time; links.cu)
double2 *st_workspace(i64 F, int most, int least, int &per);

// S_n = staple(in; mu, n)
template <int NF>
__global__ void __launch_bounds__(3 * ST_SITES, ST_MINB) k_chain_s(const __grid_constant__ StChain<NF> ch, const __grid_constant__ StU U, int mu, Geom g) {
  int grp, p, i;
  if (!st_block<3>(g, 0, grp, p, i)) return;
  const StSite s = st_site(g, i, p);
  const int r = threadIdx.y, nu = st_dir(mu, grp);
  const i64 Vh = g.Vh;
  double2 a[NF][3] = {};
  st_staple<NF>(g, s, ch.in, U.d[nu], mu, nu, r, a);
#pragma unroll
  for (int f = 0; f < NF; f++) {
    double2 *o = st_at(ch.S[f][grp], Vh, p, s.lex);
#pragma unroll
    for (int c = 0; c < 3; c++) o[(3 * r + c) * Vh] = a[f][c];
  }
}

// X_n = c3 in + cL S_n + c5 (S_r + S_s) + c7 (staple(S_r; s) + staple(S_s; r))
// for the NG directions n from the g0-th on
template <int NF, int NG>
__global__ void __launch_bounds__(3 * ST_SITES, ST_MINB) k_chain_x(const __grid_constant__ StChain<NF> ch, const __grid_constant__ StU U, StCoef co, int mu, int g0, Geom g) {
  int grp, p, i;
  if (!st_block<NG>(g, g0, grp, p, i)) return;
  const StSite s = st_site(g, i, p);
  const int r = threadIdx.y, j1 = grp == 0 ? 1 : 0, j2 = grp == 2 ? 1 : 2;
  const i64 Vh = g.Vh;
  double2 a[NF][3] = {};
  if (co.c7 != 0) {   // uniform
    const double2 *in[NF];
#pragma unroll
    for (int f = 0; f < NF; f++) in[f] = ch.S[f][j1];
    st_staple<NF>(g, s, in, U.d[st_dir(mu, j2)], mu, st_dir(mu, j2), r, a);
#pragma unroll
    for (int f = 0; f < NF; f++) in[f] = ch.S[f][j2];
    st_staple<NF>(g, s, in, U.d[st_dir(mu, j1)], mu, st_dir(mu, j1), r, a);
  }
#pragma unroll
  for (int f = 0; f < NF; f++) {
    const double2 *z = st_at(ch.in[f], Vh, p, s.lex), *sn = st_at(ch.S[f][grp], Vh, p, s.lex),
                  *s1 = st_at(ch.S[f][j1], Vh, p, s.lex), *s2 = st_at(ch.S[f][j2], Vh, p, s.lex);
    double2 *o = st_at(ch.X[f][grp], Vh, p, s.lex);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const i64 e = (3 * r + c) * Vh;
      double2 x = make_double2(co.c7 * a[f][c].x, co.c7 * a[f][c].y);
      if (co.c5 != 0) {
        const double2 d1 = s1[e], d2 = s2[e];
        x.x += co.c5 * (d1.x + d2.x);
        x.y += co.c5 * (d1.y + d2.y);
      }
      if (co.cL != 0) {
        const double2 b = sn[e];
        x.x += co.cL * b.x;
        x.y += co.cL * b.y;
      }
      if (ch.c3[f] != 0) {
        const double2 v = z[e];
        x.x += ch.c3[f] * v.x;
        x.y += ch.c3[f] * v.y;
      }
      o[e] = x;
    }
  }
}

// row r of c1 in + w sum_n staple(Y_n; n), without the n whose Y is null
__device__ __forceinline__ void st_fat_row(const Geom &g, const StSite &s, const double2 *in,
                                           const double2 *const (&Y)[3], const StU &U, double c1, double w, int mu,
                                           int r, double2 (&a)[1][3]) {
  const i64 Vh = g.Vh;
#pragma unroll 1
  for (int j = 0; j < 3; j++) {
    if (!Y[j]) continue;   // uniform
    const double2 *const y[1] = {Y[j]};
    st_staple<1>(g, s, y, U.d[st_dir(mu, j)], mu, st_dir(mu, j), r, a);
  }
  const double2 *z = st_at(in, Vh, s.p, s.lex);
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const double2 v = z[(3 * r + c) * Vh];
    a[0][c] = make_double2(c1 * v.x + w * a[0][c].x, c1 * v.y + w * a[0][c].y);
  }
}

}  // namespace qopb
