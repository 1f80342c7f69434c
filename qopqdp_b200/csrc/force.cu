// force.cu -- asqtad fermion force on the device.
// Reference: lib/asqtad_force_p.c:16-64 (QOP_asqtad_force / _multi),
// lib/asqtad_force_fnmat_p.c:4-43 (outer products of the sources, scale -1),
// :491-513 (sign flip on odd sites), :516-546 (force += -2 antiherm(U deriv^+)).
//
// deriv_mu is the derivative of
//   E(U) = Re sum_{x,mu} tr[ midF_mu(x)^+ fat_mu(x) + midN_mu(x)^+ long_mu(x) ]
// with (fat, long) = make_imp_links(U), in the convention
// dE = Re sum tr[deriv^+ dU].  It is formed by reverse-mode differentiation
// of the staple sums of make_imp_links (links.cu): for every staple
// application out += c staple(in; mu, nu) the adjoint kernels add the
// contributions to the adjoint of `in` and of U_nu, in the reverse order of
// the forward sums (7-staples, 5-staples, Lepage, 3-staples, one-link), and
// the Naik products add theirs.  Every adjoint kernel is written in gather
// form (each thread owns one output site and reads its neighbours), so no
// atomics are needed and results are deterministic.  Everything runs in
// FP64; the result is rounded once into the force handle's precision.
#include "fields.cuh"
#include "staple.cuh"
#include <vector>

namespace qopb {
namespace {

__device__ __forceinline__ void site_of(const Geom &g, i64 s, int &p, int &i, int x[4]) {
  p = (int)(s / g.Vh);
  i = (int)(s % g.Vh);
  site_coords(g, i, p, x);
}
__device__ __forceinline__ void nbr_pi(const Geom &g, const int x[4], int mu, int d, int &p, int &i) {
  int y[4];
  shifted(g, x, mu, d, y);
  par_idx(g, y, p, i);
}
__device__ __forceinline__ M3 ldf(const double2 *f, const Geom &g, int p, int i) { return ld3(fptr(f, g, p, i), g.Vh); }
__device__ __forceinline__ void accf(double2 *f, const Geom &g, int p, int i, const M3 &m, double c) {
  double2 *b = f + (i64)p * 9 * g.Vh + i;
#pragma unroll
  for (int e = 0; e < 9; e++) {
    double2 v = b[e * g.Vh];
    b[e * g.Vh] = make_double2(v.x + c * m.e[e].x, v.y + c * m.e[e].y);
  }
}

// adjoint of U_n for out += sum_k w_k staple(in_k; mu, n), with G_k the
// adjoint of out: row r of the sum over the pairs (G, in) of
//   G(z) U(z+mu) in(z+n)^+ + G(z-mu)^+ U(z-mu) in(z-mu+n)
//   + in(z-mu)^+ U(z-mu) G(z-mu+n) + in(z) U(z+mu) G(z+n)^+,   U = U_n;
// each of the two U matrices is loaded once for all pairs
constexpr int ADJ_PAIRS = 4;
struct AdjPairs {
  const double2 *G[ADJ_PAIRS], *in[ADJ_PAIRS];
  double w[ADJ_PAIRS];
};
__device__ __forceinline__ void adj_link_row(const Geom &g, const StSite &s, const AdjPairs &pr, int np,
                                             const double2 *Un, int mu, int n, int r, double2 (&acc)[3]) {
  const i64 Vh = g.Vh;
  const int fm = st_step(g, s, mu, 1), bm = st_step(g, s, mu, -1), fn = st_step(g, s, n, 1);
  const int p = s.p, q = 1 - p;
  double2 u[9], x[3], t[3];
  st_load(st_at(Un, Vh, q, s.lex + fm), Vh, u);
#pragma unroll 1
  for (int k = 0; k < np; k++) {
    const double2 *const a[2] = {pr.G[k], pr.in[k]};
    const double w = pr.w[k];
#pragma unroll
    for (int h = 0; h < 2; h++) {   // row of a[h](z) U a[1-h](z+n)^+
      st_row(st_at(a[h], Vh, p, s.lex), Vh, r, x);
#pragma unroll
      for (int c = 0; c < 3; c++) x[c] = make_double2(w * x[c].x, w * x[c].y);
      st_mul_held(x, u, t);
      st_mul_dag_add(t, st_at(a[1 - h], Vh, q, s.lex + fn), Vh, acc);
    }
  }
  st_load(st_at(Un, Vh, q, s.lex + bm), Vh, u);
#pragma unroll 1
  for (int k = 0; k < np; k++) {
    const double2 *const a[2] = {pr.G[k], pr.in[k]};
    const double w = pr.w[k];
#pragma unroll
    for (int h = 0; h < 2; h++) {   // row of a[h](z-mu)^+ U a[1-h](z-mu+n)
      st_row_dag(st_at(a[h], Vh, q, s.lex + bm), Vh, r, x);
#pragma unroll
      for (int c = 0; c < 3; c++) x[c] = make_double2(w * x[c].x, w * x[c].y);
      st_mul_held(x, u, t);
      st_mul_add(t, st_at(a[1 - h], Vh, p, s.lex + bm + fn), Vh, acc);
    }
  }
}

// The derivative for one direction mu from its chains (staple.cuh): groups
// 0-2 add the adjoint of U_n, n != mu, to D_n; group 3 adds the adjoint of
// the starting link, c1 M + w sum_n staple(Y_n; n), to D_mu; NG groups from
// the g0-th on
struct SweepArgs {
  AdjPairs pr[3];
  int np;
  const double2 *M, *Y[3];
  double2 *D[4];
  double c1, w;
};
template <int NG>
__global__ void __launch_bounds__(3 * ST_SITES, ST_MINB) k_sweep(const __grid_constant__ SweepArgs a, const __grid_constant__ StU U, int mu, int g0, Geom g) {
  int grp, p, i;
  if (!st_block<NG>(g, g0, grp, p, i)) return;
  const StSite s = st_site(g, i, p);
  const int r = threadIdx.y;
  const i64 Vh = g.Vh;
  double2 acc[1][3] = {};
  int dir = mu;
  if (grp < 3) {
    dir = st_dir(mu, grp);
    adj_link_row(g, s, a.pr[grp], a.np, U.d[dir], mu, dir, r, acc[0]);
  } else {
    st_fat_row(g, s, a.M, a.Y, U, a.c1, a.w, mu, r, acc);
  }
  double2 *o = st_at(a.D[dir], Vh, p, s.lex);
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const double2 v = o[(3 * r + c) * Vh];
    o[(3 * r + c) * Vh] = make_double2(v.x + acc[0][c].x, v.y + acc[0][c].y);
  }
}

// adjoint of long(x) = c U(x) U(x+mu) U(x+2mu), NG directions from mu0 on as groups:
// D(z) += c [N(z) (U(z+mu) U(z+2mu))^+ + U(z-mu)^+ N(z-mu) U(z+mu)^+ + (U(z-2mu) U(z-mu))^+ N(z-2mu)]
struct NaikAdjArgs {
  double2 *D[4];
  const double2 *N[4];
};
template <int NG>
__global__ void __launch_bounds__(3 * ST_SITES, ST_MINB) k_adj_naik(const __grid_constant__ NaikAdjArgs a, const __grid_constant__ StU Us, double c, int mu0, Geom g) {
  int mu, p, i;
  if (!st_block<NG>(g, mu0, mu, p, i)) return;
  const StSite s = st_site(g, i, p);
  const int r = threadIdx.y, q = 1 - p;
  const i64 Vh = g.Vh;
  const double2 *U = Us.d[mu], *N = a.N[mu];
  const int f1 = st_step(g, s, mu, 1), f2 = st_step(g, s, mu, 2), b1 = st_step(g, s, mu, -1),
            b2 = st_step(g, s, mu, -2);
  double2 x[3], t[3], o[3] = {};
  st_row(st_at(N, Vh, p, s.lex), Vh, r, x);
#pragma unroll
  for (int j = 0; j < 3; j++) t[j] = make_double2(0, 0);
  st_mul_dag_add(x, st_at(U, Vh, p, s.lex + f2), Vh, t);
  st_row_dag(st_at(U, Vh, q, s.lex + b1), Vh, r, x);
  st_mul_add(x, st_at(N, Vh, q, s.lex + b1), Vh, t);   // the first two terms share the last factor
  st_mul_dag_add(t, st_at(U, Vh, q, s.lex + f1), Vh, o);
#pragma unroll
  for (int j = 0; j < 3; j++) t[j] = make_double2(0, 0);
  st_mul_dag_add(x, st_at(U, Vh, p, s.lex + b2), Vh, t);
  st_mul_add(t, st_at(N, Vh, p, s.lex + b2), Vh, o);
  double2 *d = st_at(a.D[mu], Vh, p, s.lex);
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const double2 v = d[(3 * r + j) * Vh];
    d[(3 * r + j) * Vh] = make_double2(v.x + c * o[j].x, v.y + c * o[j].y);
  }
}

// The reference's derivative field carries, with a Lepage term, one more
// term of the form U_mu H, H Hermitian (lib/asqtad_force_fnmat_p.c:316-340):
//   D_mu(x) -= cL [F_mu(x) U_mu(x) - U_mu(x) F_mu(x+mu)],
//   F_mu = sum_{nu != mu} H_nu,  H_nu = A_nu + A_nu^+,
//   A_nu(x) = M_nu(x) U_nu(x)^+ - M_nu(x-nu)^+ U_nu(x-nu).
// The force projection TA(U D^+) removes it; the filtered U(3) adjoint of
// the HISQ force, which receives this field at the W level, does not.
// k_lep_h: H = H_nu for one nu
__global__ void k_lep_h(double2 *H, const double2 *M, const double2 *Unu, int nu, Geom g) {
  const i64 s = blockIdx.x * (i64)blockDim.x + threadIdx.x;
  if (s >= 2 * g.Vh) return;
  int p, i, z[4], pm, im;
  site_of(g, s, p, i, z);
  nbr_pi(g, z, nu, -1, pm, im);
  const M3 a = mul_na(ldf(M, g, p, i), ldf(Unu, g, p, i));
  const M3 b = mul_an(ldf(M, g, pm, im), ldf(Unu, g, pm, im));
  M3 h;
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const double2 x = a.e[3 * r + c], y = b.e[3 * r + c], xt = a.e[3 * c + r], yt = b.e[3 * c + r];
      h.e[3 * r + c] = make_double2(x.x - y.x + xt.x - yt.x, x.y - y.y - xt.y + yt.y);
    }
  st3(H + (i64)p * 9 * g.Vh + i, g.Vh, h);
}

// k_lep_fix: D_mu -= cL [F U_mu - U_mu F(x+mu)] with F the sum of the three
// H_nu (nu != mu) given in h0..h2
__global__ void k_lep_fix(double2 *D, const double2 *Umu, const double2 *h0, const double2 *h1, const double2 *h2,
                          int mu, double cL, Geom g) {
  const i64 s = blockIdx.x * (i64)blockDim.x + threadIdx.x;
  if (s >= 2 * g.Vh) return;
  int p, i, z[4], pp, ip;
  site_of(g, s, p, i, z);
  nbr_pi(g, z, mu, 1, pp, ip);
  M3 f0 = ldf(h0, g, p, i), f1 = ldf(h0, g, pp, ip);
  const M3 a0 = ldf(h1, g, p, i), a1 = ldf(h1, g, pp, ip), b0 = ldf(h2, g, p, i), b1 = ldf(h2, g, pp, ip);
#pragma unroll
  for (int e = 0; e < 9; e++) {
    f0.e[e] = make_double2(f0.e[e].x + a0.e[e].x + b0.e[e].x, f0.e[e].y + a0.e[e].y + b0.e[e].y);
    f1.e[e] = make_double2(f1.e[e].x + a1.e[e].x + b1.e[e].x, f1.e[e].y + a1.e[e].y + b1.e[e].y);
  }
  const M3 U = ldf(Umu, g, p, i);
  M3 r = mul(f0, U);
  const M3 t = mul(U, f1);
#pragma unroll
  for (int e = 0; e < 9; e++) r.e[e] = make_double2(r.e[e].x - t.e[e].x, r.e[e].y - t.e[e].y);
  accf(D, g, p, i, r, -cL);
}

__global__ void k_field_axpby(double2 *d, double a, const double2 *s, double b, i64 n) {   // d = a d + b s
  const i64 k = blockIdx.x * (i64)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const double2 x = d[k], y = s[k];
  d[k] = make_double2(a * x.x + b * y.x, a * x.y + b * y.y);
}

// midF_mu(x) = sgn(x) sum_i eps_i x_i(x) x_i(x+mu)^+ (midN: x+3mu) with
// sgn = even_sign on even and -even_sign on odd sites (asqtad: -1, HISQ: +1);
// vectors are [parity][colour][site]; directions mu0 .. mu1 - 1, the fields
// from mu0 on; midF or midN may be null
template <typename T>
__global__ void k_force_mid(double2 *midF, double2 *midN, const c2<T> *const *xs, const double *eps, int nsrc,
                            double even_sign, int mu0, int mu1, Geom g) {
  const i64 s = blockIdx.x * (i64)blockDim.x + threadIdx.x;
  if (s >= 2 * g.Vh) return;
  int p, i, x[4];
  site_of(g, s, p, i, x);
  const double sgn = p ? -even_sign : even_sign;
  const i64 Vh = g.Vh;
  for (int mu = mu0; mu < mu1; mu++) {
    for (int k = 0; k < 2; k++) {
      double2 *out = k == 0 ? midF : midN;
      if (!out) continue;
      int q, j;
      nbr_pi(g, x, mu, k == 0 ? 1 : 3, q, j);
      M3 m;
#pragma unroll
      for (int e = 0; e < 9; e++) m.e[e] = make_double2(0, 0);
      for (int n = 0; n < nsrc; n++) {
        const c2<T> *v = xs[n];
        const double w = sgn * eps[n];
        double2 a[3], b[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const c2<T> va = v[((i64)p * 3 + c) * Vh + i], vb = v[((i64)q * 3 + c) * Vh + j];
          a[c] = make_double2((double)va.x, (double)va.y);
          b[c] = make_double2((double)vb.x, (double)vb.y);
        }
#pragma unroll
        for (int r = 0; r < 3; r++)
#pragma unroll
          for (int c = 0; c < 3; c++) {   // a_r conj(b_c)
            m.e[3 * r + c].x += w * (a[r].x * b[c].x + a[r].y * b[c].y);
            m.e[3 * r + c].y += w * (a[r].y * b[c].x - a[r].x * b[c].y);
          }
      }
      st3(out + (i64)(mu - mu0) * 18 * Vh + (i64)p * 9 * Vh + i, Vh, m);
    }
  }
}

// F_mu(x) = TA(F_mu(x)): the projection the reference's ASVEC algorithm
// applies to the whole accumulated force (lib/asqtad_force_asvec_p.c:403-408)
template <typename T>
__global__ void k_force_ta_self(c2<T> *F, Geom g) {
  const i64 s = blockIdx.x * (i64)blockDim.x + threadIdx.x;
  if (s >= 8 * g.Vh) return;           // [4 mu][2 parities][Vh]
  const i64 Vh = g.Vh;
  const i64 off = (s / Vh) * 9 * Vh + s % Vh;
  double2 a[9];
#pragma unroll
  for (int e = 0; e < 9; e++) {
    const c2<T> v = F[off + (i64)e * Vh];
    a[e] = make_double2((double)v.x, (double)v.y);
  }
  double tri = 0;
#pragma unroll
  for (int k = 0; k < 3; k++) tri += a[4 * k].y;
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const double2 x = a[3 * r + c], y = a[3 * c + r];
      double re = 0.5 * (x.x - y.x), im = 0.5 * (x.y + y.y);
      if (r == c) im -= tri / 3.0;
      c2<T> &f = F[off + (i64)(3 * r + c) * Vh];
      f.x = (T)re;
      f.y = (T)im;
    }
}

// F_mu(x) += fac TA(U_mu(x) D_mu(x)^+), TA = traceless anti-Hermitian part
template <typename T>
__global__ void k_force_ta(c2<T> *F, const double2 *U, const double2 *D, double fac, Geom g) {
  const i64 s = blockIdx.x * (i64)blockDim.x + threadIdx.x;
  if (s >= 8 * g.Vh) return;           // [4 mu][2 parities][Vh]
  const i64 Vh = g.Vh;
  const i64 pm = s / Vh, i = s % Vh;   // pm = mu * 2 + parity
  const i64 off = pm * 9 * Vh + i;
  const M3 a = mul_na(ld3(U + off, Vh), ld3(D + off, Vh));
  double tri = 0;   // Im tr(a - a^+) / 2 = Im tr a
#pragma unroll
  for (int k = 0; k < 3; k++) tri += a.e[4 * k].y;
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const double2 x = a.e[3 * r + c], y = a.e[3 * c + r];
      double re = 0.5 * (x.x - y.x), im = 0.5 * (x.y + y.y);
      if (r == c) im -= tri / 3.0;
      c2<T> &f = F[off + (i64)(3 * r + c) * Vh];
      f.x = (T)((double)f.x + fac * re);
      f.y = (T)((double)f.y + fac * im);
    }
}

// adjoint of the U(3) projection W = V f(Q), Q = V^+V, f(q) = q^-1/2:
// GV = GW f + V (B + B^+),  B = Z [(Z^+ V^+ GW Z) o Gamma] Z^+,
// Gamma_ij = (f(w_i) - f(w_j)) / (w_i - w_j) = -1 / (s_i s_j (s_i + s_j)), s = sqrt(w).
// Force filter (lib/hisq_reunit_utilities_p.c:463-481): where the smallest
// eigenvalue of Q is below ff, the derivative is the one of V (Q + ff)^-1/2.
__global__ void k_reunit_adj(double2 *GV, const double2 *V, const double2 *GW, i64 n4, double ff) {
  const i64 s = blockIdx.x * (i64)blockDim.x + threadIdx.x;   // over [4 mu][2 parities][Vh]
  if (s >= n4) return;
  const i64 Vh = n4 / 8, blk = s / Vh, i = s % Vh, off = blk * 9 * Vh + i;
  const M3 v = ld3(V + off, Vh), gw = ld3(GW + off, Vh);
  M3 Z;
  double w[3], sq[3];
  herm_eig3(mul_an(v, v), w, Z);
  if (ff > 0 && fmin(w[0], fmin(w[1], w[2])) < ff) {
#pragma unroll
    for (int k = 0; k < 3; k++) w[k] += ff;
  }
#pragma unroll
  for (int k = 0; k < 3; k++) sq[k] = sqrt(w[k]);
  M3 f;
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 3; b++) {
      double2 acc = make_double2(0, 0);
#pragma unroll
      for (int k = 0; k < 3; k++) {   // Z_ak conj(Z_bk) / s_k
        const double2 za = Z.e[3 * a + k], zb = Z.e[3 * b + k];
        acc.x += (za.x * zb.x + za.y * zb.y) / sq[k];
        acc.y += (za.y * zb.x - za.x * zb.y) / sq[k];
      }
      f.e[3 * a + b] = acc;
    }
  M3 At = mul(mul_an(Z, mul_an(v, gw)), Z);
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 3; b++) {
      const double gm = -1.0 / (sq[a] * sq[b] * (sq[a] + sq[b]));
      At.e[3 * a + b] = make_double2(gm * At.e[3 * a + b].x, gm * At.e[3 * a + b].y);
    }
  const M3 B = mul_na(mul(Z, At), Z);
  M3 t;
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 3; b++)
      t.e[3 * a + b] = make_double2(B.e[3 * a + b].x + B.e[3 * b + a].x, B.e[3 * a + b].y - B.e[3 * b + a].y);
  M3 r = mul(gw, f);
  const M3 u = mul(v, t);
#pragma unroll
  for (int e = 0; e < 9; e++) r.e[e] = make_double2(r.e[e].x + u.e[e].x, r.e[e].y + u.e[e].y);
  st3(GV + off, Vh, r);
}

// D += derivative of Re sum tr[midF^+ fat + midN^+ long] with (fat, long) =
// make_imp_links(c, U): the reverse sweep over its staple sums and the Naik
// products; midN may be null.  The adjoint of a staple with respect to its
// input is the same staple, so for every direction mu the chains of staple.cuh
// run on U_mu (S_n, I_n = X_n with c3 = 0) and on M = midF_mu (A_n, X_n), and
//   D_mu += c1 M + sum_n staple(X_n; n),
//   D_n  += AL(M, I_n) + AL(X_n, U_mu) + c7 [AL(A_s, S_r) + AL(A_r, S_s)],
// AL(G, in) the link adjoint (adj_link_row), {n, r, s} the directions != mu:
// 12 link adjoints, 6 + 6 + 6 + 3 staples in three launches per direction.
// Three launches and about 52 field passes per direction where walking every
// path took 64 launches and about 300; 24^3 x 48, HISQ, 8 sources: the call
// takes 27.0 ms against 62.1 (8^4 asqtad, 2 sources: 0.17 against 1.68).
// The sweep kernel runs the FP64 pipe at 43 % and L1 at 51 % of their rates;
// the latency of L2 reads at 15 warps per SM is the rest.
constexpr int SWEEP_FIELDS = 12, SWEEP_LEAN = 7;   // work fields [2][9][Vh]
// staple applications and field sums of the sweep walked path by path: the
// unit of the flops that the force calls report
int sweep_terms(const double c[6], bool naik, bool lepage_rep) {
  const bool have5 = c[2] != 0 || c[3] != 0, have3 = c[1] != 0 || have5 || c[4] != 0;
  const int per_nu = 4 + (c[4] != 0 ? 2 : 0) + (have5 ? 2 * (4 + (c[3] != 0 ? 2 : 0)) : 0);
  return 4 * (1 + (have3 ? 3 * per_nu : 0)) + (naik && c[5] != 0 ? 4 : 0) + (lepage_rep && c[4] != 0 ? 8 : 0);
}

// The contributions of direction mu, M = midF_mu.  nx = 3: work holds
// SWEEP_FIELDS fields; nx = 1: SWEEP_LEAN (S_n, A_n and one field that takes
// I_n and then X_n of one n after the other), with twelve more launches.
void sweep_dir(const StU &Us, const double c[6], int mu, const double2 *M, double2 *D, double2 *work, int nx) {
  Context &cx = ctx();
  const Geom &g = cx.g;
  const cudaStream_t st = cx.s;
  const i64 F1 = 18 * g.Vh;
  const double c1 = c[0] - 6 * c[4], c3 = c[1], c5 = c[2], c7 = c[3], cL = c[4];
  const bool have5 = c5 != 0 || c7 != 0 || cL != 0, have3 = c3 != 0 || have5;
  if (!have3) {
    k_field_axpby<<<grid_for(F1, 256), 256, 0, st>>>(D + mu * F1, 1.0, M, c1, F1);
    QLAUNCH();
    return;
  }
  const double2 *const Umu = Us.d[mu];
  SweepArgs a{};
  for (int d = 0; d < 4; d++) a.D[d] = D + d * F1;
  a.M = M;
  a.c1 = c1;
  if (!have5) {   // three-link staples only: X_n = c3 M
    a.np = 1;
    a.w = c3;
    for (int j = 0; j < 3; j++) {
      a.pr[j] = AdjPairs{{M}, {Umu}, {c3}};
      a.Y[j] = M;
    }
    k_sweep<4><<<st_grid(g, 4), st_threads(), 0, st>>>(a, Us, mu, 0, g);
    QLAUNCH();
    return;
  }
  const StCoef co{cL, c5, c7};
  a.w = 1.0;
  StChain<2> ch;
  ch.in[0] = Umu;
  ch.in[1] = M;
  ch.c3[0] = 0;
  ch.c3[1] = c3;
  for (int f = 0; f < 2; f++)
    for (int j = 0; j < 3; j++) {
      ch.S[f][j] = work + ((nx == 3 ? 6 : 3) * f + j) * F1;
      ch.X[f][j] = work + (nx == 3 ? 6 * f + 3 + j : 6) * F1;
    }
  k_chain_s<2><<<st_grid(g, 3), st_threads(), 0, st>>>(ch, Us, mu, g);
  QLAUNCH();
  // r, s: the other two of the three directions
  auto r_of = [](int j) { return j == 0 ? 1 : 0; };
  auto s_of = [](int j) { return j == 2 ? 1 : 2; };
  if (nx == 3) {
    k_chain_x<2, 3><<<st_grid(g, 3), st_threads(), 0, st>>>(ch, Us, co, mu, 0, g);
    a.np = c7 != 0 ? 4 : 2;
    for (int j = 0; j < 3; j++) {
      a.pr[j] = AdjPairs{{M, ch.X[1][j], ch.S[1][s_of(j)], ch.S[1][r_of(j)]},
                         {ch.X[0][j], Umu, ch.S[0][r_of(j)], ch.S[0][s_of(j)]},
                         {1.0, 1.0, c7, c7}};
      a.Y[j] = ch.X[1][j];
    }
    k_sweep<4><<<st_grid(g, 4), st_threads(), 0, st>>>(a, Us, mu, 0, g);
    QLAUNCHN(2);
    return;
  }
  for (int j = 0; j < 3; j++) {
    double2 *X = ch.X[0][j];
    for (int f = 0; f < 2; f++) {   // X = I_n, then X_n
      StChain<1> one;
      one.in[0] = ch.in[f];
      one.c3[0] = ch.c3[f];
      for (int k = 0; k < 3; k++) {
        one.S[0][k] = ch.S[f][k];
        one.X[0][k] = X;
      }
      k_chain_x<1, 1><<<st_grid(g, 1), st_threads(), 0, st>>>(one, Us, co, mu, j, g);
      if (f == 0) {
        a.np = c7 != 0 ? 3 : 1;
        a.pr[j] = AdjPairs{{M, ch.S[1][s_of(j)], ch.S[1][r_of(j)]}, {X, ch.S[0][r_of(j)], ch.S[0][s_of(j)]}, {1.0, c7, c7}};
      } else {
        a.np = 1;
        a.pr[j] = AdjPairs{{X}, {Umu}, {1.0}};
        for (int k = 0; k < 3; k++) a.Y[k] = k == j ? X : nullptr;
        a.c1 = j == 0 ? c1 : 0.0;
        k_sweep<1><<<st_grid(g, 1), st_threads(), 0, st>>>(a, Us, mu, 3, g);
        QLAUNCH();
      }
      k_sweep<1><<<st_grid(g, 1), st_threads(), 0, st>>>(a, Us, mu, j, g);
      QLAUNCHN(2);
    }
  }
}

// lepage_rep adds the reference's Lepage term of the form U H (k_lep_h), for a
// derivative that feeds something other than the force projection.  work:
// SWEEP_FIELDS fields.  Returns sweep_terms.
int smear_adjoint(const double2 *U, const double c[6], const double2 *mid, const double2 *midN, double2 *D,
                  double2 *work, bool lepage_rep = false) {
  Context &cx = ctx();
  const Geom &g = cx.g;
  const i64 F1 = 18 * g.Vh;
  const int grid2 = grid_for(2 * g.Vh, 128);
  const double cL = c[4];
  auto Uf = [&](int d) { return U + d * F1; };
  auto Df = [&](int d) { return D + d * F1; };
  const StU Us{{Uf(0), Uf(1), Uf(2), Uf(3)}};
  for (int mu = 0; mu < 4; mu++) sweep_dir(Us, c, mu, mid + mu * F1, D, work, 3);
  if (midN && c[5] != 0) {
    k_adj_naik<4><<<st_grid(g, 4), st_threads(), 0, cx.s>>>(
        NaikAdjArgs{{Df(0), Df(1), Df(2), Df(3)}, {midN, midN + F1, midN + 2 * F1, midN + 3 * F1}}, Us, c[5], 0, g);
    QLAUNCH();
  }
  if (lepage_rep && cL != 0) {
    double2 *H[4] = {work, work + F1, work + 2 * F1, work + 3 * F1};   // free once the sweep is done
    for (int nu = 0; nu < 4; nu++) k_lep_h<<<grid2, 128, 0, cx.s>>>(H[nu], mid + nu * F1, Uf(nu), nu, g);
    for (int mu = 0; mu < 4; mu++) {
      const double2 *o[3];
      for (int nu = 0, k = 0; nu < 4; nu++)
        if (nu != mu) o[k++] = H[nu];
      k_lep_fix<<<grid2, 128, 0, cx.s>>>(Df(mu), Uf(mu), o[0], o[1], o[2], mu, cL, g);
    }
    QLAUNCHN(8);
  }
  return sweep_terms(c, midN != nullptr, lepage_rep);
}

// a device allocation freed at the end of its scope
template <typename E> struct Buf {
  E *p = nullptr;
  Buf() = default;
  explicit Buf(i64 n) : p(dalloc<E>(n)) {}
  Buf(const Buf &) = delete;
  Buf &operator=(const Buf &) = delete;
  ~Buf() { dfree((void *)p); }
  operator E *() const { return p; }
};

// the sources of a force call on the device
template <typename T> struct ForceSources {
  Buf<const c2<T> *> x;
  Buf<double> w;
  int n;
  ForceSources(VecT<T> *const *v, const double *weight, int n_) : x(n_), w(n_), n(n_) {
    std::vector<const c2<T> *> hx(n);
    for (int k = 0; k < n; k++) hx[k] = v[k]->d;
    QCHECK(cudaMemcpyAsync(x, hx.data(), sizeof(void *) * n, cudaMemcpyHostToDevice, ctx().s));
    QCHECK(cudaMemcpyAsync(w, weight, sizeof(double) * n, cudaMemcpyHostToDevice, ctx().s));
  }
  // their outer products along the directions mu0 .. mu1 - 1
  void mids(double2 *midF, double2 *midN, double even_sign, int mu0 = 0, int mu1 = 4) const {
    const Geom &g = ctx().g;
    k_force_mid<T><<<grid_for(2 * g.Vh, 128), 128, 0, ctx().s>>>(midF, midN, x, w, n, even_sign, mu0, mu1, g);
    QLAUNCH();
  }
};

// a gauge field in FP64: the field itself, or a copy freed at the end of the scope
struct Gauge64 {
  double2 *p;
  bool own = false;
  template <typename T> explicit Gauge64(GaugeT<T> *G) { p = gauge_fp64(G, own); }
  Gauge64(const Gauge64 &) = delete;
  Gauge64 &operator=(const Gauge64 &) = delete;
  ~Gauge64() {
    if (own) dfree(p);
  }
  operator double2 *() const { return p; }
};

}  // namespace

// Scratch: D and, where they fit, every outer product (4 fields, 8 with the
// Naik term) and the sweep's 12; otherwise one direction's outer product at a
// time and SWEEP_LEAN, 12 fields in all, so that every lattice on which a walk
// over single paths fits (4 work fields: 12, or 16 with the Naik term) is
// still taken.
template <typename T>
void asqtad_force(QOP_info_t *info, GaugeT<T> *G, GaugeT<T> *F, const QOP_asqtad_coeffs_t *cf, const double *eps,
                  VecT<T> *const *x, int nsrc) {
  Context &c = ctx();
  const Geom &g = c.g;
  const double t0 = wtime();
  const i64 Vh = g.Vh, F1 = 18 * Vh, F4 = 72 * Vh;
  const Gauge64 U(G);
  const bool naik = cf->naik != 0;
  const double co[6] = {cf->one_link, cf->three_staple, cf->five_staple, cf->seven_staple, cf->lepage, cf->naik};
  const ForceSources<T> src(x, eps, nsrc);
  Buf<double2> D(F4), w;
  dzero(D, sizeof(double2) * F4);
  const i64 nmid = naik ? 8 : 4;
  int nx = 3;
  w.p = st_workspace(F1, (int)nmid + SWEEP_FIELDS, 1 + SWEEP_LEAN, nx);
  if (nx == 3) {
    double2 *mid = w, *midN = naik ? mid + F4 : nullptr;
    src.mids(mid, midN, -1.0);   // scale -1 (fnmat_p.c:497)
    smear_adjoint(U, co, mid, midN, D, w + nmid * F1);
  } else {
    const StU Us{{U, U + F1, U + 2 * F1, U + 3 * F1}};
    for (int mu = 0; mu < 4; mu++) {
      src.mids(w, nullptr, -1.0, mu, mu + 1);
      sweep_dir(Us, co, mu, w, D, w + F1, nx);
      if (!naik) continue;
      src.mids(nullptr, w, -1.0, mu, mu + 1);
      NaikAdjArgs a{};
      a.D[mu] = D + mu * F1;
      a.N[mu] = w;
      k_adj_naik<1><<<st_grid(g, 1), st_threads(), 0, c.s>>>(a, Us, co[5], mu, g);
      QLAUNCH();
    }
  }
  // the reference's algorithm choice (lib/asqtad_force_p.c:22): FNMAT adds
  // -2 TA(U D^+); ASVEC (fewer sources than fnmat_src_min) stores
  // TA(force + C) with TA(C) = -TA(U D^+), half the FNMAT term
  const bool asvec = nsrc < c.opt.force_fnmat_src_min;
  if (asvec) {
    k_force_ta_self<T><<<grid_for(8 * Vh, 128), 128, 0, c.s>>>(F->d, g);
    QLAUNCH();
  }
  k_force_ta<T><<<grid_for(8 * Vh, 128), 128, 0, c.s>>>(F->d, U, D, asvec ? -1.0 : -2.0, g);
  QLAUNCH();
  sync();
  if (info) {
    info->final_sec = wtime() - t0;
    // outer products, adjoint staples (~4 matrix products each) and projection
    info->final_flop = (double)g.V * (4.0 * (naik ? 2 : 1) * 72 * nsrc + sweep_terms(co, naik, false) * 216.0 + 4 * 264);
    info->status = QOP_SUCCESS;
  }
}

// Scratch: 24 fields.  The W level holds the outer products (8), the adjoint
// of W (4) and the sweep's 12; the U level sweeps in the first 12, with the
// adjoint of V and the derivative in the other 12.
template <typename T>
void hisq_force(QOP_info_t *info, HisqT<T> *h, GaugeT<T> *F, const QOP_hisq_coeffs_t *cf, const double *res,
                VecT<T> *const *x, const int *n_orders) {
  Context &c = ctx();
  const Geom &g = c.g;
  const double t0 = wtime();
  if (!h->U || !h->V || !h->W)
    fail(QOP_FAIL, "hisq_force: the HISQ links carry no auxiliary U/V/W fields "
                   "(create them with QOP_hisq_links_set_opts want_aux = 1)");
  const i64 Vh = g.Vh, F1 = 18 * Vh, F4 = 72 * Vh;
  static_assert(SWEEP_FIELDS == 12, "the two halves of the scratch trade places");
  const Gauge64 U(h->U), V(h->V), W(h->W);
  Buf<double2> mid(SWEEP_FIELDS * F1), w(SWEEP_FIELDS * F1);
  double2 *GW = mid + 2 * F4, *GV = w, *D = w + F4;
  dzero(GW, sizeof(double2) * F4);
  int nterms = 0;
  for (int k = 0; k < cf->n_naiks; k++) nterms += n_orders[k];
  const double ca[6] = {cf->asqtad_one_link, cf->asqtad_three_staple, cf->asqtad_five_staple,
                        cf->asqtad_seven_staple, cf->asqtad_lepage, cf->asqtad_naik};
  const double cd[6] = {cf->difference_one_link, 0, 0, 0, 0, cf->difference_naik};
  int nk = 0, shift = 0;
  for (int k = 0; k < cf->n_naiks; k++) {
    // group 0 takes every source with the asqtad coefficients, group k >= 1
    // its own sources with the difference coefficients (fnmat2_p.c:52-113),
    // its eps_naik folded into the weights (the derivative is linear in them)
    const int first = k == 0 ? 0 : shift, count = k == 0 ? nterms : n_orders[k];
    shift += n_orders[k];
    if (count == 0) continue;
    std::vector<double> wt(res + first, res + first + count);
    if (k > 0)
      for (double &v : wt) v *= cf->eps_naik[k];
    const ForceSources<T> src(x + first, wt.data(), count);
    src.mids(mid, mid + F4, 1.0);
    nk += smear_adjoint(W, k == 0 ? ca : cd, mid, mid + F4, GW, w, true);
  }
  k_reunit_adj<<<grid_for(8 * Vh, 128), 128, 0, c.s>>>(GV, V, GW, 8 * Vh, c.opt.hisq_force_filter);
  QLAUNCH();
  const double c7[6] = {cf->fat7_one_link, cf->fat7_three_staple, cf->fat7_five_staple, cf->fat7_seven_staple,
                        c.opt.use_fat7_lepage ? cf->fat7_lepage : 0.0, 0.0};
  dzero(D, sizeof(double2) * F4);
  nk += smear_adjoint(U, c7, GV, nullptr, D, mid);
  k_force_ta<T><<<grid_for(8 * Vh, 128), 128, 0, c.s>>>(F->d, U, D, 2.0, g);   // deriv = 2 D
  QLAUNCH();
  sync();
  if (info) {
    info->final_sec = wtime() - t0;
    info->final_flop = (double)g.V * (8.0 * 72 * nterms + nk * 216.0 + 4 * 1500 + 4 * 264);
    info->status = QOP_SUCCESS;
  }
}

template void asqtad_force<float>(QOP_info_t *, GaugeT<float> *, GaugeT<float> *, const QOP_asqtad_coeffs_t *,
                                  const double *, VecT<float> *const *, int);
template void asqtad_force<double>(QOP_info_t *, GaugeT<double> *, GaugeT<double> *, const QOP_asqtad_coeffs_t *,
                                   const double *, VecT<double> *const *, int);
template void hisq_force<float>(QOP_info_t *, HisqT<float> *, GaugeT<float> *, const QOP_hisq_coeffs_t *,
                                const double *, VecT<float> *const *, const int *);
template void hisq_force<double>(QOP_info_t *, HisqT<double> *, GaugeT<double> *, const QOP_hisq_coeffs_t *,
                                 const double *, VecT<double> *const *, const int *);

}  // namespace qopb
