// dslash.cu -- asqtad/HISQ Dslash in the handle's precision (FP64 / FP32).
// Reference: lib/asqtad_dslash_p.c:1048-1092 (eo dispatch), :1246-1279
// (style-1 hop: dest = sum_k dbllinks[k](x) src(x + shift_k)), :1019-1023
// (mass term), :1106-1138 (ddagd, ddagd_norm2), :1166-1191 (dslash_dir).
#include "reduce.cuh"
#include "dslash.cuh"
#include "dd.cuh"
#include "cg.cuh"
#include "pdl.cuh"
#include "prof.cuh"

namespace qopb {

enum HopMode {
  HOP_SET = 0,      // out = hop
  HOP_MASS = 1,     // out = mass*same + hop
  HOP_MASS_ALIAS = 2,  // out = mass*hop + hop  (reference result when out == in)
  HOP_M2_MINUS = 3  // out = mass*same - hop   (ddagd epilogue, mass = m^2)
};

// neighbour (mu, d) of site x for a hop: the input vector, or on a
// decomposed lattice the up halo when the hop leaves the block upwards.
// Returns false when the term is a down-halo product, already added to a.
template <typename T, bool DD>
__device__ __forceinline__ bool hop_input(const Geom &g, const int x[4], int mu, int d, const c2<T> *src,
                                          const DdGhost<T> &gh, c2<T> &v0, c2<T> &v1, c2<T> &v2, c2<T> *a) {
  const i64 Vh = g.Vh;
  if (DD && (gh.mask >> mu & 1) && (unsigned)(x[mu] + d) >= (unsigned)g.L[mu]) {
    const int y = x[mu] + d, fh = gh.fh[mu], fi = dd_face_index(g, x, mu);
    const int sl = dd_halo_slab(g.L[mu], y, d);
    if (y < 0) {   // slab 0: the fat product at y = -1; slab -y: the long product
      const c2<T> *G = gh.dn[mu] + (i64)(sl * 3) * fh + fi;
      a[0] = cadd<T>(a[0], G[0]); a[1] = cadd<T>(a[1], G[fh]); a[2] = cadd<T>(a[2], G[2 * fh]);
      return false;
    }
    const c2<T> *G = gh.up[mu] + (i64)(sl * 3) * fh + fi;
    v0 = G[0]; v1 = G[fh]; v2 = G[2 * fh];
    return true;
  }
  const int j = nbr_index(g, x, mu, d);
  v0 = src[j]; v1 = src[Vh + j]; v2 = src[2 * Vh + j];
  return true;
}

// threads of a hop block: SPLIT 1 one thread per site, else 32 sites with
// SPLIT warps, each holding NL / SPLIT slots of every site
__host__ __device__ constexpr int hop_threads(int split) { return split == 1 ? 128 : 32 * split; }
__host__ __device__ constexpr int hop_sites(int split) { return split == 1 ? 128 : 32; }
// resident blocks of the one-thread-per-site hops (40 registers in FP32, 56
// or 64 in FP64): what keeps the most loads in flight
template <typename T> __host__ __device__ constexpr int hop_minb(int split, bool dd, int red) {
  return split > 1 ? 1 : sizeof(T) == 4 ? 12 : dd ? 7 : red ? 9 : 8;
}

// a += (slot's link) (neighbour): the stored link row by row, or, for a
// backward slot read from the forward link of the neighbour, -U^+
template <typename T>
__device__ __forceinline__ void hop_mul(c2<T> (&a)[3], const c2<T> (&U)[9], c2<T> v0, c2<T> v1, c2<T> v2, bool back) {
#pragma unroll
  for (int r = 0; r < 3; r++) {
    c2<T> u[3];
#pragma unroll
    for (int c = 0; c < 3; c++) u[c] = back ? mk<T>(-U[3 * c + r].x, U[3 * c + r].y) : U[3 * r + c];
    cfma<T>(a[r], u[0], v0);
    cfma<T>(a[r], u[1], v1);
    cfma<T>(a[r], u[2], v2);
  }
}

// RED: 0 none, 1 = sum |out|^2, 2 = sum |same|^2, 3 = Re <same, out>; DD:
// read halos (dd.cuh).
// SPLIT > 1 (where use_split says): the slots of a site are spread over SPLIT
// warps, which load their links before they wait for the kernel ahead (links
// are never written by it: the first kernel of a dependent chain is an
// ordinary launch), so a hop costs one round trip for the links instead of
// one per slot; the partial sums meet in shared memory and are added in FP64.
// On lattices beyond L2 HBM bounds it: FP32, 24^3x48, one parity, reads
// 392 MB where 390 are compulsory, at 6.1 TB/s.
// BOTH: both parities in one launch, site blocks of the two parities next to
// each other, and every link read as a forward link: a backward slot takes
// the neighbour's forward link, which the neighbour's own block has brought
// into L2.  Blocks walk the lattice in tiles of `tile` x1 coordinates so
// that the links of the few x0 slices between the two reads stay in L2.  HBM
// bounds it, the part of the second reads that misses L2 included: FP64,
// 24^3x48 reads 971 MB where 796 are compulsory, 16x32x32x64 1624 where 1258
// are, both at 6.0-6.4 TB/s with the writes.
// st: solver state of a device-driven CG (cg.cuh) or null.
template <typename T, int NL, int MODE, int RED, bool DD = false, int SPLIT = 1, bool BOTH = false>
__global__ void __launch_bounds__(hop_threads(SPLIT), hop_minb<T>(SPLIT, DD, RED))
k_hop(c2<T> *__restrict__ out, const c2<T> *src, const c2<T> *__restrict__ lk, const c2<T> *same, T mass, Geom g,
      int p, int tile, double *part, unsigned *count, double *res, CgState *st, DdGhost<T> gh = DdGhost<T>()) {
  static_assert(!DD || (SPLIT == 1 && !BOTH), "halo reads: one thread per site, one parity");
  constexpr int NS = NL / SPLIT, SITES = hop_sites(SPLIT);
  const i64 Vh = g.Vh;
  const int w = SPLIT == 1 ? 0 : threadIdx.x >> 5, k0 = w * NS;
  int i;
  bool live;
  const c2<T> *lb = lk;   // the neighbours' parity of the links (BOTH)
  if (BOTH) {
    p = blockIdx.x & 1;
    const int b = blockIdx.x >> 1, t = SPLIT == 1 ? threadIdx.x : threadIdx.x & 31;
    const int plane = g.L[2] * g.L[3] / 2;          // sites of one parity at fixed x0, x1
    const int full = g.L[1] / tile, bpr = (tile * plane + SITES - 1) / SITES, inner = bpr * g.L[0];
    const int ti = b / inner < full ? b / inner : full;   // x1 tile; the last one may be narrower
    const int wd = ti < full ? tile : g.L[1] - full * tile, run = wd * plane;
    const int nb = (run + SITES - 1) / SITES, rem = b - ti * inner, x0 = rem / nb, o = (rem - x0 * nb) * SITES + t;
    live = o < run;
    i = live ? (x0 * g.L[1] + ti * tile) * plane + o : 0;
    out += p * 3 * Vh;
    src += (1 - p) * 3 * Vh;
    same += p * 3 * Vh;
    lb = lk + (i64)(1 - p) * NL * 9 * Vh;
    lk += (i64)p * NL * 9 * Vh;
  } else {
    i = blockIdx.x * SITES + (SPLIT == 1 ? threadIdx.x : threadIdx.x & 31);
    live = i < Vh;
  }
  int x[4];
  site_coords(g, live ? i : 0, p, x);
  c2<T> a[3] = {mk<T>(0, 0), mk<T>(0, 0), mk<T>(0, 0)};
  if constexpr (SPLIT == 1) {
    pdl_wait();
    if (st && st->flag) return;   // uniform over the grid
    if (live) {
#pragma unroll
      for (int k = 0; k < NL; k++) {
        c2<T> v0, v1, v2;
        const int mu = slot_mu<NL>(k), d = slot_disp<NL>(k);
        if (!hop_input<T, DD>(g, x, mu, d, src, gh, v0, v1, v2, a)) continue;
        if (BOTH && d < 0) {   // -U^+ with the neighbour's forward link
          const c2<T> *U = lb + (i64)(k - NL / 8) * 9 * Vh + nbr_index(g, x, mu, d);
#pragma unroll
          for (int r = 0; r < 3; r++) {
            const c2<T> u0 = U[r * Vh], u1 = U[(3 + r) * Vh], u2 = U[(6 + r) * Vh];
            cfma<T>(a[r], mk<T>(-u0.x, u0.y), v0);
            cfma<T>(a[r], mk<T>(-u1.x, u1.y), v1);
            cfma<T>(a[r], mk<T>(-u2.x, u2.y), v2);
          }
        } else {
          const c2<T> *U = lk + (i64)k * 9 * Vh + i;
#pragma unroll
          for (int r = 0; r < 3; r++) {
            cfma<T>(a[r], U[3 * r * Vh], v0);
            cfma<T>(a[r], U[(3 * r + 1) * Vh], v1);
            cfma<T>(a[r], U[(3 * r + 2) * Vh], v2);
          }
        }
      }
    }
  } else {
    c2<T> U[NS][9];
    int j[NS];
    const int lex = ((x[0] * g.L[1] + x[1]) * g.L[2] + x[2]) * g.L[3] + x[3];
#pragma unroll
    for (int s = 0; s < NS; s++) {
      const int k = k0 + s, mu = slot_mu<NL>(k), d = slot_disp<NL>(k);
      const int xm = mu == 0 ? x[0] : mu == 1 ? x[1] : mu == 2 ? x[2] : x[3];
      const int Lm = mu == 0 ? g.L[0] : mu == 1 ? g.L[1] : mu == 2 ? g.L[2] : g.L[3];
      const int sm = mu == 0 ? g.L[1] * g.L[2] * g.L[3] : mu == 1 ? g.L[2] * g.L[3] : mu == 2 ? g.L[3] : 1;
      const int y = xm + d;
      j[s] = (lex + (y >= Lm ? d - Lm : y < 0 ? d + Lm : d) * sm) >> 1;
      const c2<T> *u = BOTH && d < 0 ? lb + (i64)(k - NL / 8) * 9 * Vh + j[s] : lk + (i64)k * 9 * Vh + i;
#pragma unroll
      for (int e = 0; e < 9; e++) U[s][e] = live ? u[e * Vh] : mk<T>(0, 0);
    }
    pdl_wait();
    if (st && st->flag) return;
    if (live) {
      c2<T> v[NS][3];
#pragma unroll
      for (int s = 0; s < NS; s++)
#pragma unroll
        for (int c = 0; c < 3; c++) v[s][c] = src[c * Vh + j[s]];
#pragma unroll
      for (int s = 0; s < NS; s++)
        hop_mul<T>(a, U[s], v[s][0], v[s][1], v[s][2], BOTH && slot_disp<NL>(k0 + s) < 0);
    }
    __shared__ c2<T> sh[SPLIT - 1][3][32];
    const int t = threadIdx.x & 31;
    if (w > 0) {
#pragma unroll
      for (int r = 0; r < 3; r++) sh[w - 1][r][t] = a[r];
    }
    __syncthreads();
    live = live && w == 0;
    if (live) {
#pragma unroll
      for (int r = 0; r < 3; r++) {   // one rounding for the whole sum
        double re = a[r].x, im = a[r].y;
#pragma unroll
        for (int q = 0; q < SPLIT - 1; q++) {
          re += sh[q][r][t].x;
          im += sh[q][r][t].y;
        }
        a[r] = mk<T>((T)re, (T)im);
      }
    }
  }
  double racc[1] = {0.0};
  if (live) {
    const c2<T> a0 = a[0], a1 = a[1], a2 = a[2];
    c2<T> r0, r1, r2;
    if (MODE == HOP_SET) { r0 = a0; r1 = a1; r2 = a2; }
    else if (MODE == HOP_MASS_ALIAS) {
      r0 = mk<T>(mass * a0.x + a0.x, mass * a0.y + a0.y);
      r1 = mk<T>(mass * a1.x + a1.x, mass * a1.y + a1.y);
      r2 = mk<T>(mass * a2.x + a2.x, mass * a2.y + a2.y);
    } else {
      const c2<T> s0 = same[i], s1 = same[Vh + i], s2 = same[2 * Vh + i];
      if (MODE == HOP_MASS) {
        r0 = mk<T>(mass * s0.x + a0.x, mass * s0.y + a0.y);
        r1 = mk<T>(mass * s1.x + a1.x, mass * s1.y + a1.y);
        r2 = mk<T>(mass * s2.x + a2.x, mass * s2.y + a2.y);
      } else {
        r0 = mk<T>(mass * s0.x - a0.x, mass * s0.y - a0.y);
        r1 = mk<T>(mass * s1.x - a1.x, mass * s1.y - a1.y);
        r2 = mk<T>(mass * s2.x - a2.x, mass * s2.y - a2.y);
      }
      if (RED == 2)
        racc[0] = (double)s0.x * s0.x + (double)s0.y * s0.y + (double)s1.x * s1.x + (double)s1.y * s1.y +
                  (double)s2.x * s2.x + (double)s2.y * s2.y;
      if (RED == 3)
        racc[0] = (double)s0.x * r0.x + (double)s0.y * r0.y + (double)s1.x * r1.x + (double)s1.y * r1.y +
                  (double)s2.x * r2.x + (double)s2.y * r2.y;
    }
    out[i] = r0; out[Vh + i] = r1; out[2 * Vh + i] = r2;
    if (RED == 1)
      racc[0] = (double)r0.x * r0.x + (double)r0.y * r0.y + (double)r1.x * r1.x + (double)r1.y * r1.y +
                (double)r2.x * r2.x + (double)r2.y * r2.y;
  }
  if (RED) {
    const bool last = grid_sum<1>(racc, part, count, res);
    if (MODE == HOP_M2_MINUS && last && st) {
      // <p, A p>: |D p|^2 + m^2 |p|^2 in the working precision, or the dot product
      const double pkp = RED == 2 ? (double)((T)st->dp2 + mass * (T)*res) : *res;
      st->pkp = pkp;
      if (!(pkp - pkp == 0.0)) st->flag = CG_NAN;
      else if (pkp <= 0) st->flag = CG_BREAK;
      else st->a = st->rsq / pkp;
    }
  }
}

// one direction, weighted, accumulating (style-1 dslash_dir)
template <typename T, int NL, bool DD = false>
__global__ void k_hop_dir(c2<T> *__restrict__ out, const c2<T> *__restrict__ src, const c2<T> *__restrict__ lk,
                          int k0, int nk, T w0, T w1, Geom g, int p, DdGhost<T> gh = DdGhost<T>()) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const i64 Vh = g.Vh;
  if (i >= Vh) return;
  int x[4];
  site_coords(g, i, p, x);
  c2<T> a[3] = {out[i], out[Vh + i], out[2 * Vh + i]};
  for (int kk = 0; kk < nk; kk++) {
    const int k = k0 + kk;
    const T w = kk == 0 ? w0 : w1;
    c2<T> u0, u1, u2;
    c2<T> h[3] = {mk<T>(0, 0), mk<T>(0, 0), mk<T>(0, 0)};
    if (!hop_input<T, DD>(g, x, slot_mu<NL>(k), slot_disp<NL>(k), src, gh, u0, u1, u2, h)) {
      for (int r = 0; r < 3; r++) a[r] = cadd<T>(a[r], cscale<T>(w, h[r]));   // w (-U^+ psi)
      continue;
    }
    c2<T> v[3] = {cscale<T>(w, u0), cscale<T>(w, u1), cscale<T>(w, u2)};
    const c2<T> *U = lk + (i64)k * 9 * Vh + i;
    for (int r = 0; r < 3; r++)
      for (int c = 0; c < 3; c++) cfma<T>(a[r], U[(3 * r + c) * Vh], v[c]);
  }
  out[i] = a[0]; out[Vh + i] = a[1]; out[2 * Vh + i] = a[2];
}

template <typename T, int MODE>
struct FMass {   // out = mass*in (+ out) on a parity range
  c2<T> *out; const c2<T> *in; T mass;
  __device__ void operator()(i64 i) const {
    c2<T> v = in[i];
    if (MODE == 0) out[i] = mk<T>(mass * v.x, mass * v.y);
    else { c2<T> o = out[i]; out[i] = mk<T>(mass * v.x + o.x, mass * v.y + o.y); }
  }
};

constexpr int HOP_BLOCK = 128;

// warps that share a site's slots: 4 slots (FP32) or 2 (FP64) of links per
// thread
template <typename T> constexpr int hop_split() { return sizeof(T) == 4 ? 4 : 8; }
// Where the split pays (us per call through the C ABI, split / one thread per
// site; Vh = sites per parity).
// One parity without a reduction: FP32 always (Vh 2048 16 / 24, 32768 17 / 23,
// 80000 25 / 35, 165888 44 / 51, 221184 53 / 57, 331776 80 / 94, 1048576
// 216 / 224), FP64 up to 210000 (2048 13 / 20, 32768 20 / 22, 65536 37 / 43,
// 165888 71 / 87; 249000 105 / 106, 331776 134-194 / 144: the eight partial
// rows cost more than the latency they hide once HBM is busy).
// With a reduction the blocks of 32 sites leave four times as many partial
// sums to the last block, and the line lies lower.  Operator with norm, and
// one CG iteration: FP32 65536 70 / 106 and 66 / 96, 80000 82 / 107 and
// 78 / 99, 120960 108 / 110 and 111 / 108, 165888 144 / 119 and 144 / 117,
// 1048576 772 / 536; FP64 32768 66 / 107 and 59 / 97, 65536 97 / 114 and
// 102 / 109, 80000 117 / 119 and 120 / 115, 120960 157 / 133 and 169 / 135,
// 165888 206 / 156 and 221 / 161.
// Both parities: the neighbours' links are read through L2 as often: 10400
// 20 / 24 (FP32), 23 / 26 (FP64); 32800 26 / 25 and 37 / 34.
template <typename T> static bool use_split(i64 Vh, bool both, bool red) {
  if (both) return Vh <= 20000;
  if (red) return Vh <= (sizeof(T) == 4 ? 110000 : 75000);
  return sizeof(T) == 4 || Vh <= 210000;
}

// x1 coordinates per tile of a two-parity hop: the forward links of the four
// x0 slices of a tile that lie between the two reads of a link stay within
// 64 MB of L2 (32^3x64 FP64: 580-600 us with 32, 64 or 100 MB, 615 without
// tiles, 863 with the double-stored links in two launches)
constexpr double TILE_BYTES = 64 * 1048576.0;
template <typename T> static int hop_tile(const Geom &g, int nl) {
  const double slice = (double)g.L[2] * g.L[3] * (nl / 2) * 9 * sizeof(c2<T>);   // one x0, one x1
  const int w = (int)(TILE_BYTES / (4 * slice));
  return w >= g.L[1] ? g.L[1] : w < 4 ? 4 : w;
}

template <typename T, int NL, int MODE, int RED, int SPLIT>
static void launch_hop_s(bool pdl, c2<T> *o, const c2<T> *src, const c2<T> *lk, const c2<T> *sm, double mass, int p,
                         double *res, CgState *st, double *part, unsigned *count) {
  Context &c = ctx();
  launch_k(pdl, k_hop<T, NL, MODE, RED, false, SPLIT, false>, grid_for(c.g.Vh, hop_sites(SPLIT)), hop_threads(SPLIT),
           c.s, o, src, lk, sm, (T)mass, c.g, p, 0, part, count, res, st, DdGhost<T>());
}

// pdl: launched as a programmatic dependent of the launch ahead (pdl.cuh)
template <typename T, int MODE, int RED>
static void launch_hop(FlaT<T> *f, c2<T> *out, const c2<T> *in, const c2<T> *same, double mass, int p,
                       double *res, bool pdl = false, CgState *st = nullptr) {
  Context &c = ctx();
  const Geom &g = c.g;
  const i64 lk_par = (i64)f->nlinks * 9 * g.Vh;
  c2<T> *o = out + par_off(g, p);
  const c2<T> *src = in + par_off(g, 1 - p);
  const c2<T> *lk = f->d + p * lk_par;
  const c2<T> *sm = same ? same + par_off(g, p) : nullptr;
  // compulsory bytes: every link once, the input and output vectors once,
  // plus the same-parity input of the fused mass / m^2 epilogues
  const double bytes = (double)g.Vh * sizeof(T) * 2 *
                       (f->nlinks * 9 + 3 + 3 + ((MODE == HOP_MASS || MODE == HOP_M2_MINUS) ? 3 : 0));
  if constexpr (RED != 3) {
    if (dd_active()) {
      const int grid = grid_for(g.Vh, HOP_BLOCK);
      const DdGhost<T> gh = dd_halo<T>(f, src, 1 - p);
      ProfScope ps(sizeof(T) == 8 ? "hop_f64_dd" : "hop_f32_dd", bytes);
      if (f->nlinks == 16)
        k_hop<T, 16, MODE, RED, true><<<grid, HOP_BLOCK, 0, c.s>>>(o, src, lk, sm, (T)mass, g, p, 0, c.d_part,
                                                                   c.d_count, res, nullptr, gh);
      else
        k_hop<T, 8, MODE, RED, true><<<grid, HOP_BLOCK, 0, c.s>>>(o, src, lk, sm, (T)mass, g, p, 0, c.d_part,
                                                                  c.d_count, res, nullptr, gh);
      QLAUNCH();
      return;
    }
  }
  ProfScope ps(sizeof(T) == 8 ? "hop_f64" : "hop_f32", bytes);
  constexpr int S = hop_split<T>(), ONE = sizeof(T) == 4 && RED == 0 ? S : 1;   // without a reduction FP32 is always split
#define HOP_ARGS pdl, o, src, lk, sm, mass, p, res, st, c.d_part, c.d_count
  if (use_split<T>(g.Vh, false, RED != 0)) {
    if (f->nlinks == 16) launch_hop_s<T, 16, MODE, RED, S>(HOP_ARGS);
    else launch_hop_s<T, 8, MODE, RED, S>(HOP_ARGS);
  } else {
    if (f->nlinks == 16) launch_hop_s<T, 16, MODE, RED, ONE>(HOP_ARGS);
    else launch_hop_s<T, 8, MODE, RED, ONE>(HOP_ARGS);
  }
#undef HOP_ARGS
  QLAUNCH();
}

// both parities of out = hop(in) with the mass epilogue, one launch
template <typename T, int MODE>
static void launch_hop_both(FlaT<T> *f, c2<T> *out, const c2<T> *in, const c2<T> *same, double mass) {
  Context &c = ctx();
  const Geom &g = c.g;
  const int tile = hop_tile<T>(g, f->nlinks);
  const bool split = use_split<T>(g.Vh, true, false);
  const int sites = hop_sites(split ? 4 : 1);
  const i64 plane = g.L[2] * g.L[3] / 2, full = g.L[1] / tile, last = g.L[1] - full * tile;
  const i64 blocks = 2 * g.L[0] * (full * ((tile * plane + sites - 1) / sites) + (last * plane + sites - 1) / sites);
  // compulsory bytes: each forward link once, the input and output vectors once
  ProfScope ps(sizeof(T) == 8 ? "hop_f64_both" : "hop_f32_both",
               (double)g.V * sizeof(T) * 2 * (f->nlinks / 2 * 9 + 3 + 3));
  constexpr int S = hop_split<T>();
#define HOP_BOTH(NL, SP)                                                                    \
  k_hop<T, NL, MODE, 0, false, SP, true><<<(unsigned)blocks, hop_threads(SP), 0, c.s>>>(     \
      out, in, f->d, same, (T)mass, g, 0, tile, c.d_part, c.d_count, nullptr, nullptr)
  if (split) {
    if (f->nlinks == 16) HOP_BOTH(16, S);
    else HOP_BOTH(8, S);
  } else {
    if (f->nlinks == 16) HOP_BOTH(16, 1);
    else HOP_BOTH(8, 1);
  }
#undef HOP_BOTH
  QLAUNCH();
}

template <typename T>
void Dslash<T>::hop(FlaT<T> *f, c2<T> *out, const c2<T> *in, int p) {
  launch_hop<T, HOP_SET, 0>(f, out, in, nullptr, 0.0, p, nullptr);
}

// hop on subset eo (the reference's asqtad_hop macro); when mass_sum is set
// the reference's following mass_term(out, in, mass, out) is fused in
template <typename T>
static void hop_sub(FlaT<T> *f, c2<T> *out, const c2<T> *in, int eo, bool mass_sum, double mass) {
  const Geom &g = ctx().g;
  const bool alias = (out == in);
  if (eo == QOP_EVENODD) {
    const c2<T> *src = in;
    c2<T> *tmp = nullptr;
    if (alias) {   // the even half is overwritten before the odd half is read
      tmp = dalloc<c2<T>>(vec_elems(g));
      Blas<T>::copy(tmp, in, vrange(g, QOP_EVENODD));
      src = tmp;
    }
    if (mass_sum && !dd_active()) {
      if (alias) launch_hop_both<T, HOP_MASS_ALIAS>(f, out, src, src, mass);
      else launch_hop_both<T, HOP_MASS>(f, out, src, in, mass);
    } else
    for (int p = 0; p < 2; p++) {
      if (!mass_sum) launch_hop<T, HOP_SET, 0>(f, out, src, nullptr, 0.0, p, nullptr);
      else if (alias) launch_hop<T, HOP_MASS_ALIAS, 0>(f, out, src, nullptr, mass, p, nullptr);
      else launch_hop<T, HOP_MASS, 0>(f, out, src, in, mass, p, nullptr);
    }
    if (tmp) dfree(tmp);
    return;
  }
  const int p = eo;
  if (!mass_sum) launch_hop<T, HOP_SET, 0>(f, out, in, nullptr, 0.0, p, nullptr);
  else if (alias) launch_hop<T, HOP_MASS_ALIAS, 0>(f, out, in, nullptr, mass, p, nullptr);
  else launch_hop<T, HOP_MASS, 0>(f, out, in, in, mass, p, nullptr);
}

template <typename T>
static void mass_term(c2<T> *out, const c2<T> *in, double mass, bool sum, int eo) {
  Range r = vrange(ctx().g, eo);
  if (!sum) run_map(FMass<T, 0>{out + r.off, in + r.off, (T)mass}, r.n);
  else run_map(FMass<T, 1>{out + r.off, in + r.off, (T)mass}, r.n);
}

template <typename T>
void Dslash<T>::apply(FlaT<T> *f, double mass, c2<T> *out, const c2<T> *in, int eo_out, int eo_in) {
  if (eo_in == eo_out) {
    if (eo_out == QOP_EVENODD) hop_sub<T>(f, out, in, QOP_EVENODD, true, mass);
    else mass_term<T>(out, in, mass, false, eo_out);
    return;
  }
  if (eo_out == QOP_EVEN || eo_out == QOP_EVENODD) {
    if (eo_in == QOP_ODD) hop_sub<T>(f, out, in, QOP_EVEN, false, 0);
    else if (eo_in == QOP_EVEN) mass_term<T>(out, in, mass, false, QOP_EVEN);
    else hop_sub<T>(f, out, in, QOP_EVEN, true, mass);
  }
  if (eo_out == QOP_ODD || eo_out == QOP_EVENODD) {
    if (eo_in == QOP_EVEN) hop_sub<T>(f, out, in, QOP_ODD, false, 0);
    else if (eo_in == QOP_ODD) mass_term<T>(out, in, mass, false, QOP_ODD);
    else hop_sub<T>(f, out, in, QOP_ODD, true, mass);
  }
}

template <typename T>
void Dslash<T>::dslash_dir(FlaT<T> *f, int dir, int fb, double wtfat, double wtlong, c2<T> *out,
                           const c2<T> *in, int eo_out) {
  Context &c = ctx();
  const Geom &g = c.g;
  int k0, nk;
  if (f->nlinks == 16) { k0 = fb > 0 ? 4 * dir : 4 * dir + 2; nk = 2; }
  else { k0 = fb > 0 ? 2 * dir : 2 * dir + 1; nk = 1; }
  const c2<T> *src = in;
  c2<T> *tmp = nullptr;
  if (out == in && eo_out == QOP_EVENODD) {
    tmp = dalloc<c2<T>>(vec_elems(g));
    Blas<T>::copy(tmp, in, vrange(g, QOP_EVENODD));
    src = tmp;
  }
  const i64 lk_par = (i64)f->nlinks * 9 * g.Vh;
  for (int p = 0; p < 2; p++) {
    if (eo_out != QOP_EVENODD && eo_out != p) continue;
    int grid = grid_for(g.Vh, HOP_BLOCK);
    if (dd_active()) {
      const DdGhost<T> gh = dd_halo<T>(f, src + par_off(g, 1 - p), 1 - p);
      if (f->nlinks == 16)
        k_hop_dir<T, 16, true><<<grid, HOP_BLOCK, 0, c.s>>>(out + par_off(g, p), src + par_off(g, 1 - p),
                                                            f->d + p * lk_par, k0, nk, (T)wtfat, (T)wtlong, g, p, gh);
      else
        k_hop_dir<T, 8, true><<<grid, HOP_BLOCK, 0, c.s>>>(out + par_off(g, p), src + par_off(g, 1 - p),
                                                           f->d + p * lk_par, k0, nk, (T)wtfat, (T)wtlong, g, p, gh);
      QLAUNCH();
      continue;
    }
    if (f->nlinks == 16)
      k_hop_dir<T, 16><<<grid, HOP_BLOCK, 0, c.s>>>(out + par_off(g, p), src + par_off(g, 1 - p), f->d + p * lk_par,
                                                     k0, nk, (T)wtfat, (T)wtlong, g, p);
    else
      k_hop_dir<T, 8><<<grid, HOP_BLOCK, 0, c.s>>>(out + par_off(g, p), src + par_off(g, 1 - p), f->d + p * lk_par,
                                                    k0, nk, (T)wtfat, (T)wtlong, g, p);
    QLAUNCH();
  }
  if (tmp) dfree(tmp);
}

template <typename T>
double Dslash<T>::ddagd(FlaT<T> *f, double mass, c2<T> *out, const c2<T> *in, int eo, c2<T> *tmp, bool want_norm) {
  Context &c = ctx();
  const int p = eo, q = 1 - eo;
  const T m2 = (T)mass * (T)mass;
  if (!want_norm) {
    launch_hop<T, HOP_SET, 0>(f, tmp, in, nullptr, 0.0, q, nullptr);
    launch_hop<T, HOP_M2_MINUS, 0>(f, out, tmp, in, (double)m2, p, nullptr, true);
    return 0.0;
  }
  launch_hop<T, HOP_SET, 1>(f, tmp, in, nullptr, 0.0, q, c.d_res);
  launch_hop<T, HOP_M2_MINUS, 2>(f, out, tmp, in, (double)m2, p, c.d_res + 1, true);
  dd_allreduce(c.d_res, 2);
  QCHECK(cudaMemcpyAsync(c.h_res, c.d_res, 2 * sizeof(double), cudaMemcpyDeviceToHost, c.s));
  QCHECK(cudaStreamSynchronize(c.s));
  // the reference returns |D in|^2 + m^2 |in|^2 in the working precision
  return (double)((T)c.h_res[0] + m2 * (T)c.h_res[1]);
}

template <typename T>
void Dslash<T>::cg_hops(FlaT<T> *f, double mass, c2<T> *out, const c2<T> *in, int eo, c2<T> *tmp, CgState *st,
                        bool dot, bool first) {
  const int p = eo, q = 1 - eo;
  const T m2 = (T)mass * (T)mass;
  if (dot) {
    launch_hop<T, HOP_SET, 0>(f, tmp, in, nullptr, 0.0, q, nullptr, !first, st);
    launch_hop<T, HOP_M2_MINUS, 3>(f, out, tmp, in, (double)m2, p, &st->pn, true, st);
  } else {
    launch_hop<T, HOP_SET, 1>(f, tmp, in, nullptr, 0.0, q, &st->dp2, !first, st);
    launch_hop<T, HOP_M2_MINUS, 2>(f, out, tmp, in, (double)m2, p, &st->pn, true, st);
  }
}

template <typename T>
void Dslash<T>::ddagd_norm2_ws(FlaT<T> *f, double mass, c2<T> *out, const c2<T> *in, int eo, c2<T> *tmp_block,
                               double *part, unsigned *count, double *res) {
  Context &c = ctx();
  const Geom &g = c.g;
  const int p = eo, q = 1 - eo;
  const T m2 = (T)mass * (T)mass;
  const i64 lk_par = (i64)f->nlinks * 9 * g.Vh;
  const int grid = grid_for(g.Vh, HOP_BLOCK);
  // t = D_qp in (sum |t|^2 -> res[0]); out_p = m^2 in_p - D_pq t (sum |in_p|^2 -> res[1])
  if (f->nlinks == 16) {
    k_hop<T, 16, HOP_SET, 1><<<grid, HOP_BLOCK, 0, c.s>>>(tmp_block, in + par_off(g, p), f->d + q * lk_par, nullptr,
                                                          (T)0, g, q, 0, part, count, res, nullptr);
    k_hop<T, 16, HOP_M2_MINUS, 2><<<grid, HOP_BLOCK, 0, c.s>>>(out + par_off(g, p), tmp_block, f->d + p * lk_par,
                                                               in + par_off(g, p), m2, g, p, 0, part, count, res + 1, nullptr);
  } else {
    k_hop<T, 8, HOP_SET, 1><<<grid, HOP_BLOCK, 0, c.s>>>(tmp_block, in + par_off(g, p), f->d + q * lk_par, nullptr,
                                                         (T)0, g, q, 0, part, count, res, nullptr);
    k_hop<T, 8, HOP_M2_MINUS, 2><<<grid, HOP_BLOCK, 0, c.s>>>(out + par_off(g, p), tmp_block, f->d + p * lk_par,
                                                              in + par_off(g, p), m2, g, p, 0, part, count, res + 1, nullptr);
  }
  QLAUNCHN(2);
}

template struct Dslash<float>;
template struct Dslash<double>;

}  // namespace qopb
