// cg.cu -- the inner iterations of the reference algorithms' CG and
// single-mass CGMS (lib/invert_cg_p.c:1-128, :130-402) without a host round
// trip per scalar: the step length, the new residual norm and the direction
// coefficient are formed by the last block of the kernel that reduces them,
// and the host reads the state once per CG_CHUNK iterations.  The four
// kernels of an iteration are programmatic dependents (pdl.cuh).
//
// What bounds it: on small lattices the latency of four dependent kernels
// (L2 round trips, the two reductions), on large ones HBM.  Reading the
// scalars on the host cost two synchronisations and two to three more
// launches per iteration (8^4 FP32 CG 11.2 -> 4.2 ms, 16^3x32 FP64 EVENODD
// 75.2 -> 44.5 ms).
#include "cg.cuh"
#include "pdl.cuh"
#include "prof.cuh"
#include "reduce.cuh"
#include <vector>

namespace qopb {

constexpr int CG_CHUNK = 32;   // iterations per host check

template <typename T>
__global__ void __launch_bounds__(RED_THREADS)
k_cg_update(c2<T> *__restrict__ x, c2<T> *__restrict__ r, const c2<T> *p, const c2<T> *Ap,
            int n, CgState *st, double *part, unsigned *count) {
  pdl_wait();
  if (st->flag) return;
  const T a = (T)st->a;
  double acc[1] = {0.0};
  for (int i = blockIdx.x * RED_THREADS + threadIdx.x; i < n; i += gridDim.x * RED_THREADS) {
    c2<T> xv = x[i], rv = r[i];
    const c2<T> pv = p[i], av = Ap[i];
    xv.x += a * pv.x; xv.y += a * pv.y;
    rv.x -= a * av.x; rv.y -= a * av.y;
    x[i] = xv;
    r[i] = rv;
    acc[0] += (double)rv.x * rv.x + (double)rv.y * rv.y;
  }
  if (grid_sum<1>(acc, part, count, &st->pn)) {
    st->oldrsq = st->rsq;
    st->rsq = st->pn;
    st->b = st->rsq / st->oldrsq;
    st->done += 1;
    if (--st->left <= 0 || st->rsq * st->fac < st->stop) st->flag = CG_EVENT;
  }
}

template <typename T>
__global__ void __launch_bounds__(RED_THREADS)
k_cg_p(c2<T> *__restrict__ p, const c2<T> *r, int n, const CgState *st) {
  pdl_wait();
  if (st->flag) return;
  const T b = (T)st->b;
  for (int i = blockIdx.x * RED_THREADS + threadIdx.x; i < n; i += gridDim.x * RED_THREADS) {
    const c2<T> u = p[i], v = r[i];
    p[i] = mk<T>(v.x + b * u.x, v.y + b * u.y);
  }
}

template <typename T>
void cg_run(LinOp<T> &L, c2<T> *x, c2<T> *r, c2<T> *p, c2<T> *Ap, int eo, bool dot, CgState &s) {
  static_assert(sizeof(CgState) <= 64 * sizeof(double), "the state travels through the reduction scratch");
  Context &c = ctx();
  const Range q = vrange(c.g, eo);
  const int n = (int)q.n, grid = red_grid(q.n);
  s.flag = CG_RUN;
  s.done = 0;
  CgState *st = (CgState *)dmalloc(sizeof(CgState));
  std::vector<int> mark;   // timing records before each iteration of a chunk
  try {
    QCHECK(cudaMemcpyAsync(st, &s, sizeof s, cudaMemcpyHostToDevice, c.s));
    while (s.flag == CG_RUN) {
      const int chunk = s.left < CG_CHUNK ? s.left : CG_CHUNK, done0 = s.done;
      mark.clear();
      for (int k = 0; k < chunk; k++) {
        mark.push_back(prof_mark());
        Dslash<T>::cg_hops(L.f, L.mass, Ap, p, eo, L.tmp, st, dot, k == 0);
        launch_k(true, k_cg_update<T>, grid, RED_THREADS, c.s, x + q.off, r + q.off, (const c2<T> *)(p + q.off),
                 (const c2<T> *)(Ap + q.off), n, st, c.d_part, c.d_count);
        launch_k(true, k_cg_p<T>, grid, RED_THREADS, c.s, p + q.off, (const c2<T> *)(r + q.off), n,
                 (const CgState *)st);
        QLAUNCHN(2);
      }
      QCHECK(cudaMemcpyAsync(c.h_res, st, sizeof s, cudaMemcpyDeviceToHost, c.s));
      sync();
      memcpy(&s, c.h_res, sizeof s);
      // drop timing records of hops that found the flag set (no work); a
      // breakdown is found by an iteration that is not counted
      const int ran = s.done - done0 + (s.flag == CG_BREAK || s.flag == CG_NAN ? 1 : 0);
      if (ran < chunk)
        for (int k = mark[ran], end = prof_mark(); k < end; k++) prof_discard(k);
    }
  } catch (...) {
    dfree(st);
    throw;
  }
  dfree(st);
}

template void cg_run<float>(LinOp<float> &, c2<float> *, c2<float> *, c2<float> *, c2<float> *, int, bool, CgState &);
template void cg_run<double>(LinOp<double> &, c2<double> *, c2<double> *, c2<double> *, c2<double> *, int, bool,
                             CgState &);

}  // namespace qopb
