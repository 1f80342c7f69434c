// cg.cuh -- iterations of the reference algorithms' CG with the scalars on the
// device (cg.cu).
#pragma once
#include "qopb.h"
#include "solvers.cuh"

namespace qopb {

// CG_EVENT: the driver has something to decide (iterations used up, residual
// target reached); CG_BREAK: <p, A p> <= 0; CG_NAN: <p, A p> not finite
enum { CG_RUN = 0, CG_EVENT = 1, CG_BREAK = 2, CG_NAN = 3 };
struct CgState {
  double rsq, oldrsq, pkp, a, b;   // |r|^2, the one before, <p, A p>, step length, direction coefficient
  double dp2, pn;                  // sums of the two hops
  double fac, stop;                // event when rsq * fac < stop
  int left, done, flag, pad;       // iterations until an event, and run
};

// Runs x += a p, r -= a A p, p = r + b p from p, r and s.rsq until the state's
// flag is set, with the arithmetic of the drivers' own loops; p is not
// updated in the last iteration.  dot: step length from <p, A p>, else from
// |D p|^2 + m^2 |p|^2.
template <typename T>
void cg_run(LinOp<T> &L, c2<T> *x, c2<T> *r, c2<T> *p, c2<T> *Ap, int eo, bool dot, CgState &s);

// the driver may use cg_run: one process, and no output per iteration wanted
inline bool cg_on_device(int eo) {
  return eo != QOP_EVENODD && !dd_active() && ctx().verbosity < QOP_VERB_HI;
}

}  // namespace qopb
