// Scalars and stopping decisions of the CGs whose loop graph runs on the device
// (solver_full.cu, staggered.cu): the loop of conjugate_gradient.h:66-104, which goes on while
// |r|^2 >= target.  A sum that is not finite ends the solve as a breakdown, as in the even-odd
// CG (dslash_f64.cu).
#pragma once

#include "kernels.h"

namespace hw {

__device__ __forceinline__ void cg_decide(CgState *st) {
    if (!(st->rr >= st->target_rr))
        st->status = CG_CONVERGED;
    else if (st->iter >= st->maxiter)
        st->status = CG_MAXITER;
    else
        st->status = CG_RUNNING;
}

// |r|^2 and |b|^2 of the initial guess
__device__ __forceinline__ void cg_start(CgState *st, double rr, double bb, double acc2, int maxiter) {
    st->rr = rr;
    st->src_norm2 = bb;
    st->target_rr = acc2 * bb;
    st->iter = 0;
    st->maxiter = maxiter;
    st->alpha = st->beta = 0.0;
    st->do_pupdate = 0;
    st->bodies = 0;
    if (!isfinite(rr) || !isfinite(bb))
        st->status = CG_BREAKDOWN;
    else if (bb == 0.0)
        st->status = CG_CONVERGED;
    else
        cg_decide(st);
}

// |M p|^2 -> alpha
__device__ __forceinline__ void cg_alpha(CgState *st, double pAp) {
    st->pAp = pAp;
    if (!(pAp > 0.0) || !isfinite(pAp))
        st->status = CG_BREAKDOWN, st->do_pupdate = 0;
    else
        st->alpha = st->rr / pAp;
}

// |r|^2 after the step -> beta
__device__ __forceinline__ void cg_step(CgState *st, double rr) {
    st->iter += 1;
    if (!isfinite(rr)) {
        st->status = CG_BREAKDOWN, st->do_pupdate = 0;
        return;
    }
    st->beta = rr / st->rr;
    st->rr = rr;
    st->do_pupdate = 1;
    cg_decide(st);
}

}  // namespace hw
