// Scalar recursions of the FP64 BiCGStab solvers (solver_fp64.cu), run by the
// last block of the reduction that completes their inputs: in the operator
// sweep for alpha and omega (dslash.cu), in the residual update for beta.
#pragma once

#include "cvcb_internal.h"

namespace cvcb {

__device__ __forceinline__ double2 c_div(double2 a, double2 b) {
  // _co_eq_co_ti_co_inv (cvc_complex.h): a / b = a conj(b) / |b|^2
  const double n = b.x * b.x + b.y * b.y;
  return make_double2((a.x * b.x + a.y * b.y) / n, (a.y * b.x - a.x * b.y) / n);
}
__device__ __forceinline__ double2 c_mul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ bool finite2(double2 a) { return isfinite(a.x) && isfinite(a.y); }

// w = <r2, p2>; alpha = rho / w  (invert_Qtm.c:161-163), for the iteration
// that follows: beyond the last one it decides nothing
__device__ __forceinline__ void epi_alpha(SolverScalars *S, double re, double im) {
  S->w = make_double2(re, im);
  S->alpha = c_div(S->rho, S->w);
  if (!finite2(S->alpha) && S->iter <= S->itmax) {
    S->done = 2;
    S->niter = S->iter;
  }
}

// w = <t, s>, u = <t, t>; omega = w / u  (invert_Qtm.c:182-184).  :184 writes
// _co_eq_co_ti_re(&omega, &w, 1./u); the macro argument is not
// parenthesised, so it evaluates w.re*1./u = w.re / u.
__device__ __forceinline__ void epi_omega(SolverScalars *S, double re, double im, double u) {
  S->u = u;
  S->omega = make_double2(re / u, im / u);
  if (!finite2(S->omega)) {
    S->done = 2;
    S->niter = S->iter;
  }
}

// norm = <r1, r1>, stop if norm <= prec * normb (invert_Qtm.c:192-201); else
// w = <r2, r1>, beta = (w / rho)(alpha / omega), rho = w (:214-218)
__device__ __forceinline__ void epi_norm_beta(SolverScalars *S, double norm, double2 w) {
  S->norm = norm;
  if (norm <= S->prec * S->normb) {
    S->done = 1;
    S->niter = S->iter;
    return;
  }
  if (!isfinite(norm)) {
    S->done = 2;
    S->niter = S->iter;
    return;
  }
  S->beta = c_mul(c_div(w, S->rho), c_div(S->alpha, S->omega));
  S->rho = w;
  S->iter += 1;
  if (!finite2(S->beta)) {  // the solution still takes this iteration's step
    S->done = 2;
    S->niter = S->iter;
    S->xlast = S->iter;
  }
}

// What an operator sweep out = A in does besides: with a = <f, out> (kind 1)
// epi_alpha, with <out, f> and <out, out> (kind 2) epi_omega.
struct TmDot {
  int kind = 0;
  const double2 *f = nullptr;
  double *partials = nullptr;  // 3 per block
  unsigned *counter = nullptr;
  SolverScalars *S = nullptr;
};

}  // namespace cvcb
