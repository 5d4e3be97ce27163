// FP64 BiCGStab solvers with the reference's algorithm, update order and
// stopping rule: invert_Qtm (BiCGStab on Q, invert_Qtm.c:86-270) and
// invert_Qtm_her (BiCGStab on Qf5(mu) Qf5(-mu) with right-hand side g5 phi,
// then x = Qf5(-mu) y, invert_Qtm.c:276-478).
//
// The recursion scalars live on the device (SolverScalars): the last block of
// each reduction computes alpha, omega, beta and the convergence flag
// (bicgstab.cuh; alpha and omega in the operator sweeps themselves), and
// every later kernel of the iteration reads them from HBM.  An iteration thus
// costs no host round trip; the host checks the flag once per chunk of
// iterations.  Once the flag is set, all remaining kernels of the chunk
// return immediately, so the state is exactly that of the iteration at which
// the reference would have left its loop.
#include <algorithm>
#include <cmath>

#include "bicgstab.cuh"
#include "cvcb_internal.h"
#include "reduce.cuh"

namespace cvcb {

namespace {

// s = r1 - alpha p2   (invert_Qtm.c:171-176)
__global__ void k_s_update(double2 *__restrict__ s, const double2 *__restrict__ r1,
                           const double2 *__restrict__ p2, const SolverScalars *__restrict__ S,
                           size_t n) {
  if (S->done) return;
  const double2 al = S->alpha;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
       k += (size_t)gridDim.x * blockDim.x) {
    const double2 q = c_mul(__ldg(p2 + k), al);
    const double2 r = __ldg(r1 + k);
    s[k] = make_double2(r.x - q.x, r.y - q.y);
  }
}

// r1 = s - omega t; norm = <r1, r1>, w = <r2, r1>  (invert_Qtm.c:192-216)
struct RedR1Beta {
  double2 *r1;
  const double2 *s, *t, *r2;
  const SolverScalars *S;
  __device__ void operator()(size_t k, double (&acc)[3]) const {
    const double2 q = c_mul(__ldg(t + k), S->omega);
    const double2 a = __ldg(s + k), u = __ldg(r2 + k);
    const double2 r = make_double2(a.x - q.x, a.y - q.y);
    r1[k] = r;
    acc[0] += r.x * r.x + r.y * r.y;
    acc[1] += u.x * r.x + u.y * r.y;
    acc[2] += u.x * r.y - u.y * r.x;
  }
};
struct EpiNormBeta {
  SolverScalars *S;
  __device__ void operator()(const double (&t)[3]) const {
    epi_norm_beta(S, t[0], make_double2(t[1], t[2]));
  }
};

// x += omega s + alpha p (invert_Qtm.c:204-211) and p = r1 + beta (p - omega
// p2) (:224-231) of iteration `iter`.  Skipped once converged: the reference
// leaves the loop before the update of x; a beta that is not finite still
// lets x take its step.
__global__ void k_xp_update(double2 *__restrict__ x, double2 *__restrict__ p,
                            const double2 *__restrict__ s, const double2 *__restrict__ r1,
                            const double2 *__restrict__ p2, const SolverScalars *__restrict__ S,
                            int iter, size_t n) {
  if (S->done && S->xlast != iter) return;
  const bool go = !S->done;
  const double2 al = S->alpha, om = S->omega, be = S->beta;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
       k += (size_t)gridDim.x * blockDim.x) {
    const double2 pv = p[k];
    double2 xv = x[k];
    const double2 a = c_mul(__ldg(s + k), om);
    xv.x += a.x; xv.y += a.y;
    const double2 b = c_mul(pv, al);
    xv.x += b.x; xv.y += b.y;
    x[k] = xv;
    if (!go) continue;
    const double2 q = c_mul(__ldg(p2 + k), om);
    const double2 d = make_double2(pv.x - q.x, pv.y - q.y);
    const double2 e = c_mul(d, be);
    const double2 r = __ldg(r1 + k);
    p[k] = make_double2(r.x + e.x, r.y + e.y);
  }
}

// y = a - b
__global__ void k_sub(double2 *__restrict__ y, const double2 *__restrict__ a,
                      const double2 *__restrict__ b, size_t n) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
       k += (size_t)gridDim.x * blockDim.x) {
    const double2 u = __ldg(a + k), v = __ldg(b + k);
    y[k] = make_double2(u.x - v.x, u.y - v.y);
  }
}

struct RedNorm {
  const double2 *a;
  __device__ void operator()(size_t k, double (&acc)[1]) const {
    const double2 u = __ldg(a + k);
    acc[0] += u.x * u.x + u.y * u.y;
  }
};

struct EpiNormb {
  SolverScalars *S;
  __device__ void operator()(const double (&t)[1]) const { S->normb = t[0]; }
};
struct EpiStart {
  SolverScalars *S;
  __device__ void operator()(const double (&t)[1]) const {
    S->norm = t[0];
    S->rho = make_double2(t[0], 0.0);  // <r2, r1> with r1 = r2 = p
    if (S->norm <= S->prec * S->normb) { S->done = 3; S->niter = 0; }
  }
};

int elem_blocks(size_t n) {
  size_t b = (n + 255) / 256;
  return (int)(b > 4096 ? 4096 : b);
}

}  // namespace

// The operator of each solver on device-layout FP64 fields.
static int apply_op(cvcb_lattice *L, bool her, double2 *out, const double2 *in, double2 *aux,
                    const int *done, const TmDot *dot = nullptr) {
  const double a = 0.5 / L->kappa;
  if (!her) return launch_tm_full(L, out, in, a, L->mu, -0.5, false, done, dot);
  CVCB_TRY(launch_tm_full(L, aux, in, a, -L->mu, -0.5, true, done));    // Qf5(aux, in, -mu)
  return launch_tm_full(L, out, aux, a, L->mu, -0.5, true, done, dot);  // Qf5(out, aux, +mu)
}

int invert_bicgstab(cvcb_lattice *L, bool her, double *xi, const double *phi, double prec,
                    int niter_max, double *true_res2) {
  const Geom &g = L->g;
  const size_t n = (size_t)g.V * 12;
  const size_t fb = n * sizeof(double2);
  void *base;
  CVCB_TRY(ensure_buffer(L, SLOT_F2, 10 * fb + (size_t)tm_full_blocks(g) * 3 * sizeof(double), &base));
  double2 *F = static_cast<double2 *>(base);
  double2 *x = F, *rhs = F + n, *r1 = F + 2 * n, *r2 = F + 3 * n, *s = F + 4 * n,
          *t = F + 5 * n, *p = F + 6 * n, *p2 = F + 7 * n, *aux = F + 8 * n, *phid = F + 9 * n;
  SolverScalars *S = L->scal;
  const int eb = elem_blocks(n);
  double *part = reinterpret_cast<double *>(F + 10 * n);
  // alpha from <r2, p2> with the sweep that writes p2, omega from <t, s> and
  // <t, t> with the one that writes t
  const TmDot dot_alpha{1, r2, part, L->red_counter, S}, dot_omega{2, s, part, L->red_counter, S};

  CVCB_TRY(spinor_in(L, phid, phi, g.V));
  CVCB_TRY(spinor_in(L, x, xi, g.V));

  SolverScalars h{};
  h.prec = prec;
  h.itmax = niter_max;
  h.xlast = -1;
  CVCB_CUDA(cudaMemcpyAsync(S, &h, sizeof h, cudaMemcpyHostToDevice, L->stream));

  // normb = <phi, phi>  (invert_Qtm.c:129 / :329)
  CVCB_TRY(launch_reduce<1>(L, RedNorm{phid}, EpiNormb{S}, n));
  if (her) {
    CVCB_CUDA(cudaMemcpyAsync(rhs, phid, fb, cudaMemcpyDeviceToDevice, L->stream));
    CVCB_TRY(launch_g5(L, rhs, g.V));
  } else {
    rhs = phid;
  }
  // p = rhs - A x ; norm = <p,p>
  CVCB_TRY(apply_op(L, her, p, x, aux, nullptr));
  k_sub<<<eb, 256, 0, L->stream>>>(p, rhs, p, n);
  CVCB_LAUNCHED(L);
  CVCB_TRY(launch_reduce<1>(L, RedNorm{p}, EpiStart{S}, n));
  SolverScalars hs;
  CVCB_CUDA(cudaMemcpyAsync(&hs, S, sizeof hs, cudaMemcpyDeviceToHost, L->stream));
  CVCB_CUDA(cudaStreamSynchronize(L->stream));
  if (hs.done == 3) {
    // start guess already solves: the reference returns 0 and leaves xi as
    // it was (invert_Qtm.c:144-147, :344-347).
    if (true_res2) *true_res2 = hs.norm / hs.normb;
    return 0;
  }

  CVCB_CUDA(cudaMemcpyAsync(r1, p, fb, cudaMemcpyDeviceToDevice, L->stream));
  CVCB_CUDA(cudaMemcpyAsync(r2, p, fb, cudaMemcpyDeviceToDevice, L->stream));
  CVCB_TRY(apply_op(L, her, p2, p, aux, nullptr, &dot_alpha));

  const int *done = &S->done;
  const int chunk = 16;
  int launched = 0;
  for (;;) {
    const int todo = std::min(chunk, niter_max + 1 - launched);
    for (int it = 0; it < todo; ++it) {
      k_s_update<<<eb, 256, 0, L->stream>>>(s, r1, p2, S, n);
      CVCB_LAUNCHED(L);
      CVCB_TRY(apply_op(L, her, t, s, aux, done, &dot_omega));
      CVCB_TRY(launch_reduce<3>(L, RedR1Beta{r1, s, t, r2, S}, EpiNormBeta{S}, n, done));
      k_xp_update<<<eb, 256, 0, L->stream>>>(x, p, s, r1, p2, S, launched + it + 1, n);
      CVCB_LAUNCHED(L);
      CVCB_TRY(apply_op(L, her, p2, p, aux, done, &dot_alpha));
    }
    launched += todo;
    CVCB_CUDA(cudaMemcpyAsync(&hs, S, sizeof hs, cudaMemcpyDeviceToHost, L->stream));
    CVCB_CUDA(cudaStreamSynchronize(L->stream));
    if (hs.done || launched > niter_max) break;
  }
  const int niter = hs.done == 1 ? hs.niter : niter_max + 1;
  const bool converged = hs.done == 1 && niter <= niter_max;

  if (her) {
    // x = Qf5(x, -mu)  (invert_Qtm.c:443-446), done whether or not converged
    CVCB_TRY(launch_tm_full(L, aux, x, 0.5 / L->kappa, -L->mu, -0.5, true, nullptr));
    std::swap(x, aux);
  }
  CVCB_TRY(spinor_out(L, xi, x, g.V));
  if (!converged) {
    CVCB_CUDA(cudaStreamSynchronize(L->stream));
    if (hs.done == 2) {  // a non-finite alpha, omega or beta stopped the recursion
      set_error("BiCGStab broke down after %d iterations (relative residual^2 %g)", hs.niter,
                hs.norm / hs.normb);
      return CVCB_BREAKDOWN;
    }
    set_error("no convergence after %d iterations (relative residual^2 %g)", niter,
              hs.norm / hs.normb);
    return CVCB_NO_CONVERGENCE;
  }
  if (true_res2) {
    // true residual |Q x - phi|^2 / |phi|^2 (invert_Qtm.c:257-267 / :466-475)
    CVCB_TRY(launch_tm_full(L, t, x, 0.5 / L->kappa, L->mu, -0.5, false, nullptr));
    k_sub<<<eb, 256, 0, L->stream>>>(t, t, phid, n);
    CVCB_LAUNCHED(L);
    double r2n;
    CVCB_TRY(dot_re(L, t, t, n, &r2n));
    *true_res2 = r2n / hs.normb;
  }
  CVCB_CUDA(cudaStreamSynchronize(L->stream));
  return niter;
}

}  // namespace cvcb

extern "C" {

int cvcb_invert_Qtm(cvcb_lattice *L, double *xi, const double *phi, double solver_precision,
                    int niter_max, double *true_res2) {
  if (!L || !xi || !phi) return CVCB_ERR_NULL;
  if (!L->have_gauge) {
    cvcb::set_error("no gauge field uploaded");
    return CVCB_ERR_STATE;
  }
  CVCB_CUDA(cudaSetDevice(L->device));
  return cvcb::invert_bicgstab(L, false, xi, phi, solver_precision, niter_max, true_res2);
}

int cvcb_invert_Qtm_her(cvcb_lattice *L, double *xi, const double *phi, double solver_precision,
                        int niter_max, double *true_res2) {
  if (!L || !xi || !phi) return CVCB_ERR_NULL;
  if (!L->have_gauge) {
    cvcb::set_error("no gauge field uploaded");
    return CVCB_ERR_STATE;
  }
  CVCB_CUDA(cudaSetDevice(L->device));
  return cvcb::invert_bicgstab(L, true, xi, phi, solver_precision, niter_max, true_res2);
}

}  // extern "C"
