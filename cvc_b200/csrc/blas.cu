// Reductions behind spinor_scalar_product_co/_re (invert_Qtm.c:28-84) and
// the C-ABI entry points of the operators.
#include <time.h>

#include <cmath>

#include "cvcb_internal.h"
#include "reduce.cuh"

namespace cvcb {

struct DotCo {
  const double2 *__restrict__ a;
  const double2 *__restrict__ b;
  __device__ void operator()(size_t k, double (&acc)[2]) const {
    const double2 x = __ldg(a + k), y = __ldg(b + k);
    acc[0] += x.x * y.x + x.y * y.y;  // Re conj(x) y
    acc[1] += x.x * y.y - x.y * y.x;  // Im conj(x) y
  }
};

int dot_co(cvcb_lattice *L, const double2 *a, const double2 *b, size_t n, double out[2]) {
  CVCB_TRY(launch_reduce<2>(L, DotCo{a, b}, StoreTotals<2>{L->red_result}, n));
  CVCB_CUDA(cudaMemcpyAsync(out, L->red_result, 2 * sizeof(double), cudaMemcpyDeviceToHost,
                            L->stream));
  CVCB_CUDA(cudaStreamSynchronize(L->stream));
  return CVCB_OK;
}

int dot_re(cvcb_lattice *L, const double2 *a, const double2 *b, size_t n, double *out) {
  double w[2];
  CVCB_TRY(dot_co(L, a, b, n, w));
  *out = w[0];
  return CVCB_OK;
}

}  // namespace cvcb

using namespace cvcb;

namespace {

int need_gauge(cvcb_lattice *L) {
  if (!L) return CVCB_ERR_NULL;
  if (!L->have_gauge) {
    set_error("no gauge field uploaded (cvcb_upload_gauge)");
    return CVCB_ERR_STATE;
  }
  return CVCB_OK;
}

// a clock of some milliseconds' resolution, read without a system call
double coarse_seconds() {
  timespec t;
  clock_gettime(CLOCK_MONOTONIC_COARSE, &t);
  return (double)t.tv_sec + 1e-9 * (double)t.tv_nsec;
}

// out = op(in) with the full-lattice kernel on CVC-layout fields, in place on
// device arrays; host arrays go through staging, and so does an input that
// overlaps the output or is managed or another GPU's memory (the kernel's bulk
// copies read this GPU's own).
int apply_full(cvcb_lattice *L, double *xi, const double *phi, double a, double b, double c,
               bool g5out) {
  CVCB_TRY(need_gauge(L));
  if (!xi || !phi) return CVCB_ERR_NULL;
  CVCB_CUDA(cudaSetDevice(L->device));
  const size_t n = (size_t)L->g.V * 24, fb = n * sizeof(double);
  const uintptr_t x = reinterpret_cast<uintptr_t>(xi), p = reinterpret_cast<uintptr_t>(phi);
  const bool out_dev = is_device_ptr(xi);
  const double *in = phi;
  double *out = xi;
  void *f;
  if (!is_own_device_ptr(L, phi) || (out_dev && x < p + fb && p < x + fb)) {
    CVCB_TRY(ensure_buffer(L, SLOT_F0, fb, &f));
    CVCB_CUDA(cudaMemcpyAsync(f, phi, fb, cudaMemcpyDefault, L->stream));
    in = static_cast<const double *>(f);
  }
  if (!out_dev) {
    CVCB_TRY(ensure_buffer(L, SLOT_F1, fb, &f));
    out = static_cast<double *>(f);
  }
  const double t0 = coarse_seconds();
  CVCB_TRY(launch_tm_full_cvc(L, out, in, a, b, c, g5out));
  if (!out_dev) CVCB_CUDA(cudaMemcpyAsync(xi, out, fb, cudaMemcpyDeviceToHost, L->stream));
  CVCB_CUDA(cudaStreamSynchronize(L->stream));
  // half the limit leaves room for two clocks that differ
  return coarse_seconds() - t0 > 0.5 * kCvcWaitSeconds ? tm_full_cvc_status(L) : CVCB_OK;
}

// Stage one CVC-layout field (host or device) to a device pointer usable by
// a reduction that ignores site order.
int stage_raw(cvcb_lattice *L, int slot, const double *src, int V, const double2 **out) {
  if (is_device_ptr(src)) {
    *out = reinterpret_cast<const double2 *>(src);
    return CVCB_OK;
  }
  void *st;
  CVCB_TRY(ensure_buffer(L, slot, (size_t)V * 24 * sizeof(double), &st));
  CVCB_CUDA(cudaMemcpyAsync(st, src, (size_t)V * 24 * sizeof(double), cudaMemcpyHostToDevice,
                            L->stream));
  *out = static_cast<const double2 *>(st);
  return CVCB_OK;
}

}  // namespace

extern "C" {

int cvcb_Q_phi_tbc(cvcb_lattice *L, double *xi, const double *phi) {
  if (!L) return CVCB_ERR_NULL;
  return apply_full(L, xi, phi, 0.5 / L->kappa, L->mu, -0.5, false);
}

int cvcb_Q_phi(cvcb_lattice *L, double *xi, const double *phi, double mutm) {
  if (!L) return CVCB_ERR_NULL;
  return apply_full(L, xi, phi, 0.5 / L->kappa, mutm, -0.5, false);
}

int cvcb_Qf5(cvcb_lattice *L, double *xi, const double *phi, double mutm) {
  if (!L) return CVCB_ERR_NULL;
  return apply_full(L, xi, phi, 0.5 / L->kappa, mutm, -0.5, true);
}

int cvcb_Hopping(cvcb_lattice *L, double *xi, const double *phi) {
  if (!L) return CVCB_ERR_NULL;
  return apply_full(L, xi, phi, 0.0, 0.0, -L->kappa, false);
}

int cvcb_g5_phi(cvcb_lattice *L, double *phi) {
  if (!L || !phi) return CVCB_ERR_NULL;
  CVCB_CUDA(cudaSetDevice(L->device));
  void *f0;
  CVCB_TRY(ensure_buffer(L, SLOT_F0, (size_t)L->g.V * 12 * sizeof(double2), &f0));
  CVCB_TRY(spinor_in(L, static_cast<double2 *>(f0), phi, L->g.V));
  CVCB_TRY(launch_g5(L, static_cast<double2 *>(f0), L->g.V));
  CVCB_TRY(spinor_out(L, phi, static_cast<const double2 *>(f0), L->g.V));
  CVCB_CUDA(cudaStreamSynchronize(L->stream));
  return CVCB_OK;
}

int cvcb_mul_one_pm_imu_inv(cvcb_lattice *L, double *phi, double sign, int V) {
  if (!L || !phi) return CVCB_ERR_NULL;
  if (V < 0 || V > L->g.V) {
    set_error("V = %d outside [0, %d]", V, L->g.V);
    return CVCB_ERR_ARG;
  }
  if (V == 0) return CVCB_OK;
  CVCB_CUDA(cudaSetDevice(L->device));
  void *f0;
  CVCB_TRY(ensure_buffer(L, SLOT_F0, (size_t)L->g.V * 12 * sizeof(double2), &f0));
  CVCB_TRY(spinor_in(L, static_cast<double2 *>(f0), phi, V));
  CVCB_TRY(launch_one_pm_imu_inv(L, static_cast<double2 *>(f0), sign, V));
  CVCB_TRY(spinor_out(L, phi, static_cast<const double2 *>(f0), V));
  CVCB_CUDA(cudaStreamSynchronize(L->stream));
  return CVCB_OK;
}

int cvcb_spinor_scalar_product_co(cvcb_lattice *L, double *w, const double *xi, const double *phi,
                                  int V) {
  if (!L || !w || !xi || !phi) return CVCB_ERR_NULL;
  if (V < 0 || V > L->g.V) {
    set_error("V = %d outside [0, %d]", V, L->g.V);
    return CVCB_ERR_ARG;
  }
  if (V == 0) {
    w[0] = w[1] = 0.0;
    return CVCB_OK;
  }
  CVCB_CUDA(cudaSetDevice(L->device));
  const double2 *a, *b;
  CVCB_TRY(stage_raw(L, SLOT_STAGE_A, xi, V, &a));
  CVCB_TRY(stage_raw(L, SLOT_STAGE_B, phi, V, &b));
  return dot_co(L, a, b, (size_t)V * 12, w);
}

int cvcb_spinor_scalar_product_re(cvcb_lattice *L, double *r, const double *xi, const double *phi,
                                  int V) {
  if (!r) return CVCB_ERR_NULL;
  double w[2];
  int rc = cvcb_spinor_scalar_product_co(L, w, xi, phi, V);
  if (rc < 0) return rc;
  *r = w[0];
  return CVCB_OK;
}

}  // extern "C"
