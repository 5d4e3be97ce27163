// An operator call whose bulk copies are late: the flag that k_tm_full_cvc
// raises when a wait of its runs out is raised here on the host instead.  The
// call that finds it reports an error, the calls after it do not.
#include <cstdio>
#include <vector>

#include "../../cvc_b200/csrc/cvcb_internal.h"

int main() {
  cvcb_lattice *L = nullptr;
  if (cvcb_lattice_create(&L, 16, 8, 8, 10, 0) != CVCB_OK) return 2;
  const size_t V = 16 * 8 * 8 * 10;
  std::vector<double> g(72 * V), phi(24 * V), xi(24 * V);
  cvcb_gauge_random(g.data(), 16, 8, 8, 10, 0.3, 5);
  if (cvcb_upload_gauge(L, g.data()) != CVCB_OK) return 2;
  for (size_t k = 0; k < phi.size(); ++k) phi[k] = 1.0 / (1.0 + k % 97);
  if (cvcb_Q_phi_tbc(L, xi.data(), phi.data()) != CVCB_OK) return 2;
  const std::vector<double> want = xi;
  const unsigned one = 1;
  cudaMemcpy(L->red_counter + cvcb::kLateFlag, &one, sizeof one, cudaMemcpyHostToDevice);
  const int late = cvcb::tm_full_cvc_status(L);
  const int next = cvcb_Q_phi_tbc(L, xi.data(), phi.data());
  std::printf("%d %d %d\n", late == CVCB_ERR_CUDA, next == CVCB_OK, xi == want);
  cvcb_lattice_destroy(L);
  return 0;
}
