// Instantiations of the transposed step's passes (adjoint_registry.h).
#include "adjoint_registry.h"

namespace jxf {

namespace {

template <int MODE, bool KAPPA, int V>
AdjKernels make(bool cbarr) {
  return AdjKernels{cbarr ? k3a_pass<true, MODE, V, KAPPA, true>
                          : k3a_pass<true, MODE, V, KAPPA, false>,
                    k3a_pass<false, MODE, V, KAPPA, false>, V};
}

// Two cells per thread where rows are even (aligned pairs): with four, the
// pass over the E adjoint would need more registers than five blocks per SM
// leave it (per cell: E, H, forward H, cb, psi and an FP64 sum).
template <int MODE, bool KAPPA>
AdjKernels pick(bool cbarr, int nz) {
  return nz % 2 == 0 ? make<MODE, KAPPA, 2>(cbarr) : make<MODE, KAPPA, 1>(cbarr);
}

}  // namespace

AdjKernels adj_kernels(int mode, bool kappa, bool cbarr, int nz) {
  if (mode == MODE_CPML)
    return kappa ? pick<MODE_CPML, true>(cbarr, nz) : pick<MODE_CPML, false>(cbarr, nz);
  return pick<MODE_ABSORB, false>(cbarr, nz);
}

}  // namespace jxf
