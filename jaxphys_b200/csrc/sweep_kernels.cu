// Instantiations of the in-place two-pass step kernels (sweep_registry.h).
#include "sweep_registry.h"

namespace jxf {

namespace {

template <int MODE, bool KAPPA, int V0, int V1>
SweepKernels make(bool cbarr) {
  constexpr int B = MODE == MODE_PERIODIC ? MODE_ABSORB : MODE;
  return SweepKernels{k3d_sweep<true, MODE, V0, V1, KAPPA, false>,
                      cbarr ? k3d_sweep<false, MODE, V0, V1, KAPPA, true>
                            : k3d_sweep<false, MODE, V0, V1, KAPPA, false>,
                      // (periodic grids are not batched, and have no adjoint)
                      MODE == MODE_PERIODIC ? nullptr : k3d_sweep_group<true, B, V0, V1, KAPPA, false>,
                      MODE == MODE_PERIODIC ? nullptr
                      : cbarr               ? k3d_sweep_group<false, B, V0, V1, KAPPA, true>
                                            : k3d_sweep_group<false, B, V0, V1, KAPPA, false>,
                      MODE == MODE_PERIODIC ? nullptr
                      : cbarr               ? k3d_sweep_snap<B, V0, V1, KAPPA, true>
                                            : k3d_sweep_snap<B, V0, V1, KAPPA, false>,
                      V0, V1, sweep_threads(MODE, V0)};
}

// The widest loads that nz allows (rows of a multiple of V cells keep every
// access aligned); z-slab cells go in pairs: four per thread cost the CPML
// kernel registers (128^3, 10 layers: 27.6 us a step against 24.0).
template <int MODE, bool KAPPA>
SweepKernels pick(bool cbarr, int nz) {
  if (nz % 4 == 0) return make<MODE, KAPPA, 4, MODE == MODE_CPML ? 2 : 4>(cbarr);
  if (nz % 2 == 0) return make<MODE, KAPPA, 2, 2>(cbarr);
  return make<MODE, KAPPA, 1, 1>(cbarr);
}

}  // namespace

SweepKernels sweep_kernels(int mode, bool kappa, bool cbarr, int nz) {
  if (mode == MODE_PERIODIC) return pick<MODE_PERIODIC, false>(cbarr, nz);
  if (mode == MODE_CPML)
    return kappa ? pick<MODE_CPML, true>(cbarr, nz) : pick<MODE_CPML, false>(cbarr, nz);
  return pick<MODE_ABSORB, false>(cbarr, nz);
}

}  // namespace jxf
