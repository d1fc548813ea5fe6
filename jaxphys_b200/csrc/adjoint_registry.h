// Registry of the transposed step's passes (fdtd3d_adjoint.cuh), instantiated
// in adjoint_kernels.cu (its own translation unit, compiled in parallel with
// the host code).
#pragma once

#include "fdtd3d_adjoint.cuh"

namespace jxf {

using AdjKernel = void (*)(const Adj3D, const SweepPlan);

struct AdjKernels {
  AdjKernel e, h;  // pass over the E adjoint, over the H adjoint
  int v;           // cells per thread
};

// mode: MODE_ABSORB (also PEC with unit tables) or MODE_CPML; kappa: CPML with
// kappa > 1; cbarr: per-cell E factors.
AdjKernels adj_kernels(int mode, bool kappa, bool cbarr, int nz);

}  // namespace jxf
