// Registry of the in-place two-pass step kernels (fdtd3d_sweep.cuh).  The
// kernels are instantiated in sweep_kernels.cu (its own translation unit,
// compiled in parallel with the host code).
#pragma once

#include "fdtd3d_sweep.cuh"

namespace jxf {

using SweepKernel = void (*)(const Step3D, const SweepPlan);
using SweepSnapKernel = void (*)(const Step3D, const SweepPlan, const SweepSnap);
using SweepGroupKernel = void (*)(const SweepGroup);

struct SweepKernels {
  SweepKernel h, e;
  SweepGroupKernel group_h, group_e;
  SweepSnapKernel snap_e;
  int v0, v1;   // cells per thread outside / inside the z slabs
  int threads;  // per block
};

// Kernels of a grid: MODE_ABSORB (also PEC with unit tables), MODE_PERIODIC or
// MODE_CPML; kappa: CPML with kappa > 1; cbarr: per-cell E factors.
SweepKernels sweep_kernels(int mode, bool kappa, bool cbarr, int nz);

}  // namespace jxf
