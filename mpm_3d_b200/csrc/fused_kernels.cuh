// The instantiations of the fused kernel, by form, point precision and points
// per item. They are compiled apart from the engine, one object file per group
// (fused_kernels.cu): the compiler takes minutes for all of them, the groups
// build in parallel, and a kernel's code does not depend on what else is
// compiled with it.
#pragma once

#include <cstddef>

namespace mpmb200 {

// One instantiation as cudaLaunchKernel takes it; its argument is a
// FusedLaunch<PT>.
struct FusedKernel {
  const void* fn = nullptr;
  int threads = 0;
  size_t smem = 0;
};

// Point-per-thread kernel (3D): items of CAP points; elastic: every body is
// IsotropicLinearElasticity.
template <typename PT, int CAP>
FusedKernel lean_kernel(bool normal, bool single, bool elastic);

// Staged kernel; single: one-body launches (items of 512 points only).
template <typename PT, bool DET>
FusedKernel staged_kernel(int dim, int cap, bool normal, bool single);

}  // namespace mpmb200
