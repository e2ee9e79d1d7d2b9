// One group of the fused kernel's instantiations per object file, chosen with
// -DMPM_LEAN_CAP=<points per item> (point-per-thread kernel) or
// -DMPM_STAGED_DET=<0 or 1> (staged kernel) and -DMPM_POINT=<float or double>.
#include "fused_kernels.cuh"

#include "fused.cuh"
#include "fused_lean.cuh"

namespace mpmb200 {

#if defined(MPM_LEAN_CAP)

template <typename PT, int CAP, bool NORMAL, bool SINGLE, int MAT>
static FusedKernel lean_entry() {
  constexpr int NT = CAP == 128 ? 128 : 256;
  FusedKernel k;
  k.fn = reinterpret_cast<const void*>(&k_g2p2g_lean<3, PT, NT, CAP / NT, NORMAL, SINGLE, MAT>);
  k.threads = NT;
  k.smem = lean_smem_bytes<3, PT, CAP>();
  return k;
}

template <typename PT, int CAP>
FusedKernel lean_kernel(bool normal, bool single, bool elastic) {
  auto pick = [&](FusedKernel e, FusedKernel any) { return elastic ? e : any; };
  if (normal)
    return single ? pick(lean_entry<PT, CAP, true, true, 0>(), lean_entry<PT, CAP, true, true, -1>())
                  : pick(lean_entry<PT, CAP, true, false, 0>(), lean_entry<PT, CAP, true, false, -1>());
  return single ? pick(lean_entry<PT, CAP, false, true, 0>(), lean_entry<PT, CAP, false, true, -1>())
                : pick(lean_entry<PT, CAP, false, false, 0>(), lean_entry<PT, CAP, false, false, -1>());
}
template FusedKernel lean_kernel<MPM_POINT, MPM_LEAN_CAP>(bool, bool, bool);

#else

template <int DIM, typename PT, int CAP, bool NORMAL, bool SINGLE, bool DET>
static FusedKernel staged_entry() {
  FusedKernel k;
  k.fn = reinterpret_cast<const void*>(&k_g2p2g<DIM, PT, CAP, NORMAL, SINGLE, DET>);
  k.threads = fused_threads<PT, CAP>();
  k.smem = fused_smem_bytes<DIM, PT, CAP, NORMAL, DET>();
  return k;
}

template <int DIM, typename PT, int CAP, bool DET>
static FusedKernel staged_sized(bool normal, bool single) {
  if constexpr (CAP == 512) {
    if (single)
      return normal ? staged_entry<DIM, PT, CAP, true, true, DET>() : staged_entry<DIM, PT, CAP, false, true, DET>();
  }
  return normal ? staged_entry<DIM, PT, CAP, true, false, DET>() : staged_entry<DIM, PT, CAP, false, false, DET>();
}

template <typename PT, bool DET>
FusedKernel staged_kernel(int dim, int cap, bool normal, bool single) {
  if (dim == 2) return staged_sized<2, PT, 512, DET>(normal, single);
  // 3D; the deterministic form has two tile levels, which leave room for 256
  if constexpr (!DET) {
    if constexpr (sizeof(PT) == 4) {
      if (cap == 1024) return staged_sized<3, PT, 1024, DET>(normal, single);
    }
    if (cap == 512) return staged_sized<3, PT, 512, DET>(normal, single);
  }
  return staged_sized<3, PT, 256, DET>(normal, single);
}
template FusedKernel staged_kernel<MPM_POINT, MPM_STAGED_DET != 0>(int, int, bool, bool);

#endif

}  // namespace mpmb200
