// Kernels of the explicit step around the fused gather/scatter kernel (all
// nodal work is FP64 in every form): active-block compaction, grid update
// (contact, boundary, moveGrid) and the exact triplet export.
#pragma once

#include "exact_map.cuh"
#include "geom.cuh"
#include "state.cuh"

namespace mpmb200 {

// Sets n int32 values to v.
__global__ void k_fill_i32(int32_t* p, int64_t n, int32_t v) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) p[i] = v;
}

// Compacts the flagged node blocks of the batch's block space into `list`,
// clears the flags and keeps the per-block activity of this step in
// `was_active`.
__global__ void k_compact(const BatchHdr* hdr, uint32_t* flags, int64_t* list, unsigned long long* count,
                          uint8_t* was_active) {
  const int64_t nblocks = hdr->blocks;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  for (int64_t base = blockIdx.x * (int64_t)blockDim.x; base < nblocks; base += stride) {
    const int64_t blk = base + threadIdx.x;
    const bool on = blk < nblocks && flags[blk] != 0u;
    if (blk < nblocks) {
      was_active[blk] = on ? 1 : 0;
      if (on) flags[blk] = 0u;
    }
    const unsigned mask = __ballot_sync(0xffffffffu, on);
    if (mask == 0u) continue;
    unsigned long long first = 0;
    if (lane == 0) first = atomicAdd(count, (unsigned long long)__popc(mask));
    first = __shfl_sync(0xffffffffu, first, 0);
    if (on) list[first + __popc(mask & ((1u << lane) - 1u))] = blk;
  }
}

// Grid update of one node (slot li of block gblk of the batch's block space):
// ContactHuang::generateRules normalisation and applyRules
// (contact_huang.cpp:80-197), CartesianBox (cartesian_box.cpp:73-85) and
// moveGrid (explicit_usl.cpp:233-264). Returns the bodies that have mass there
// (the grid term of the step's traffic).
template <int DIM>
__device__ __forceinline__ int grid_node(const InstDev* insts, const GridBody* bodies, const int32_t* blk_inst,
                                         int64_t gblk, int li) {
  const InstDev& I = insts[blk_inst[gblk]];
  const Geom& g = I.g;
  const StepParams& sp = I.sp;
  const double dt = sp.dt;
  const GridBody* GB = bodies + I.body0;
  const int64_t blk = gblk - I.block_off;
  int i, j, k;
  slot_ijk(g, blk, li, i, j, k);
  if (!(i < g.nn[0] && j < g.nn[1] && k < g.nn[2])) return 0;
  const int64_t s = blk * 64 + li;
  int with_mass = 0;
  for (int b = 0; b < I.nb; b++) with_mass += GB[b].A.m[s] > 0.0 ? 1 : 0;
  if (GB[0].Ar.m != nullptr) {
    // deterministic form: each nodal value arrived as two exactly summed
    // parts (level 0 in A, level 1 in Ar); one fixed rounding joins them
    for (int b = 0; b < I.nb; b++) {
      const NodesAcc& A = GB[b].A;
      const NodesAcc& R = GB[b].Ar;
      A.m[s] = A.m[s] + R.m[s];
      R.m[s] = 0.0;
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        A.mx[d][s] = A.mx[d][s] + R.mx[d][s];
        A.f[d][s] = A.f[d][s] + R.f[d][s];
        R.mx[d][s] = 0.0;
        R.f[d][s] = 0.0;
        if (A.nrm[0] != nullptr) {
          A.nrm[d][s] = A.nrm[d][s] + R.nrm[d][s];
          R.nrm[d][s] = 0.0;
        }
      }
    }
  }
  // the scatter leaves out the body force; S * (m b) summed over points is
  // the nodal mass times g (explicit_usl.cpp:150-154, b uniform)
  for (int b = 0; b < I.nb; b++) {
    const NodesAcc& A = GB[b].A;
    const double m = A.m[s];
#pragma unroll
    for (int d = 0; d < DIM; d++)
      if (sp.grav[d] != 0.0) A.f[d][s] = A.f[d][s] + m * sp.grav[d];
  }
  // CartesianFrictionalBox reads the nodal force before contact
  // (bcNodalForce: S (m b) - gradS (V T), cartesian_frictional_box.cpp:86-108)
  double fpre[kMaxBodies][3];
  for (int b = 0; b < I.nb; b++)
    if (GB[b].has_boundary == 3)
#pragma unroll
      for (int d = 0; d < DIM; d++) fpre[b][d] = GB[b].A.f[d][s];
  for (int c = 0; c < I.nc; c++) {
    const NodesAcc& A1 = GB[I.cb1[c]].A;
    const NodesAcc& A2 = GB[I.cb2[c]].A;
    double n[3] = {0.0, 0.0, 0.0};
    double nn = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; d++) {
      n[d] = A1.nrm[d][s];
      nn += n[d] * n[d];
    }
    const double m1 = A1.m[s], m2 = A2.m[s];
    if (!I.reflected[c]) {
      const double inv_norm = 1.0 / sqrt(nn);
#pragma unroll
      for (int d = 0; d < DIM; d++) n[d] *= inv_norm;
    } else if (m1 > 0) {
      // ContactHuang_ReflectedBoundary (contact_huang_reflected_boundary.cpp:
      // 90-114): the components normal to a wall of the box are dropped
      // before the normalisation, at nodes where body 1 has mass
      nn = 0.0;
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        const int cd = d == 0 ? i : (d == 1 ? j : k);
        if (cd == 0 || cd == g.N[d]) n[d] = 0.0;
        nn += n[d] * n[d];
      }
      const double inv_norm = 1.0 / sqrt(nn);
#pragma unroll
      for (int d = 0; d < DIM; d++) n[d] *= inv_norm;
    }
    double fc[3] = {0.0, 0.0, 0.0};
    if (m1 > 0 && m2 > 0) {
      double mv1[3], mv2[3], vcm[3];
      double f1[3], f2[3];
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        f1[d] = A1.f[d][s];
        f2[d] = A2.f[d][s];
        if (sp.contact_spec == 1) {
          mv1[d] = A1.mx[d][s] + dt * f1[d];
          mv2[d] = A2.mx[d][s] + dt * f2[d];
        } else {
          mv1[d] = A1.mx[d][s];
          mv2[d] = A2.mx[d][s];
        }
      }
      const double inv_m12 = 1.0 / (m1 + m2);
      const double inv_m1 = 1.0 / m1;
      double test = 0.0;
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        vcm[d] = (mv1[d] + mv2[d]) * inv_m12;
        test += (mv1[d] * inv_m1 - vcm[d]) * n[d];
      }
      if (test > 0) {
        double vcm_n = 0.0, mv1_n = 0.0;
#pragma unroll
        for (int d = 0; d < DIM; d++) {
          vcm_n += vcm[d] * n[d];
          mv1_n += mv1[d] * n[d];
        }
        const double fn = m1 / dt * (vcm_n - mv1_n / m1);
        const double m1dt = m1 / dt;
        double s1[3], ss = 0.0;
#pragma unroll
        for (int d = 0; d < DIM; d++) {
          s1[d] = m1dt * (vcm[d] - mv1[d] * inv_m1) - fn * n[d];
          ss += s1[d] * s1[d];
        }
        const double ft = sqrt(ss);
        if (ft != 0) {
          const double inv = 1.0 / ft;
#pragma unroll
          for (int d = 0; d < DIM; d++) s1[d] *= inv;
        }
        const double a = (fn < 0.0) ? fn : 0.0;  // std::min(0.0, fn)
        const double mufn = I.mu[c] * fabs(fn);
        const double b = (fabs(ft) < mufn) ? fabs(ft) : mufn;  // std::min(mu|fn|, |ft|)
#pragma unroll
        for (int d = 0; d < DIM; d++) {
          fc[d] = a * n[d] + b * s1[d];
          A1.f[d][s] = f1[d] + fc[d];
          A2.f[d][s] = f2[d] - fc[d];
        }
      }
    }
    if (I.normal_out[c] != nullptr) {
#pragma unroll
      for (int d = 0; d < 3; d++) {
        I.normal_out[c][3 * s + d] = (d < DIM) ? n[d] : 0.0;
        I.force_out[c][3 * s + d] = fc[d];
      }
    }
  }
  const bool on_face = (i == 0 || i == g.N[0] || j == 0 || j == g.N[1] || (DIM == 3 && (k == 0 || k == g.N[2])));
  for (int b = 0; b < I.nb; b++) {
    const NodesAcc& A = GB[b].A;
    const NodesVel& V = GB[b].V;
    const double m = A.m[s];
    double mx[3], f[3];
#pragma unroll
    for (int d = 0; d < DIM; d++) {
      mx[d] = A.mx[d][s];
      f[d] = A.f[d][s];
    }
    const int kind = GB[b].has_boundary;
    if (kind == 1 && on_face) {
      // CartesianBox (cartesian_box.cpp:73-85): every component of a node
      // on any wall
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        mx[d] = 0.0;
        f[d] = 0.0;
      }
    } else if (kind == 2 && on_face) {
      // CartesianSmoothBox (cartesian_smooth_box.cpp:69-83): the
      // wall-normal components only
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        const int c = d == 0 ? i : (d == 1 ? j : k);
        if (c == 0 || c == g.N[d]) {
          mx[d] = 0.0;
          f[d] = 0.0;
        }
      }
    } else if (kind == 3 && on_face) {
      // CartesianFrictionalBox (cartesian_frictional_box.cpp:94-143): the
      // closing momentum of each wall component gives the normal force,
      // the component is zeroed, and friction of at most mu_f times the
      // normal force opposes the remaining motion (interior nodes: no
      // normal force, no change)
      double dmom[3] = {0.0, 0.0, 0.0};
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        const int c = d == 0 ? i : (d == 1 ? j : k);
        const double closing = mx[d] + dt * fpre[b][d];
        if (c == 0) {
          dmom[d] = -((closing < 0.0) ? closing : 0.0);   // -std::min(0.0, .)
          mx[d] = 0.0;
          f[d] = 0.0;
        } else if (c == g.N[d]) {
          dmom[d] = -((0.0 < closing) ? closing : 0.0);   // -std::max(0.0, .)
          mx[d] = 0.0;
          f[d] = 0.0;
        }
      }
      double nn = 0.0;
#pragma unroll
      for (int d = 0; d < DIM; d++) nn += dmom[d] * dmom[d];
      const double f_normal = sqrt(nn) / dt;
      double mm = 0.0;
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        dmom[d] = mx[d] + dt * f[d];
        mm += dmom[d] * dmom[d];
      }
      const double nrm = sqrt(mm);
      if (nrm > 0) {
        const double a = nrm / dt, bnd = f_normal * GB[b].mu_f;
        const double cf = (bnd < a) ? bnd : a;   // std::min(|dm| / dt, f_normal mu_f)
        // vector / scalar multiplies by the reciprocal (mpm_vector.hpp:609-615)
        const double inv = 1.0 / nrm;
#pragma unroll
        for (int d = 0; d < DIM; d++) f[d] = f[d] - (cf * dmom[d]) * inv;
      }
    }
    double inv = 0.0;
    if (m > 0) inv = 1.0 / m;
#pragma unroll
    for (int d = 0; d < DIM; d++) {
      mx[d] = mx[d] + dt * f[d];
      V.vt[d][s] = (m > 0) ? mx[d] * inv : 0.0;
      V.dv[d][s] = (m > 0) ? (dt * f[d]) * inv : 0.0;
    }
    const NodesAcc& Sn = GB[b].snap;
    if (Sn.m != nullptr) {
      Sn.m[s] = m;
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        Sn.mx[d][s] = mx[d];
        Sn.f[d][s] = f[d];
      }
    }
    // the next step's scatter accumulates into zeroed arrays
    A.m[s] = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; d++) {
      A.mx[d][s] = 0.0;
      A.f[d][s] = 0.0;
      if (A.nrm[0] != nullptr) A.nrm[d][s] = 0.0;
    }
  }
  return with_mass;
}

// Grid update over the listed node blocks (k_compact): one CTA of 64 threads
// per block, one thread per node; each node is owned by exactly one thread.
template <int DIM>
__global__ void __launch_bounds__(64) k_grid(const InstDev* insts, const GridBody* bodies, const int32_t* blk_inst,
                                             const int64_t* list, const unsigned long long* count,
                                             unsigned long long* active_nodes) {
  const int64_t cnt = (int64_t)*count;
  for (int64_t e = blockIdx.x; e < cnt; e += gridDim.x) {
    const int with_mass =
        __reduce_add_sync(0xffffffffu, grid_node<DIM>(insts, bodies, blk_inst, list[e], threadIdx.x));
    if ((threadIdx.x & 31) == 0 && with_mass > 0) atomicAdd(active_nodes, (unsigned long long)with_mass);
  }
}

// The same for small block spaces, straight from the flags: a CTA of 256
// threads looks at 256 flags at a time (groups of four neighbours, dealt out
// to the CTAs in turn, since active blocks lie together), clears them, keeps
// the activity of this step in `was_active`, and takes its active blocks four
// at once. Without the list a step is two launches, not three: measured (us
// per step, list -> scan) 144 points in 2D 24.5 -> 20.7, 1,728 points on 343
// blocks 32.2 -> 27.8, two bodies on 4,096 blocks 40.3 -> 35.7; on 36,000
// blocks 109 -> 111 and on the column's 139,000 381 -> 390, where the list
// deals the blocks out more evenly. Hence the line at kScanBlocks.
constexpr int64_t kScanBlocks = 16384;
constexpr int kGridThreads = 256;
template <int DIM>
__global__ void __launch_bounds__(kGridThreads) k_grid_scan(const BatchHdr* hdr, const InstDev* insts,
                                                       const GridBody* bodies, const int32_t* blk_inst,
                                                       uint32_t* flags, uint8_t* was_active,
                                                       unsigned long long* active_nodes) {
  __shared__ int64_t list[kGridThreads];
  __shared__ int warp_cnt[kGridThreads / 32];
  const int64_t nblocks = hdr->blocks;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int with_mass = 0;
  for (int64_t r = 0; r * (kGridThreads / 4) * gridDim.x * 4 < nblocks; r++) {
    const int64_t gblk =
        4 * ((r * (kGridThreads / 4) + (threadIdx.x >> 2)) * gridDim.x + blockIdx.x) + (threadIdx.x & 3);
    const bool on = gblk < nblocks && flags[gblk] != 0u;
    if (gblk < nblocks) {
      was_active[gblk] = on ? 1 : 0;
      if (on) flags[gblk] = 0u;
    }
    const unsigned mask = __ballot_sync(0xffffffffu, on);
    if (lane == 0) warp_cnt[warp] = __popc(mask);
    __syncthreads();
    int before = 0, count = 0;
#pragma unroll
    for (int w = 0; w < kGridThreads / 32; w++) {
      before += w < warp ? warp_cnt[w] : 0;
      count += warp_cnt[w];
    }
    if (on) list[before + __popc(mask & ((1u << lane) - 1u))] = gblk;
    __syncthreads();
    for (int e = threadIdx.x >> 6; e < count; e += kGridThreads / 64)
      with_mass += grid_node<DIM>(insts, bodies, blk_inst, list[e], threadIdx.x & 63);
    __syncthreads();   // the list is written again
  }
  with_mass = __reduce_add_sync(0xffffffffu, with_mass);
  if (lane == 0 && with_mass > 0) atomicAdd(active_nodes, (unsigned long long)with_mass);
}

// Exact triplet export (mpmgpu_dump_map).
template <int DIM>
__global__ void k_export_map(Geom g, int cpdi, PointsDev P, int32_t* node_out, double* s_out, double* g_out) {
  constexpr int cp = 1 << DIM;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < P.n; p += stride) {
    // slots in original point order (P.pid), so the host reads triplets in
    // the reference's point-major order whatever the storage order
    const int64_t slot = (int64_t)P.pid[p] * cp * cp;
    if (!P.active[p]) {
      for (int k = 0; k < cp * cp; k++) node_out[slot + k] = -1;
      continue;
    }
    double x[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int d = 0; d < DIM; d++) x[d] = P.x[d][p];
    if (export_point<DIM>(g, cpdi, x, P.ext[p], node_out, s_out, g_out, slot) < 0) P.active[p] = 0;
  }
}

}  // namespace mpmb200
