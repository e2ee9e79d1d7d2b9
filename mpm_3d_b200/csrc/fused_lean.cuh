// Lean form of the fused gather + point update + scatter kernel: each thread
// takes its points from gather to the new map, and the nodal sums of a work
// item are formed per cell in registers, with no shared-memory atomics on
// FP64 values.
//
// A CTA of NT threads works on one work item at a time (at most PPT * NT
// points of one bin of one body, PPT points per thread):
//   0. the CTA stages the nodal velocities of the bin's node tile;
//   1. each thread takes its points (their arrays staged in shared memory by
//      bulk copies) through gather, state update (movePoints,
//      calculateStrainRate, updateDensity, updateStress) and map build at the
//      new position, writes what the scatter needs of the point (a record: two
//      numbers per axis and the 10 scatter sources) over its staged state and
//      links it into the list of its window's base cell;
//   2. four threads per non-empty cell, one per node row (y, z offset 0 or 1)
//      of the cell's window, walk the cell's list and accumulate the row's
//      nodes in registers, then add them into the global accumulators (one
//      global atomic per row node and value).
//
// Why: an FP64 add into shared memory is a load, an add and a 64-bit compare
// and swap in a loop, and a point adds 56 to 189 of them (8 to 27 nodes, 7
// values), one chain after the other. That chain, not memory, set the time of
// a work item (45 us for the one item of an SM on a 27,000-point body). A
// cell's points share their nodes, so summing them in registers leaves one
// add per cell, node and value, and that one goes to L2 as a reduction that
// no thread waits for.
//
// Measured against the kernel that added every point's contributions to a
// shared tile (us per step): column collapse of 3.1 M points 499 -> 386 (the
// kernel alone 468 -> 359, 291 algorithmic bytes per point: 2.0 -> 2.5 TB/s),
// two-body collision of 0.52 M points 171 -> 108, 21 block drops of 2.6 M points
// in all 952 -> 657, 1,728 points 51 -> 23. The column's figures are those of
// its initial lattice, where no window spans three nodes: once half of its
// points have a wide axis a step takes 600 us (a wide point gathers in rolled
// loops, and one wide along y or z enters two or four cells' lists). What bounds
// it now: 16 warps per SM (128 registers, 110 KB of shared memory per CTA) on
// chains of FP64 operations of 11 cycles each: on the column 41 % of the issue
// slots, FP64 pipe 29 %, shared-memory wavefronts 42 %. Tried and slower: 24
// warps at 80 registers with items of 256 points (item costs are paid twice, 472
// us on the column), the velocity tile as whole node blocks by bulk copies (the
// node blocks then straddle the bins, whose adds meet in twice the memory
// sectors: 4 to 15 %), the rows' sums combined in shared memory before the adds
// (spills), an L2 prefetch of the next item's arrays (1 %).
#pragma once

#include "fused.cuh"

namespace mpmb200 {

// Points per work item: 128 (CTAs of 128 threads), 256 (256 threads) or 512 (256
// threads, two points each: one tile load and one set of nodal adds for a whole
// 4x4x4 bin of 8 points per cell). The engine's defaults choose between 128 and
// 512 (kSmallPoints, items_for_bin); 256 is for the autotuner and the caller.
__host__ __device__ constexpr bool lean_size_ok(int cap) { return cap == 128 || cap == 256 || cap == 512; }
constexpr int kDefaultLeanCap = 512;

// Resident CTAs per SM the register budget is sized for.
template <typename PT, int NT, int PPT>
__host__ __device__ constexpr int lean_min_ctas() {
  return PPT == 2 ? 2 : (NT == 128 ? 4 : 3);
}

// Cells a window inside the tile can have its base in: T - 1 per axis.
constexpr int kLeanSide = 6;
constexpr int kLeanCells = kLeanSide * kLeanSide * kLeanSide;
constexpr int kLeanMask = (kLeanCells + 31) / 32;

// Staged copy of an item's point arrays, one row of cap_row elements per
// array: x v u s vol m ext (kFx .. kFext), then in the mixed form the low
// words of x, v and m. A point's thread reads its column and, when it has
// its new map, overwrites the column with the point's record for the
// scatter (its own column only, so no barrier is needed between the two):
// two numbers per axis (LeanMap::a and b), then the sources scaled by the
// map's scales, mass and momentum (always FP64, two rows each in the mixed
// form) and V sigma, and the scale of the contact normal.
constexpr int kFxl = kNF, kFvl = kNF + 3, kFml = kNF + 6;
constexpr int kRab = 0, kRm = 6;
template <typename PT>
constexpr int kRs = sizeof(PT) == 8 ? 10 : 14;
template <typename PT>
constexpr int kRgm = kRs<PT> + 6;
template <typename PT>
__host__ __device__ constexpr int lean_rows() {
  return sizeof(PT) == 8 ? kNF : kNF + 7;
}

// Shared memory: mbarriers (points, table entry slots 0 and 1) | table entry
// slots [2] | velocity tile [2 DIM][TN] in the point precision (mixed form:
// and in FP64 as loaded) | staged
// points [rows][cap_row] | active [cap_row] | list links | cell heads and
// mask | far points | cell list.
template <int DIM, typename PT>
__host__ __device__ constexpr size_t lean_off_tvel() {
  return kOffCtx + 2 * ctx_bytes<PT>();
}
template <int DIM, typename PT>
__host__ __device__ constexpr size_t lean_off_traw() {   // mixed form: the tile as it is in global memory
  return (lean_off_tvel<DIM, PT>() + sizeof(PT) * 2 * DIM * fused_tile_nodes<DIM, fused_bin<DIM>()>() + 15) / 16 * 16;
}
template <int DIM, typename PT>
__host__ __device__ constexpr size_t lean_off_pts() {
  return lean_off_traw<DIM, PT>() +
         (sizeof(PT) == 4 ? sizeof(double) * 2 * DIM * fused_tile_nodes<DIM, fused_bin<DIM>()>() : 0);
}
template <int DIM, typename PT, int CAP>
__host__ __device__ constexpr size_t lean_off_act() {
  return lean_off_pts<DIM, PT>() + sizeof(PT) * lean_rows<PT>() * cap_row<CAP>();
}
template <int DIM, typename PT, int CAP>
__host__ __device__ constexpr size_t lean_off_next() {
  return lean_off_act<DIM, PT, CAP>() + sizeof(int32_t) * cap_row<CAP>();
}
template <int DIM, typename PT, int CAP>
__host__ __device__ constexpr size_t lean_off_head() {
  return lean_off_next<DIM, PT, CAP>() + sizeof(uint16_t) * 2048;
}
template <int DIM, typename PT, int CAP>
__host__ __device__ constexpr size_t lean_off_far() {
  return lean_off_head<DIM, PT, CAP>() + sizeof(uint32_t) * (kLeanCells + kLeanMask + 1);
}
template <int DIM, typename PT, int CAP>
__host__ __device__ constexpr size_t lean_smem_bytes() {
  return lean_off_far<DIM, PT, CAP>() + sizeof(uint16_t) * CAP + kLeanCells;
}
static_assert(lean_off_pts<3, double>() % 16 == 0 && lean_off_pts<3, float>() % 16 == 0 &&
                  (cap_row<128>() * 4) % 16 == 0,
              "bulk copies write rows on 16-byte boundaries");

// Array f of the staged rows in global memory (the pointers of PointsT lie
// one behind the other: x v u s vol m ext, and xl vl ml).
static_assert(offsetof(PointsT<float>, ext) == offsetof(PointsT<float>, x) + kFext * sizeof(float*) &&
                  offsetof(PointsT<float>, ml) == offsetof(PointsT<float>, xl) + 6 * sizeof(float*),
              "staged rows follow the order of PointsT");
template <typename PT>
__device__ __forceinline__ const PT* lean_array(const PointsT<PT>& P, int f) {
  return f < kNF ? (&P.x[0])[f] : (&P.xl[0])[f - kNF];
}

// A staged position, velocity or mass in double: the FP64 form's value, or
// the mixed form's two words (hi + lo).
template <int ROW, typename PT>
__device__ __forceinline__ double lean_two(const PT* col, int hi, int lo) {
  if constexpr (sizeof(PT) == 8) return col[hi * ROW];
  else return (double)col[hi * ROW] + (double)col[lo * ROW];
}

// Stores a position or velocity (the mixed form splits it into its two words).
template <typename PT>
__device__ __forceinline__ void lean_store_two(PT* hi, PT* lo, int64_t p, double v) {
  if constexpr (sizeof(PT) == 8) {
    hi[p] = v;
  } else {
    float h, l;
    split_two_word(v, h, l);
    hi[p] = h;
    lo[p] = l;
  }
}

// Stress update of one point for material MAT (-1: the body's kind at run
// time). s6 holds the stress before the step on entry, after it on exit.
template <int DIM, int MAT, typename R, typename PT>
__device__ __forceinline__ void lean_stress(const BodyCtx<PT>& c, int64_t p, const R L[3][3], R* s6, R m, R vol,
                                            R dt) {
  const PointsT<PT>& P = c.P;
  const int kind = MAT >= 0 ? MAT : c.mat.kind;
  if (kind == 1) {
    neohookean_update<R>(P.ms, p, L, s6, (R)c.mat.G, (R)c.mat.lambda, dt);
  } else if (kind == 2) {
    sand_update<DIM, R>(P.ms, p, L, s6, m, vol, c.mat, dt);
  } else {
    jaumann_point<DIM, R>(L, s6, c.mat, c.sp.dt);
  }
}

// The map of one point in the compact form of its record. Per axis, with
// hat values wl at the lower corner's element and wh at the upper's:
//   narrow (both corners in one element): a = wl0 + wh0, b = wh0 - wl0;
//     weights {a, 2 - a}, gradient weights {b, -b}
//   wide (corners in neighbouring elements): a = wl0, b = wh1; weights
//     {a, (1 - a) + (1 - b), b}, gradient weights {-a, a - b, b}
//   point-sampled: a = 1 - r, b = -1/h; weights {a, 1 - a}, gradients {b, -b}
// which are PointMapT's W and G (a hat function's two values in an element
// sum to one, so the second is one minus the first, as it is rounded there).
// fl: bit d set for a wide axis d, bit 3 for the point-sampled map.
constexpr int kLeanSampled = 8;
template <typename R>
struct LeanMap {
  int base[3];
  R a[3], b[3];
  int fl;
  R sS, sG;
};

// Element of coordinate c on axis d and the offset within it in cells: the
// decisions of axis_element_fast (floor(c N / L), with the exact
// two-rounding form within 1e-9 of an integer). The rounding to an integer
// is two additions of 1.5 * 2^52, in the full-rate FP64 pipe (floor and the
// conversions to and from int run at a quarter of it), and the offset is
// what is left of c N / L: with the rounding of c itself it is as far from
// the exact one as (c - x_n) / h.
//
// `near` collects whether c N / L was within 1e-9 of an integer; the caller
// then takes lean_element_exact (one branch for all the corners of a point,
// so that their chains of additions overlap).
__device__ __forceinline__ int lean_element(const MapConst& mc, int d, double c, double& off, bool& near) {
  constexpr double kMagic = 6755399441055744.0;
  const double t = c * mc.NL[d];
  const double big = __dadd_rn(t, kMagic);
  const double r = __dadd_rn(big, -kMagic);
  off = t - r;
  near = near || fabs(off) < 1e-9;
  const bool below = off < 0.0;
  off = off + (below ? 1.0 : 0.0);
  return __double2loint(big) - (below ? 1 : 0);
}
// Within that band the offset is rounding, and its sign and its being zero
// decide weights and gradients: it is formed as build_map_fast forms it.
__device__ __forceinline__ int lean_element_exact(const Geom& g, const MapConst& mc, int d, double c, double& off) {
  const int i = axis_element_fast(g, mc, d, c);
  off = (c - g.h[d] * (double)i) * mc.invh[d];
  return i;
}

// Offset from a node (in cells) up to which a sampled point takes the general
// path: above the FP32 rounding of an offset in [0, 1].
constexpr double kLeanNodeBand = 1e-7;

// Builds the compact map (3D) with the decisions of build_map_fast and
// build_map_f32. Returns -1 outside the domain, 0 without triplets, 1
// otherwise, 2 for the two rare cases the compact form does not hold: an
// upper corner on the domain's upper face (it has no element) and a sampled
// point on a node or within rounding of one (its gradient is 0/0 or, by the
// offset's sign, jumps between -1/h and 1/h or falls away).
template <typename R>
__device__ __forceinline__ int lean_map(const Geom& g, const MapConst& mc, int cpdi_spec, const double* x, R extent,
                                        R sG, LeanMap<R>& lm, int* err) {
  const double a = 0.5 * (double)extent;
  lm.fl = 0;
  bool corners = cpdi_spec == 1 && a >= 0.0;
#pragma unroll
  for (int d = 0; d < 3; d++) corners = corners && x[d] - a >= 0.0 && x[d] + a < g.L[d];
  if (corners) {
    // both corners inside, so the point is
    int elo[3], ehi[3];
    double ol[3], oh[3];
    bool near = false;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      elo[d] = lean_element(mc, d, x[d] - a, ol[d], near);
      ehi[d] = lean_element(mc, d, x[d] + a, oh[d], near);
    }
    if (near) {
#pragma unroll 1
      for (int d = 0; d < 3; d++) {
        double l, h;
        const int el = lean_element_exact(g, mc, d, sel3(x, d) - a, l), eh = lean_element_exact(g, mc, d, sel3(x, d) + a, h);
#pragma unroll
        for (int k = 0; k < 3; k++)
          if (k == d) {
            elo[k] = el;
            ehi[k] = eh;
            ol[k] = l;
            oh[k] = h;
          }
      }
    }
    bool alias = false, spread = false;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      alias = alias || elo[d] >= g.N[d] || ehi[d] >= g.N[d];
      spread = spread || (unsigned)(ehi[d] - elo[d]) > 1u;
    }
    if (alias) {
      atomicOr(err, kErrElemAlias);
      return 0;
    }
    if (spread) atomicOr(err, kErrWideSpan);
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const bool wide = ehi[d] - elo[d] == 1;
      const R rl = fabs((R)ol[d]), rh = (R)oh[d];
      lm.base[d] = elo[d];
      lm.fl |= wide ? 1 << d : 0;
      const R wl0 = R(1) - rl;
      const R wh = R(1) - fabs(rh - (wide ? R(1) : R(0)));   // wide: wh1, else wh0
      lm.a[d] = wide ? wl0 : wl0 + wh;
      lm.b[d] = wide ? wh : wh - wl0;
    }
    lm.sS = R(0.125);
    lm.sG = sG;
    return 1;
  }
  if (!in_domain<3>(g, x)) return -1;
  bool closed = cpdi_spec == 1;
#pragma unroll
  for (int d = 0; d < 3; d++)
    if (!(x[d] - a <= g.L[d] && x[d] - a >= 0.0) || !(x[d] + a <= g.L[d] && x[d] + a >= 0.0)) closed = false;
  if (closed) return 2;   // an upper corner on the upper face
#pragma unroll
  for (int d = 0; d < 3; d++)
    if (!(x[d] < g.L[d])) return 0;
  lm.fl = kLeanSampled;
  bool on_node = false;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    double off;
    lm.base[d] = lean_element_exact(g, mc, d, x[d], off);
    if (lm.base[d] >= g.N[d]) {
      atomicOr(err, kErrElemAlias);
      return 0;
    }
    on_node = on_node || !(off > kLeanNodeBand && off < 1.0 - kLeanNodeBand);
    lm.a[d] = R(1) - (R)off;
    lm.b[d] = sizeof(R) == 8 ? (R)-mc.invh[d] : (R)-mc.invhf[d];
  }
  lm.sS = R(1);
  lm.sG = R(1);
  return on_node ? 2 : 1;
}

// Weight and gradient weight of axis node k (0..2) from a record's a, b.
template <typename R>
__device__ __forceinline__ void lean_node_weight(R a, R b, bool wide, R sum, int k, R& w, R& g) {
  if (wide) {
    w = k == 0 ? a : (k == 1 ? (R(1) - a) + (R(1) - b) : b);
    g = k == 0 ? -a : (k == 1 ? a - b : b);
  } else {
    w = k == 0 ? a : sum - a;
    g = k == 0 ? b : -b;
  }
}

template <int T, typename R>
__device__ __forceinline__ bool lean_in_tile(const LeanMap<R>& lm, const int* o) {
  bool in = true;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const int l = lm.base[d] - o[d];
    in = in && l >= 0 && l + ((lm.fl >> d) & 1) <= T - 2;
  }
  return in;
}

// Gather of one point from the staged tile: the sums are formed per node row
// (x nodes first, then the row's y and z weights). ANYW: some lane of the
// warp has a wide axis; the loops then run over the warp's union of offsets,
// rolled to keep the code small.
template <int T, int TN, bool ANYW, typename R>
__device__ __forceinline__ GatherSum<R> lean_gather(const LeanMap<R>& lm, const int* o, const R* tvel, int any) {
  using TL = TileLayout<3, T>;
  GatherSum<R> gs;
  const R sum = lm.fl & kLeanSampled ? R(1) : R(2);
  const R* t0 = tvel + (lm.base[0] - o[0]) + TL::RL * (lm.base[1] - o[1]);
  const int bz = lm.base[2] - o[2];
  R w0[3], g0[3];
#pragma unroll
  for (int k = 0; k < (ANYW ? 3 : 2); k++)
    lean_node_weight(lm.a[0], lm.b[0], ANYW && (lm.fl & 1), sum, k, w0[k], g0[k]);
  const bool wx = ANYW && (lm.fl & 1), wy = ANYW && (lm.fl & 2), wz = ANYW && (lm.fl & 4);
  auto row = [&](int k1, int k2, R W1, R G1, R W2, R G2) {
    const R* t = t0 + TL::RL * k1 + TL::zoff(bz + k2);
    const R W12 = W1 * W2, G1W2 = G1 * W2, W1G2 = W1 * G2;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const R va = t[d * TN], vb = t[d * TN + 1];
      R p = w0[0] * va + w0[1] * vb;
      R q = g0[0] * va + g0[1] * vb;
      R r = w0[0] * t[(3 + d) * TN] + w0[1] * t[(3 + d) * TN + 1];
      if (ANYW && wx) {
        const R vc = t[d * TN + 2];
        p += w0[2] * vc;
        q += g0[2] * vc;
        r += w0[2] * t[(3 + d) * TN + 2];
      }
      gs.du[d] += W12 * p;
      gs.dv[d] += W12 * r;
      gs.L[d][0] += W12 * q;
      gs.L[d][1] += G1W2 * p;
      gs.L[d][2] += W1G2 * p;
    }
  };
  if constexpr (!ANYW) {
    const R W1[2] = {lm.a[1], sum - lm.a[1]}, W2[2] = {lm.a[2], sum - lm.a[2]};
#pragma unroll
    for (int k2 = 0; k2 < 2; k2++)
#pragma unroll
      for (int k1 = 0; k1 < 2; k1++)
        row(k1, k2, W1[k1], k1 ? -lm.b[1] : lm.b[1], W2[k2], k2 ? -lm.b[2] : lm.b[2]);
  } else {
    const int K1 = any & 2 ? 3 : 2, K2 = any & 4 ? 3 : 2;
#pragma unroll 1
    for (int k2 = 0; k2 < K2; k2++) {
      R W2, G2;
      lean_node_weight(lm.a[2], lm.b[2], wz, sum, k2, W2, G2);
      const bool on2 = k2 < 2 || wz;
#pragma unroll 1
      for (int k1 = 0; k1 < K1; k1++) {
        if (!on2 || (k1 == 2 && !wy)) continue;
        R W1, G1;
        lean_node_weight(lm.a[1], lm.b[1], wy, sum, k1, W1, G1);
        row(k1, k2, W1, G1, W2, G2);
      }
    }
  }
#pragma unroll
  for (int d = 0; d < 3; d++) {
    gs.du[d] *= lm.sS;
    gs.dv[d] *= lm.sS;
#pragma unroll
    for (int b = 0; b < 3; b++) gs.L[d][b] *= lm.sG;
  }
  return gs;
}

// Shared memory of the scatter.
template <typename PT, int CAP>
struct LeanShared {
  PT* pts;           // staged points and records (column 0 of the item's first point)
  uint16_t* next;
  uint32_t* head;
  uint32_t* mask;    // kLeanMask words, then the count of far points
  uint8_t* cells;
  uint16_t* far;
};

// Points that the tile or the compact map does not hold (drift since the
// last binning, an upper corner on the domain's upper face) leave the fast
// path for a list, which the CTA works off node by node after the others:
// kept out of lean_point, their general loops do not cost it registers.
// kFarPoint: the whole point; kFarScatter: its scatter only.
constexpr uint16_t kFarPoint = 0, kFarScatter = 512;
template <typename PT, int CAP>
__device__ __forceinline__ void lean_far_push(const LeanShared<PT, CAP>& sh, int j, uint16_t kind) {
  const uint32_t k = atomicAdd(sh.mask + kLeanMask, 1u);
  sh.far[k] = (uint16_t)(j | kind);
}

// List entries: the point's index in the item (9 bits), the second-entry
// bits of its y and z axes (2 bits) and its map's flags (4 bits).
constexpr uint32_t kLeanEnd = 0xffffu;

// Point update from the gathered sums: movePoints, calculateStrainRate,
// updateDensity and updateStress. x, vd, vol and s6 hold the point's state
// before the step on entry, after it on exit (and in its arrays).
template <int MAT, typename PT>
__device__ __forceinline__ void lean_update(const BodyCtx<PT>& c, int64_t p, const GatherSum<PT>& gs, double* x,
                                            double* vd, const PT* u, PT& vol, PT* s6, PT m) {
  using R = PT;
  const PointsT<PT>& P = c.P;
  const R dt = (R)c.sp.dt;
  // movePoints (explicit_usl.cpp:279-292); the mixed form adds the
  // increments to its two-word x and x_t in FP64
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const R dx = dt * gs.du[d];
    x[d] = x[d] + (double)dx;
    vd[d] = vd[d] + (double)gs.dv[d];
    const R un = u[d] + dx;
    lean_store_two(P.x[d], P.xl[d], p, x[d]);
    lean_store_two(P.v[d], P.vl[d], p, vd[d]);
    P.u[d][p] = un;
  }
  vol = vol * exp(dt * (gs.L[0][0] + gs.L[1][1] + gs.L[2][2]));
  P.vol[p] = vol;
  if (c.mat.has_material) {
    lean_stress<3, MAT, R>(c, p, gs.L, s6, m, vol, dt);
#pragma unroll
    for (int k = 0; k < 6; k++) P.s[k][p] = s6[k];
  }
  if (P.L != nullptr) {
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int k = 0; k < 3; k++) P.L[9 * p + 3 * i + k] = (double)gs.L[i][k];
  }
}

// One point of the far list, node by node from and to global memory. A visit
// counts as drift where the window is outside the item's tile (origin o), not
// where only the compact map does not hold it.
template <bool NORMAL, int MAT, typename PT>
__device__ __forceinline__ void lean_far_point(const BodyCtx<PT>& c, int* err, unsigned long long* drift, int64_t p,
                                               bool whole, const int* o, const double* vref, int stepping) {
  using R = PT;
  const PointsT<PT>& P = c.P;
  const R ext = P.ext[p];
  double x[3], vd[3];
  R s6[6];
#pragma unroll
  for (int d = 0; d < 3; d++) x[d] = two_word(P.x[d], P.xl[d], p);
#pragma unroll
  for (int d = 0; d < 3; d++) vd[d] = two_word(P.v[d], P.vl[d], p);
  R vol = P.vol[p];
#pragma unroll
  for (int k = 0; k < 6; k++) s6[k] = P.s[k][p];
  PointMapT<R> pm;
  if (whole) {
    GatherSum<R> gs;
    if (build_map<3>(c.g, c.mc, c.sp.cpdi, x, ext, pm, err) > 0) {
      if (!window_in_tile<3>(pm, o, kLeanSide + 1)) atomicAdd(drift, 1ull);
      gs = gather_general<3, kLeanSide + 1, 1, false>(c, drift, pm, nullptr, (const R*)nullptr, vref);
      if constexpr (sizeof(PT) == 4) add_reference<3>(pm, vref, gs);
    }
    const R u[3] = {P.u[0][p], P.u[1][p], P.u[2][p]};
    lean_update<MAT>(c, p, gs, x, vd, u, vol, s6, MAT == 2 || MAT < 0 ? P.m[p] : R(0));
  }
  const int st = build_map<3>(c.g, c.mc, c.sp.cpdi, x, ext, pm, err);
  if (st < 0) P.active[p] = stepping ? 2 : 0;
  if (st <= 0) return;
  ScatterSrc<R> q;
  q.m = two_word(P.m, P.ml, p);
#pragma unroll
  for (int d = 0; d < 3; d++) q.mv[d] = q.m * vd[d];
  R vs[6];
#pragma unroll
  for (int k = 0; k < 6; k++) vs[k] = s6[k] * vol;
  const R V3[3][3] = {{vs[0], vs[3], vs[5]}, {vs[3], vs[1], vs[4]}, {vs[5], vs[4], vs[2]}};
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int k = 0; k < 3; k++) q.V3[i][k] = V3[i][k];
  if (!window_in_tile<3>(pm, o, kLeanSide + 1)) atomicAdd(drift, 1ull);
  scatter_general<3, kLeanSide + 1, 1, NORMAL, false, false>(c, drift, pm, nullptr, q, (double*)nullptr,
                                                             (uint8_t*)nullptr, nullptr);
}

// One point from gather to its record. `a` is its active state (1 active, 2
// left the domain at the last move), `col` its column of the staged arrays.
template <int T, int TN, int CAP, bool NORMAL, int MAT, typename PT>
__device__ __forceinline__ void lean_point(const BodyCtx<PT>& c, int* err, int64_t p, int j, int a, PT* col,
                                           const int* o, const PT* tvel, const double* vref,
                                           const LeanShared<PT, CAP>& sh, int do_g2p, int stepping) {
  using R = PT;
  constexpr int ROW = cap_row<CAP>();
  const PointsT<PT>& P = c.P;
  if (do_g2p && a == 2) {
    // left the domain at the last move; generateMap deactivates it now
    P.active[p] = 0;
    return;
  }
  const R ext = col[kFext * ROW];
  const R sG = map_grad_scale(c.g, ext);
  // Position in double (the mixed form's two words), velocity vd.
  double x[3], vd[3];
  R s6[6], vol;
#pragma unroll
  for (int d = 0; d < 3; d++) x[d] = lean_two<ROW>(col, kFx + d, kFxl + d);
  LeanMap<R> lm;
  if (do_g2p) {
    GatherSum<R> gs;
    const int st = lean_map<R>(c.g, c.mc, c.sp.cpdi, x, ext, sG, lm, err);
    if (st > 0) {
      if (st == 2 || !lean_in_tile<T>(lm, o)) {
        lean_far_push(sh, j, kFarPoint);
        return;
      }
      // over the lanes that are here together: each of them gets the mask that
      // names them all, and any such set gives a lane loops that cover its own bits
      const int any = __reduce_or_sync(__activemask(), lm.fl & 7);
      gs = any == 0 ? lean_gather<T, TN, false>(lm, o, tvel, 0) : lean_gather<T, TN, true>(lm, o, tvel, any);
      if constexpr (sizeof(PT) == 4) {
#pragma unroll
        for (int d = 0; d < 3; d++) gs.du[d] += (R)vref[d];
      }
    }
    R u[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      vd[d] = lean_two<ROW>(col, kFv + d, kFvl + d);
      u[d] = col[(kFu + d) * ROW];
    }
    vol = col[kFvol * ROW];
#pragma unroll
    for (int k = 0; k < 6; k++) s6[k] = col[(kFs + k) * ROW];
    lean_update<MAT>(c, p, gs, x, vd, u, vol, s6, MAT == 2 || MAT < 0 ? col[kFm * ROW] : R(0));
  } else {
#pragma unroll
    for (int d = 0; d < 3; d++) vd[d] = lean_two<ROW>(col, kFv + d, kFvl + d);
    vol = col[kFvol * ROW];
#pragma unroll
    for (int k = 0; k < 6; k++) s6[k] = col[(kFs + k) * ROW];
  }
  if (a != 1) return;
  // map build at the new position (mapPointsToNodes, explicit_usl.cpp:112-164;
  // contact normal, contact_huang.cpp:91)
  const int st = lean_map<R>(c.g, c.mc, c.sp.cpdi, x, ext, sG, lm, err);
  if (st < 0) {
    // outside the domain: inactive from the next map build on
    // (default_points.cpp:217-219); before the first step, at once
    P.active[p] = stepping ? 2 : 0;
    return;
  }
  if (st == 0) return;
  if (st == 2 || !lean_in_tile<T>(lm, o)) {
    lean_far_push(sh, j, kFarScatter);
    return;
  }
  // the record: the map's scales go into the sources once
  const double m = lean_two<ROW>(col, kFm, kFml);
  const double sm = (double)lm.sS * m;
  const R sv = lm.sG * vol;
  const double mm[4] = {sm, sm * vd[0], sm * vd[1], sm * vd[2]};
#pragma unroll
  for (int d = 0; d < 3; d++) {
    col[(kRab + 2 * d) * ROW] = lm.a[d];
    col[(kRab + 2 * d + 1) * ROW] = lm.b[d];
  }
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if constexpr (sizeof(PT) == 8) {
      col[(kRm + k) * ROW] = mm[k];
    } else {
      col[(kRm + 2 * k) * ROW] = __int_as_float(__double2loint(mm[k]));
      col[(kRm + 2 * k + 1) * ROW] = __int_as_float(__double2hiint(mm[k]));
    }
  }
#pragma unroll
  for (int k = 0; k < 6; k++) col[(kRs<PT> + k) * ROW] = sv * s6[k];
  if constexpr (NORMAL) col[kRgm<PT> * ROW] = lm.sG * (R)m;
  // A point wide along y (z) also enters the list of the next cell along
  // that axis, which holds its third node row.
  const int cell = (lm.base[0] - o[0]) + kLeanSide * ((lm.base[1] - o[1]) + kLeanSide * (lm.base[2] - o[2]));
  auto push = [&](int cl, int var) {
    const uint32_t e = (uint32_t)(j | (var << 9));
    const uint32_t old = atomicExch(sh.head + cl, e | ((uint32_t)lm.fl << 11));
    sh.next[e] = (uint16_t)old;
    if (old == kLeanEnd) atomicOr(sh.mask + (cl >> 5), 1u << (cl & 31));
  };
  push(cell, 0);
  if (lm.fl & 6) {
    if (lm.fl & 2) push(cell + kLeanSide, 1);
    if (lm.fl & 4) push(cell + kLeanSide * kLeanSide, 2);
    if ((lm.fl & 6) == 6) push(cell + kLeanSide * (kLeanSide + 1), 3);
  }
}

// The sums of one node row (offset ky, kz from the cell) over the cell's
// list, added into the global accumulators.
template <int CAP, bool NORMAL, typename PT>
__device__ __forceinline__ void lean_row(const BodyCtx<PT>& c, const LeanShared<PT, CAP>& sh, int cell, int row,
                                         const int* o, bool on) {
  using R = PT;
  constexpr int NV = fused_nacc(NORMAL);
  constexpr int ROW = cap_row<CAP>();
  const int ky = row & 1, kz = row >> 1;
  double acc[3][NV];
#pragma unroll
  for (int n = 0; n < 3; n++)
#pragma unroll
    for (int v = 0; v < NV; v++) acc[n][v] = 0.0;
  const R sy = ky ? R(-1) : R(1), cy = ky ? R(2) : R(0), sz = kz ? R(-1) : R(1), cz = kz ? R(2) : R(0);
  bool third = false;
  uint32_t e = on ? sh.head[cell] : kLeanEnd;
  while (e != kLeanEnd) {
    const uint32_t en = sh.next[e & 2047u];
    const R* col = sh.pts + (e & 511u);
    R a[3], b[3], s[6];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      a[d] = col[(kRab + 2 * d) * ROW];
      b[d] = col[(kRab + 2 * d + 1) * ROW];
    }
    double mm[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if constexpr (sizeof(PT) == 8)
        mm[k] = col[(kRm + k) * ROW];
      else
        mm[k] = __hiloint2double(__float_as_int(col[(kRm + 2 * k + 1) * ROW]), __float_as_int(col[(kRm + 2 * k) * ROW]));
    }
#pragma unroll
    for (int k = 0; k < 6; k++) s[k] = col[(kRs<PT> + k) * ROW];
    R W1 = sy * a[1] + cy, G1 = sy * b[1], W2 = sz * a[2] + cz, G2 = sz * b[2];
    R w0 = a[0], w1 = R(2) - a[0], g0 = b[0], g1 = -b[0];
    const uint32_t fl = e >> 11;
    if (fl != 0) {
      const R sum = fl & kLeanSampled ? R(1) : R(2);
      const int vy = (int)((e >> 9) & 1u), vz = (int)((e >> 10) & 1u);
      lean_node_weight(a[1], b[1], (fl & 2u) != 0, sum, ky + vy, W1, G1);
      lean_node_weight(a[2], b[2], (fl & 4u) != 0, sum, kz + vz, W2, G2);
      // a second entry's first row is the first entry's second
      if (vy && !ky) W1 = G1 = R(0);
      if (vz && !kz) W2 = G2 = R(0);
      lean_node_weight(a[0], b[0], (fl & 1u) != 0, sum, 0, w0, g0);
      lean_node_weight(a[0], b[0], (fl & 1u) != 0, sum, 1, w1, g1);
    }
    const R W12 = W1 * W2, G1W2 = G1 * W2, W1G2 = W1 * G2;
    // nodal force -V sigma . grad S = -(g A + w B) along the row
    const R A[3] = {s[0] * W12, s[3] * W12, s[5] * W12};
    const R B[3] = {s[3] * G1W2 + s[5] * W1G2, s[1] * G1W2 + s[4] * W1G2, s[4] * G1W2 + s[2] * W1G2};
    auto node = [&](int n, R w, R g) {
      const double S = (double)(w * W12);
      acc[n][0] += S * mm[0];
#pragma unroll
      for (int d = 0; d < 3; d++) {
        acc[n][1 + d] += S * mm[1 + d];
        if constexpr (sizeof(PT) == 8) {
          acc[n][4 + d] -= g * A[d];
          acc[n][4 + d] -= w * B[d];
        } else {
          acc[n][4 + d] -= (double)(g * A[d] + w * B[d]);
        }
      }
      if constexpr (NORMAL) {
        const R gm = col[kRgm<PT> * ROW];
        acc[n][7] += (double)(g * W12 * gm);
        acc[n][8] += (double)(w * G1W2 * gm);
        acc[n][9] += (double)(w * W1G2 * gm);
      }
    };
    node(0, w0, g0);
    node(1, w1, g1);
    if (fl & 1u) {
      node(2, b[0], b[0]);   // the third node's weight and gradient weight
      third = true;
    }
    e = en;
  }
  // A cell's second node is the first of the next cell along x: where that
  // is the next quad of the warp it takes over the sums (its third node's go
  // two quads on), which leaves one node per row and cell to add to L2
  // (measured 1 % on the column, 2 % on the block drops).
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int prev = __shfl_up_sync(full, on ? cell : -9, 4);
  const bool adj = on && lane >= 4 && prev + 1 == cell && cell % kLeanSide != 0;
  const bool taken = __shfl_down_sync(full, adj ? 1 : 0, 4) != 0 && lane < 28;
  if (__any_sync(full, third)) {
#pragma unroll
    for (int v = 0; v < NV; v++) {
      const double u = __shfl_up_sync(full, acc[2][v], 4);
      if (adj) acc[1][v] += u;
    }
  }
#pragma unroll
  for (int v = 0; v < NV; v++) {
    const double u = __shfl_up_sync(full, acc[1][v], 4);
    if (adj) acc[0][v] += u;
  }
  if (!on) return;
  const int i = o[0] + cell % kLeanSide, j = o[1] + (cell / kLeanSide) % kLeanSide + ky,
            k = o[2] + cell / (kLeanSide * kLeanSide) + kz;
#pragma unroll
  for (int n = 0; n < 3; n++) {
    if (n >= 1 && taken) break;
    if (n == 2 && !third) break;
    const int64_t s = node_slot(c.g, i + n, j, k);
    c.flags[s >> 6] = 1u;
    atomicAdd(c.A.m + s, acc[n][0]);
#pragma unroll
    for (int d = 0; d < 3; d++) {
      atomicAdd(c.A.mx[d] + s, acc[n][1 + d]);
      atomicAdd(c.A.f[d] + s, acc[n][4 + d]);
      if constexpr (NORMAL) atomicAdd(c.A.nrm[d] + s, acc[n][7 + d]);
    }
  }
}

template <int DIM, typename PT, int NT, int PPT, bool NORMAL, bool SINGLE, int MAT>
__global__ void __launch_bounds__(NT, lean_min_ctas<PT, NT, PPT>())
    k_g2p2g_lean(const __grid_constant__ FusedLaunch<PT> fl) {
  constexpr int B = fused_bin<DIM>();
  constexpr int T = B + 3;
  constexpr int TN = fused_tile_nodes<DIM, B>();
  constexpr int CAP = NT * PPT;
  constexpr int ROW = cap_row<CAP>();
  constexpr int AL = 16 / (int)sizeof(PT);   // elements per 16 bytes
  static_assert(DIM == 3 && T == kLeanSide + 1 && CAP <= 512, "list entries and cells are laid out for these");
  constexpr uint32_t kCtxBytes = (uint32_t)ctx_bytes<PT>();
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t* bar_ctx = reinterpret_cast<uint64_t*>(smem + 8);   // table entry slots 0, 1
  auto slot_ctx = [&](int i) { return reinterpret_cast<BodyCtx<PT>*>(smem + kOffCtx + (size_t)i * kCtxBytes); };
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem);   // point arrays
  PT* tvel = reinterpret_cast<PT*>(smem + lean_off_tvel<DIM, PT>());
  PT* pts = reinterpret_cast<PT*>(smem + lean_off_pts<DIM, PT>());
  int32_t* act = reinterpret_cast<int32_t*>(smem + lean_off_act<DIM, PT, CAP>());
  LeanShared<PT, CAP> sh;
  sh.next = reinterpret_cast<uint16_t*>(smem + lean_off_next<DIM, PT, CAP>());
  sh.head = reinterpret_cast<uint32_t*>(smem + lean_off_head<DIM, PT, CAP>());
  sh.mask = sh.head + kLeanCells;
  sh.far = reinterpret_cast<uint16_t*>(smem + lean_off_far<DIM, PT, CAP>());
  sh.cells = smem + lean_off_far<DIM, PT, CAP>() + sizeof(uint16_t) * CAP;

  publish_counts(fl);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    mbar_init(bar_ctx, 1);
    mbar_init(bar_ctx + 1, 1);
    mbar_init_fence();
  }
  __syncthreads();
  uint32_t parity = 0;
  // the tile nodes this thread loads: slots threadIdx.x + i NT, packed
  // tx | ty << 8 | tz << 16 (-1: none)
  // Launches over the table keep them in registers, one-body launches form
  // them per item (column 393 -> 386 us per step; 21 block drops 656 -> 672).
  constexpr int TI = (TN + NT - 1) / NT;
  int tnode[TI];
#pragma unroll
  for (int i = 0; i < TI && !SINGLE; i++) {
    const int t = (int)threadIdx.x + i * NT;
    int tx, ty, tz;
    tnode[i] = t < TN && TileLayout<DIM, T>::node(t, tx, ty, tz) ? tx | ty << 8 | tz << 16 : -1;
  }
  const int nwork = SINGLE ? fl.nwork_body[fl.one_body] : *fl.nwork;
  // launches over every body: the table entry of each work item arrives by
  // a bulk copy issued one item ahead (slot k & 1 for the CTA's k-th item)
  if (!SINGLE && threadIdx.x == 0 && (int)blockIdx.x < nwork) {
    mbar_arrive_expect_tx(bar_ctx, kCtxBytes);
    bulk_copy_g2s(slot_ctx(0), fl.bodies + fl.flat_body[blockIdx.x], kCtxBytes, bar_ctx);
  }
  // the CTA's next item (claim_item) and its index in the work list, slot
  // k & 1 for its k-th item: written by thread 0 before a barrier of the
  // item, read by every thread after it
  __shared__ int next_item[2], next_id[2];

  auto bin_origin = [&](const BodyCtx<PT>& c, int bin, int* o) {
    const int r = bin / c.bg.nbx;
    o[0] = (bin % c.bg.nbx) * B - 1;
    o[1] = (r % c.bg.nby) * B - 1;
    o[2] = (r / c.bg.nby) * B - 1;
  };
  // starts the copies of the bin's nodal velocities into the tile
  double* traw = sizeof(PT) == 8 ? reinterpret_cast<double*>(tvel)
                                 : reinterpret_cast<double*>(smem + lean_off_traw<DIM, PT>());
  const int lane = threadIdx.x & 31;
  const bool copier = threadIdx.x >= NT - 32;   // the warp that issues the bulk copies
  auto load_tile = [&](const BodyCtx<PT>& c, const int* o) {
    const Geom& g = c.g;
#pragma unroll
    for (int i = 0; i < TI; i++) {
      int tx, ty, tz;
      if constexpr (SINGLE) {
        const int t0 = (int)threadIdx.x + i * NT;
        if (!(t0 < TN && TileLayout<DIM, T>::node(t0, tx, ty, tz))) continue;
      } else {
        if (tnode[i] < 0) continue;
        tx = tnode[i] & 255;
        ty = (tnode[i] >> 8) & 255;
        tz = tnode[i] >> 16;
      }
      const int x = o[0] + tx, y = o[1] + ty, z = o[2] + tz;
      if (x < 0 || y < 0 || z < 0 || x >= g.nn[0] || y >= g.nn[1] || z >= g.nn[2]) continue;
      const int64_t s = node_slot(g, x, y, z);
      double* t = traw + threadIdx.x + i * NT;
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        async_copy8(t + d * TN, c.V.vt[d] + s);
        async_copy8(t + (3 + d) * TN, c.V.dv[d] + s);
      }
    }
  };

  int id = 0, bin = 0, start = 0, end = 0;   // the current item
  if ((int)blockIdx.x < nwork) {
    id = SINGLE ? fl.item_off[fl.one_body] + (int)blockIdx.x : fl.flat_item[blockIdx.x];
    bin = fl.work_bin[id];
    start = fl.work_start[id];
    end = fl.work_end[id];
  }
  bool tile_ahead = false;   // the current item's tile copies were started during the previous item
  int k = 0;
  for (int w = blockIdx.x; w < nwork; k++) {
    // thread 0 claims the next item now and publishes it (and, over the
    // table, starts the copy of its entry) before the item's first barrier,
    // so that the claim's latency overlaps the item's own copies
    int wn = SINGLE ? w + (int)gridDim.x : 0;
    bool ahead = false;   // thread 0: the next entry's copy is in flight
    if (!SINGLE && threadIdx.x == 0) wn = claim_item(fl.queue);
    auto publish_next = [&]() {
      if (SINGLE || threadIdx.x != 0) return;
      next_item[k & 1] = wn;
      if (wn < nwork) {
        next_id[k & 1] = fl.flat_item[wn];
        // the other slot was last read by the previous item (all threads
        // passed its closing barrier)
        const int other = (k & 1) ^ 1;
        fence_async_shared();
        mbar_arrive_expect_tx(bar_ctx + other, kCtxBytes);
        bulk_copy_g2s(slot_ctx(other), fl.bodies + fl.flat_body[wn], kCtxBytes, bar_ctx + other);
        ahead = true;
      }
    };
    // the next item's description: loads issued after the first barrier,
    // used at the end of the item
    int nid = 0, nbin = 0, nstart = 0, nend = 0;
    auto read_next = [&]() {
      if (!SINGLE) wn = next_item[k & 1];
      if (wn >= nwork) return;
      nid = SINGLE ? id + (int)gridDim.x : next_id[k & 1];
      nbin = fl.work_bin[nid];
      nstart = fl.work_start[nid];
      nend = fl.work_end[nid];
    };
    auto advance = [&]() {
      w = wn;
      id = nid;
      bin = nbin;
      start = nstart;
      end = nend;
    };
    if (!SINGLE) {
      const int slot = k & 1;
      const bool got = mbar_wait_bounded(bar_ctx + slot, (uint32_t)((k >> 1) & 1), fl.err, fl.wait_polls);
      if (__syncthreads_or(got ? 0 : 1)) {
        // let the copies in flight land before leaving (the next entry's
        // copy is not issued yet)
        async_copy_wait();
        if (threadIdx.x == 0) {
          if (!got) mbar_wait_bounded(bar_ctx + slot, (uint32_t)((k >> 1) & 1), fl.err);
          queue_done(fl.queue);
        }
        return;
      }
    }
    const BodyCtx<PT>& c = SINGLE ? fl.one : *slot_ctx(k & 1);
    const int prime = c.prime;
    // items of the other kind (contact normal or not) belong to the other
    // launch, and a priming pass takes the bodies still to prime only
    auto skipped = [&](const BodyCtx<PT>& b) {
      return (!SINGLE && (b.needs_normal != 0) != NORMAL) || (fl.prime_pass && !b.prime);
    };
    if (skipped(c)) {
      publish_next();
      __syncthreads();
      read_next();
      advance();
      __syncthreads();   // every thread has read the staged entry and the next item
      continue;
    }
    const int do_g2p = (prime || !(fl.phases & 1)) ? 0 : 1;
    const PointsT<PT>& P = c.P;
    const int64_t pstart = start;
    const int n = end - start;
    if (n > CAP && threadIdx.x == 0) atomicOr(fl.err, kErrItemCap);   // the work list was cut for another size
    // the item's point arrays: one bulk copy per array by the lanes of the
    // last warp (16-byte aligned windows)
    const int64_t sp0 = pstart & ~(int64_t)(AL - 1), s4 = pstart & ~(int64_t)3;
    const int offp = (int)(pstart - sp0), off4 = (int)(pstart - s4);
    if (copier) {
      const int nc = n < CAP ? n : CAP;
      const uint32_t bytes = (uint32_t)(((offp + nc + AL - 1) & ~(AL - 1)) * sizeof(PT));
      const uint32_t bytes4 = (uint32_t)((off4 + nc + 3) & ~3) * 4u;
      // orders the previous item's accesses (before its closing barrier)
      // before the copies' writes
      fence_async_shared();
      if (lane == 0) mbar_arrive_expect_tx(bar, lean_rows<PT>() * bytes + bytes4);
      __syncwarp();
      if (lane < lean_rows<PT>())
        bulk_copy_g2s(pts + lane * ROW, lean_array(P, lane) + sp0, bytes, bar);
      else if (lane == lean_rows<PT>())
        bulk_copy_g2s(act, P.active + s4, bytes4, bar);
    }
    sh.pts = pts + offp;
    int o[3];
    bin_origin(c, bin, o);
    if (do_g2p && !tile_ahead) load_tile(c, o);
    for (int t = threadIdx.x; t < kLeanCells + kLeanMask + 1; t += NT) sh.head[t] = t < kLeanCells ? kLeanEnd : 0u;
    publish_next();
    async_copy_wait();
    const bool arrived = mbar_wait_bounded(bar, parity, fl.err, fl.wait_polls);
    // one decision for the whole CTA (also the barrier after the tile copies)
    if (__syncthreads_or(arrived ? 0 : 1)) {
      // let copies in flight land before leaving
      if (!arrived) mbar_wait_bounded(bar, parity, fl.err);
      if (threadIdx.x == 0) {
        if (ahead) mbar_wait_bounded(bar_ctx + ((k & 1) ^ 1), (uint32_t)(((k + 1) >> 1) & 1), fl.err);
        if (!SINGLE) queue_done(fl.queue);
      }
      return;
    }
    parity ^= 1u;
    read_next();
    // reference velocity of the mixed form: the item's first point (any
    // value is exact; one close to the item's velocities keeps the
    // differences small)
    double vref[3] = {0.0, 0.0, 0.0};
    if constexpr (sizeof(PT) == 4) {
      if (do_g2p) {
#pragma unroll
        for (int d = 0; d < DIM; d++) vref[d] = (double)sh.pts[(kFv + d) * ROW];
        for (int t = threadIdx.x; t < TN; t += NT) {
#pragma unroll
          for (int d = 0; d < DIM; d++) {
            tvel[d * TN + t] = (PT)(traw[d * TN + t] - vref[d]);
            tvel[(3 + d) * TN + t] = (PT)traw[(3 + d) * TN + t];
          }
        }
        __syncthreads();
      }
    }
#pragma unroll 1
    for (int r = 0; r < PPT; r++) {
      const int j = (int)threadIdx.x + r * NT;
      const int a = j < n ? act[off4 + j] : 0;
      if (a != 0)
        lean_point<T, TN, CAP, NORMAL, MAT>(c, fl.err, pstart + j, j, a, sh.pts + j, o, tvel, vref, sh, do_g2p,
                                            prime ? 0 : 1);
    }
    __syncthreads();
    // the tile is free: the next item's copies run during the scatter
    tile_ahead = false;
    if (wn < nwork) {
      bool entry = true;
      if (!SINGLE) entry = mbar_wait_bounded(bar_ctx + ((k & 1) ^ 1), (uint32_t)(((k + 1) >> 1) & 1), fl.err);
      const BodyCtx<PT>& cn = SINGLE ? fl.one : *slot_ctx((k & 1) ^ 1);
      if (entry && !skipped(cn) && !(cn.prime || !(fl.phases & 1))) {
        int on[3];
        bin_origin(cn, nbin, on);
        load_tile(cn, on);
        tile_ahead = true;
      }
    }
    // the non-empty cells, in cell order (x fastest)
    int ncell = 0;
    {
      uint32_t m[kLeanMask];
#pragma unroll
      for (int w = 0; w < kLeanMask; w++) {
        m[w] = sh.mask[w];
        ncell += __popc(m[w]);
      }
      for (int cl = threadIdx.x; cl < kLeanCells; cl += NT) {
        int pos = 0;
        bool on = false;
#pragma unroll
        for (int w = 0; w < kLeanMask; w++) {
          const uint32_t below = cl >= 32 * (w + 1) ? 0xffffffffu : (cl < 32 * w ? 0u : (1u << (cl & 31)) - 1u);
          pos += __popc(m[w] & below);
          if ((cl >> 5) == w) on = (m[w] >> (cl & 31)) & 1u;
        }
        if (on) sh.cells[pos] = (uint8_t)cl;
      }
    }
    __syncthreads();
    // four lanes per cell: the record a quad reads is one address, which one
    // shared-memory wavefront serves
    for (int t = threadIdx.x; (t & ~31) < 4 * ncell; t += NT) {
      const bool on = t < 4 * ncell;
      lean_row<CAP, NORMAL>(c, sh, on ? sh.cells[t >> 2] : 0, t & 3, o, on);
    }
    const int nfar = (int)sh.mask[kLeanMask];
    for (int t = threadIdx.x; t < nfar; t += NT) {
      const int f = sh.far[t];
      int fo[3];   // o, formed again: held through the row sums it costs 10 us of the column's step
      bin_origin(c, bin, fo);
      lean_far_point<NORMAL, MAT>(c, fl.err, fl.drift, pstart + (f & 511), f < kFarScatter, fo, vref,
                                  prime ? 0 : 1);
    }
    advance();
    __syncthreads();
  }
  if (!SINGLE && threadIdx.x == 0) queue_done(fl.queue);
}

}  // namespace mpmb200
