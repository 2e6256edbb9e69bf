// cryo_kernels.cuh -- declarations of the device kernels (one definition file
// each: cryo_grid.cu, cryo_physics.cu, cryo_phase.cu, cryo_control.cu).
#pragma once

#include "cryo_common.cuh"

namespace cryo {

// Cells per block of the cell-table scan.
constexpr int kScanThreads = 256;
constexpr int kScanCells = 2048;

// Arrays of the sort by cell key (cryo_grid.cu).
struct CellSort {
  uint32_t *key, *slot;          // per particle: its cell, its number among the cell's draws
  uint32_t *sorted_key, *drawn;  // per sorted place: the cell, the particle in drawn order
  uint32_t* perm;                // per sorted place: the particle of the stable sort (reuses slot's storage)
  int *count, *local, *sums;     // per cell: particles (zero between builds), prefix in its block; per block: prefix
};
// Key of particle i, counted: lanes of the warp that share a cell draw their
// numbers with one atomic (neighbours in the previous order mostly do).
__device__ inline void count_key(const CellSort& S, int i, uint32_t key) {
  const unsigned peers = __match_any_sync(__activemask(), key);
  const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(S.count + key, __popc(peers));
  base = __shfl_sync(peers, base, leader);
  S.key[i] = key;
  S.slot[i] = (uint32_t)(base + __popc(peers & ((1u << lane) - 1u)));
}

// Layout of the FP64 partials of one reduction: partials[v * max_chunks + c].
struct Reduce {
  double* partials;
  unsigned* ticket;
  int max_chunks;
};


// Last-block ticket: true in exactly one block, after every block of the grid
// has published its partials (each block fences before taking a ticket).
__device__ inline bool last_block(unsigned* ticket) {
  __shared__ bool is_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) is_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (is_last && threadIdx.x == 0) *ticket = 0u;  // ready for the next launch
  return is_last;
}
// Compensated two-sum accumulation (Neumaier).
__device__ inline void neumaier(double& s, double& c, double x) {
  const double t = s + x;
  c += fabs(s) >= fabs(x) ? (s - t) + x : (x - t) + s;
  s = t;
}
// (s, c) += (s2, c2) for compensated pairs: two-sum of the heads, the
// rounding error and both tails into the tail.
__device__ inline void neumaier_pair(double& s, double& c, double s2, double c2) {
  const double t = s + s2;
  c += (fabs(s) >= fabs(s2) ? (s - t) + s2 : (s2 - t) + s) + c2;
  s = t;
}
// Sum of value v over chunks [0, nchunks), computed by the whole (last) block
// in a fixed order that depends on nothing but nchunks: thread t sums chunks
// t, t + blockDim, ... (compensated), the 32 lanes of a warp combine in a
// fixed down-shift tree, and thread 0 combines the warps in order.  Every
// thread of the block must call it; the result is valid in thread 0.
// Compensated sum of p[k] for k = k0, k0 + step, ... below n, in that order;
// the loads go out kBatch at a time ahead of the additions, so a thread
// waits on one round trip per batch instead of one per element.
__device__ inline void strided_neumaier(const double* p, int k0, int step, int n, double& s, double& c) {
  constexpr int kBatch = 8;
  for (int kb = k0; kb < n; kb += kBatch * step) {
    double x[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int k = kb + u * step;
      x[u] = k < n ? __ldcg(p + k) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u)
      if (kb + u * step < n) neumaier(s, c, x[u]);
  }
}
__device__ inline double block_sum_partials(const Reduce& R, int v, int nchunks) {
  __shared__ double ws[kBlock / 32], wc[kBlock / 32];
  double s = 0, c = 0;
  const double* p = R.partials + (size_t)v * R.max_chunks;
  strided_neumaier(p, threadIdx.x, blockDim.x, nchunks, s, c);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double s2 = __shfl_down_sync(0xffffffffu, s, o), c2 = __shfl_down_sync(0xffffffffu, c, o);
    neumaier_pair(s, c, s2, c2);  // lanes >= 32 - o combine garbage that lane 0 never sees
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    ws[warp] = s;
    wc[warp] = c;
  }
  __syncthreads();
  double r = 0;
  if (threadIdx.x == 0) {
    double S = ws[0], C = wc[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) neumaier_pair(S, C, ws[w], wc[w]);
    r = S + C;
  }
  __syncthreads();
  return r;
}
// Sum of value v over chunks [0, nchunks) by one warp, in a fixed order that
// depends on nothing but nchunks: lane l sums chunks l, l + 32, ...
// (compensated), then a fixed down-shift tree.  The result is valid in lane 0.
// Several warps of a block can each take their own values at once.
__device__ inline double warp_sum_partials(const Reduce& R, int v, int nchunks) {
  const int lane = threadIdx.x & 31;
  double s = 0, c = 0;
  const double* p = R.partials + (size_t)v * R.max_chunks;
  strided_neumaier(p, lane, 32, nchunks, s, c);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double s2 = __shfl_down_sync(0xffffffffu, s, o), c2 = __shfl_down_sync(0xffffffffu, c, o);
    neumaier_pair(s, c, s2, c2);
  }
  return s + c;
}
// In-place exclusive scan of the (integral) chunk values of row v by the whole
// block; returns the total (all threads).  Integral doubles add exactly, so
// the parallel order gives the serial result.
__device__ inline double block_exclusive_scan(const Reduce& R, int v, int nchunks) {
  __shared__ double wtot[kBlock / 32];
  __shared__ double total;
  double* p = R.partials + (size_t)v * R.max_chunks;
  const int per = (nchunks + blockDim.x - 1) / blockDim.x;
  const int lo = threadIdx.x * per, hi = min(lo + per, nchunks);
  double seg = 0;
  for (int k = lo; k < hi; ++k) seg += __ldcg(p + k);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double x = seg;  // inclusive scan over the warp
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wtot[warp] = x;
  __syncthreads();
  if (threadIdx.x == 0) {
    double run = 0;
    for (int w = 0; w < nw; ++w) {
      const double t = wtot[w];
      wtot[w] = run;
      run += t;
    }
    total = run;
  }
  __syncthreads();
  double run = wtot[warp] + (x - seg);
  for (int k = lo; k < hi; ++k) {
    const double y = __ldcg(p + k);
    p[k] = run;
    run += y;
  }
  const double t = total;
  __syncthreads();
  return t;
}
// Writes the block sums of NV values (one per thread each) for chunk c:
// every warp reduces its lanes, then lane k of warp 0 adds value k's warp
// sums in warp order (from 0.0, one after another) and stores it, so the
// values are finished side by side rather than one after another by one
// thread; each value's additions are the same either way.  `sh` must hold
// NV * (blockDim / 32) doubles; every thread of the block must call it.
template <int NV>
__device__ inline void publish_chunk(const Reduce& R, int c, double (&v)[NV], double* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = warp_sum(v[k]);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) sh[k * nw + warp] = v[k];
  __syncthreads();
  if (warp == 0)
    for (int k = lane; k < NV; k += 32) {
      double s = 0;
      for (int w = 0; w < nw; ++w) s += sh[k * nw + w];
      R.partials[(size_t)k * R.max_chunks + c] = s;
    }
  __syncthreads();  // sh is free again
}
// Sums over neighbours that L lanes visit side by side (NbrRounds): every lane
// brings its neighbour's terms t, and each sum takes the lanes' terms one
// after another in lane order -- the neighbours' order -- so that every lane
// holds the sums a single thread walking the list would have.  Every lane of
// the warp must take part.
template <int L, int K>
__device__ inline void add_terms(float (&s)[K], const float (&t)[K]) {
  const int lead = L > 1 ? (threadIdx.x & 31) & ~(L - 1) : 0;
#pragma unroll
  for (int u = 0; u < L; ++u)
#pragma unroll
    for (int k = 0; k < K; ++k) s[k] += L > 1 ? __shfl_sync(0xffffffffu, t[k], lead + u) : t[k];
}
__device__ inline int num_chunks(int n) { return (n + kChunk - 1) / kChunk; }

// grid (cryo_grid.cu)
__global__ void k_keys(Params P, View V, CellSort S);
__global__ void k_cell_scan(Params P, CellSort S, uint32_t* cell_kinds, unsigned* ticket);
__global__ void k_cell_scatter(Params P, CellSort S, DynState* dyn, int* cell_begin);
__global__ void k_cell_order(Params P, CellSort S, const DynState* dyn, const int* cell_begin);
__global__ void k_gather(Params P, View src, View dst, const uint32_t* perm, const uint32_t* cells, Reduce R, int reset_maxima);
enum { LISTS_ONLY = 0, LISTS_PHASE = 1 };
template <int L>
__global__ void k_build_lists(Params P, View V, Reduce R, int mode);
__global__ void k_nbr_count(Params P, View V, int stored, int* counts);
__global__ void k_nbr_fill(Params P, View V, int stored, const long long* offsets, int* list);

// physics (cryo_physics.cu).  Fused rate pass; `what` selects the sub-passes (FORCE_* bits).
enum { FORCE_TRANSPORT = 1, FORCE_MOMENTUM = 2, FORCE_CSF = 4, FORCE_AKINCI = 8, FORCE_DRHO = 16,
       FORCE_THERMAL = 32, FORCE_MAXIMA = 64, FORCE_THERMAL_ALWAYS = 128,
       FORCE_TAPE = 256,      // compile-time only: also store the sums into V.tape
       FORCE_COMMON = 512 };  // compile-time only: the rarer options are off (cryo_physics.cu)
// cryo_physics.cu is compiled twice.  namespace exact: the reference's IEEE
// single-precision operation sequence (no FMA contraction, IEEE division and
// square root), bit-identical to its CPU build.  namespace fast: the same
// source with FMA contraction and the approximate (2 ulp) division and square
// root, as the reference's own CUDA build contracts; fields then agree with
// the exact sequence to ~1e-6 relative per pass.  The neighbour lists, keys
// and sort are not in that file, so they stay bit-exact in both.
#define CRYO_FIELD_KERNELS                                                           \
  __global__ void k_density(Params P, View V, int fuse_eos);                        \
  __global__ void k_aux(Params P, View V);                                          \
  __global__ void k_normalize_masses(Params P, View V);                             \
  __global__ void k_eos(Params P, View V);                                          \
  __global__ void k_wall(Params P, View V);                                         \
  template <int TAPE>                                                               \
  __global__ void k_interface(Params P, View V, int sorted);                        \
  __global__ void k_sps(Params P, View V);                                          \
  __global__ void k_smooth_normals(Params P, View V);                               \
  template <int WHAT>                                                               \
  __global__ void k_forces_t(Params P, View V, int what_rt);                        \
  __global__ void k_maxima(Params P, View V);                                       \
  __global__ void k_shift_compute(Params P, View V);                                \
  __global__ void k_shift_apply(Params P, View V);                                  \
  template <int LANES>                                                              \
  __global__ void k_probe(Params P, View V, const float* pts, int np, float* out);
namespace exact {
CRYO_FIELD_KERNELS
}
namespace fast {
CRYO_FIELD_KERNELS
}
// cryo_lanes.cu: the exact passes with PASS_LANES lanes per particle.
namespace lanes {
__global__ void k_density(Params P, View V);
__global__ void k_wall(Params P, View V);
template <int TAPE>
__global__ void k_interface(Params P, View V, int sorted);
template <int WHAT>
__global__ void k_forces_t(Params P, View V);
}
// TAPE: also store the sums into V.tape (the recomputation of a differentiated window).
constexpr int INTERFACE_BLOCK = 128;
constexpr int FORCE_BASE = FORCE_TRANSPORT | FORCE_MOMENTUM | FORCE_MAXIMA;
// Block shape of the force pass.  The pass is bound by the latency of each
// particle's neighbour chain, so what matters is how many particles are in
// flight at once.  Asking for 9 resident 64-thread blocks per SM makes the
// compiler fit 5 warps in each SM sub-partition's register file (96
// registers), 20 warps per SM: the 82k fluid particles of the dam break run
// in one wave.  A 112-register cap fits only 4 warps per sub-partition (16
// per SM) and needs two waves, 30 % slower there.
#ifndef FORCES_BLOCK
#define FORCES_BLOCK 64
#endif
#ifndef FORCES_MIN_BLOCKS
#define FORCES_MIN_BLOCKS 9
#endif
// The sub-pass sets with surface tension or heat take 8 blocks per SM (4 warps
// per sub-partition, 128 registers); the instances with FORCE_COMMON 10 (96):
// 778 us against 874 at 1.06 M particles in the fast arithmetic, 3619 against
// 3842 at 4.08 M in the exact one.  Some of them spill 4-48 bytes at 10 (the
// exact sets with the density rate, and the fast CSF with heat) and are still
// ahead of their general instances at 8: CSF with heat and density rate 1027 us
// against 1270 at 729 k fluid particles, CSF with density rate 972 against
// 1181, heat with density rate 709 against 841 at 405 k.  At 12 they spill more
// (963 and 4599 us).
#ifndef FORCES_MIN_BLOCKS_HEAVY
#define FORCES_MIN_BLOCKS_HEAVY 8
#endif
#ifndef FORCES_MIN_BLOCKS_COMMON
#define FORCES_MIN_BLOCKS_COMMON 10
#endif
constexpr int forces_min_blocks(int what) {
  return !(what >= 0 && (what & (FORCE_CSF | FORCE_THERMAL))) ? FORCES_MIN_BLOCKS
         : what & FORCE_COMMON                                ? FORCES_MIN_BLOCKS_COMMON
                                                              : FORCES_MIN_BLOCKS_HEAVY;
}
// Neighbour-loop unroll of the force-pass variants with surface tension or
// heat (the two-phase tanks): 2 takes the 4 M-particle LH2 sphere 3 % faster.
#ifndef FORCES_UNROLL_HEAVY
#define FORCES_UNROLL_HEAVY 2
#endif
// Neighbour-list build: LIST_LANES lanes per particle up to LIST_LANES_MAX
// particles, one above (k_build_lists).  One thread against lanes, us: 42 / 39
// at 37 k particles, 52 / 57 at 55 k, 50 / 47 at 60 k (free surface, twice the
// walls), 60 / 74 at 85 k.  In an ensemble other members' kernels fill the chip
// meanwhile, and the members together may hold LIST_LANES_MAX_BESIDE fluid
// particles (a wall's list is short, so the fluid sets the work).  Step of all,
// one thread / lanes, exact and fast, by fluid particles together: two-phase
// tanks 32 k 323 / 315 and 380 / 385, 47 k 451 / 450 and 444 / 447, 55 k 572 /
// 586 and 522 / 518, 59 k 480 / 492 and 439 / 455; dam breaks 34 k 275 / 273 and
// 319 / 310, 53 k 360 / 360 and 345 / 344, 65 k 354 / 373 and 348 / 361.
constexpr int LIST_LANES = 4;
constexpr int kListPad = 8;  // records the build may load beyond the last particle
#ifndef LIST_LANES_MAX
#define LIST_LANES_MAX 60000
#endif
#ifndef LIST_LANES_MAX_BESIDE
#define LIST_LANES_MAX_BESIDE 56000
#endif
// The neighbour passes that come in two shapes, one thread per particle and
// PASS_LANES lanes per particle, take the second up to these counts (fluid
// particles; walls for the wall pass; in an ensemble those of the tanks that
// step side by side).  Lanes shorten the chain of a particle's ~75 neighbours
// but add shuffles and rows, so they pay while the chip has room for the
// threads.  One thread against lanes, us per launch in the exact arithmetic
// (event overhead of ~5 us included), boxes at 4 mm:
//   fluid particles       1 000   13 800   32 800    54 900    74 100   97 300  125 000  157 500
//   force pass, 2 phases 148/37   149/58  163/101   174/153   187/196  199/249  217/316  253/395
//   density               27/15    31/20    33/32     35/44     35/55    40/71    42/86   50/110
//   vapour rebalance      33/17    37/21    40/31     41/43     42/49    44/63    56/74    59/94
//   interface, 2 phases   69/21    70/27    76/42     81/54     84/67    87/75    89/96   90/100
//   ph.-change normalize  29/13    29/14    42/17     42/17     42/20    43/21    44/21    34/21
//   phase-change apply    37/18    39/19    50/27     50/29     51/35    51/44    52/48    47/56
//   fluid, free surface   2 300    18 400   30 300    55 000    70 000   87 700  107 800  161 200
//   force pass           117/31    131/59   142/95   165/150   184/189  194/236  271/285  318/427
//   force pass, Akinci        -    262/84  273/117   291/185   301/226  331/278  439/325        -
//   interface             54/18     56/24    58/27     58/36     61/42    61/46    66/50    68/64
//   interface, Akinci         -     78/41    80/55     84/83    89/102   94/124   98/145        -
//   walls                 2 900    12 800   22 100    30 300    35 600   42 600   49 900   57 800
//   wall pass, 2 phases   19/13     21/13    21/19     21/21     21/23    23/27    22/29    23/33
//   wall pass, 1 phase        -     20/13    21/13     21/15     21/17    21/19    21/21    23/23
// The interface pass crosses late where only walls count (no vapour), early in
// Akinci's model, which sums over every neighbour.  The force pass's line is
// the step's: with lanes 280 -> 275 us at 48 400 fluid particles (free surface),
// 419 -> 380 at 46 700 (two phases), but 288 -> 299 at 55 000 (free surface).
// In an ensemble the wall pass has lines of its own (step of all, one thread /
// lanes): two-phase tanks 246 / 241 at 30 000 walls together, 253 / 246 at
// 34 800, 294 / 293 at 40 000, 366 / 389 at 58 000; dam breaks 156 / 152 at
// 60 500, 181 / 179 at 78 000, 207 / 207 at 88 000, 198 / 203 at 100 000.
constexpr int PASS_LANES = 8;
constexpr int FORCES_LANED_BLOCK = 128;
#ifndef FORCES_LANES_MAX
#define FORCES_LANES_MAX 50000
#endif
#ifndef PASS_LANES_MAX  // density, vapour rebalance
#define PASS_LANES_MAX 40000
#endif
#ifndef PC_LANES_MAX  // phase-change normalize and apply
#define PC_LANES_MAX 130000
#endif
#ifndef INTERFACE_LANES_MAX
#define INTERFACE_LANES_MAX 110000
#endif
#ifndef INTERFACE_LANES_MAX_WALLS  // no vapour: walls only
#define INTERFACE_LANES_MAX_WALLS 130000
#endif
#ifndef INTERFACE_LANES_MAX_AKINCI
#define INTERFACE_LANES_MAX_AKINCI 55000
#endif
#ifndef WALL_LANES_MAX
#define WALL_LANES_MAX 30000
#endif
#ifndef WALL_LANES_MAX_LIQUID  // no vapour
#define WALL_LANES_MAX_LIQUID 57000
#endif
#ifndef WALL_LANES_MAX_BESIDE
#define WALL_LANES_MAX_BESIDE 38000
#endif
#ifndef WALL_LANES_MAX_BESIDE_LIQUID
#define WALL_LANES_MAX_BESIDE_LIQUID 85000
#endif

// Points a pressure probe gives a warp each; more take a thread each.  A warp
// shortens a point's chain but adds its ~75 terms one after another for 32
// lanes.  Kernel, us, warps against threads (27 k / 204 k / 840 k particles):
//   random points, 1 024    17 / 17 / 17      against  206 / 266 / 269
//   a lattice,    32 768    80 / 94 / 97               102 / 126 / 209
//   a lattice,    64 000   150 / 168 / 181             110 / 157 / 226
//   a lattice, 1 061 208  2249 / 2682 / 2802           659 / 959 / 1188
#ifndef PROBE_WARPS_MAX
#define PROBE_WARPS_MAX 32768
#endif

// integrator + phase change (cryo_phase.cu)
__global__ void k_kick_drift(Params P, View V, int continuity, int tvf);
enum { KICK_SOURCES = 1, KICK_HEAT = 2 };
__global__ void k_kick(Params P, View V, int flags);
__global__ void k_pc_sources(Params P, View V);
template <int L>
__global__ void k_pc_normalize(Params P, View V, int gated);
template <int L>
__global__ void k_pc_apply(Params P, View V, Reduce R, int gated);
template <int L>
__global__ void k_rebalance1(Params P, View V, int gated);
__global__ void k_rebalance2_mark(Params P, View V, Reduce R, uint32_t* flag, int rebalance, int gated);
__global__ void k_split(Params P, View V, Reduce R, const uint32_t* flag, int gated);
__global__ void k_venting(Params P, View V, Reduce R, float relax, int gated);
__global__ void k_scale_velocities(View V, float factor, int scale_vmax);

// step control + reductions (cryo_control.cu)
enum { BEGIN_STEP = 0, BEGIN_RATES = 1 };
__global__ void k_begin_step(Params P, View V, int mode);
__global__ void k_heat_norm(Params P, View V, Reduce R);
__global__ void k_heat_sum(Params P, View V, Reduce R);
// The ullage pressure and saturation temperature from the phase sums
// (sph_solver.cu:586-607).
__device__ inline void saturation_update(const Params& P, DynState* d, bool closed, double m_liq, double m_vap,
                                         double mT_vap) {
  bool done = false;
  if (closed) {
    if (!(d->fluid_volume0 > 0)) d->fluid_volume0 = m_liq / P.f_rho_l + m_vap / P.f_rho_v;
    const double v_ullage = d->fluid_volume0 - m_liq / P.f_rho_l;
    const double ratio = v_ullage > 0 && m_vap > 0 ? (mT_vap / v_ullage) / ((double)P.f_rho_v * P.f_T_sat) : 0.0;
    if (isfinite(ratio) && ratio > 0) {
      d->p_ullage = P.f_p_sat * ratio;
      // FluidProperties::saturation_temperature (fluid_properties.cpp:7-10)
      const float p = (float)d->p_ullage;
      const double inv_T = 1.0 / P.f_T_sat - ((double)P.f_R_gas / P.f_h_fg) * log((double)p / P.f_p_sat);
      d->T_sat = (float)(1.0 / inv_T);
      done = true;
    }
  }
  if (!done) {
    d->p_ullage = P.f_p_sat;
    d->T_sat = P.f_T_sat;
  }
}
__global__ void k_saturation(Params P, View V, Reduce R, int end_of_step);
__global__ void k_begin_kick_drift_keys(Params P, View V, CellSort S);
__global__ void k_kick_saturation(Params P, View V, Reduce R);
__global__ void k_diagnostics(Params P, View V, Reduce R, double* out);

// Packed per-particle telemetry record (telemetry.hpp:28-31).
struct TelemetryRecord {
  float x, y, z, T, p, speed;
  uint32_t phase;
};
__global__ void k_telemetry_pack(View V, TelemetryRecord* out);

// Number of FP64 values per chunk of the diagnostics reduction.
constexpr int kDiagValues = 30;

// tank lattice generator (cryo_setup.cu)
constexpr int kGeomNodes = CRYO_GEOM_MAX_NODES;
// One geometry node with the offsets of its Translated ancestors, root first
// (applied to the query point in that order, as the nested sdf calls do).
struct GeomNode {
  int kind, a, b, nofs;
  double p[3];
  double ofs[kGeomNodes][3];
};
// Lattice nodes at ((i0 + i + 1/2) h, ...), i < nx, ...; band = wall_layers h.
// Slab decomposition of one tank (cryo_slab.cu).
__global__ void k_slab_bounds(Params P, View V, int zb, int ze);
__global__ void k_halo_pull(Params P, View dst, View src, int z);
__global__ void k_slab_heat(Params P, DynState* const* dyns, int nslabs, DynState* mine, int heat_mode);
__global__ void k_slab_split(DynState* const* dyns, int nslabs, int rank, DynState* mine);
__global__ void k_slab_end(Params P, DynState* const* dyns, int nslabs, DynState* mine, int saturation);
__global__ void k_slab_assemble(Params P, View dst, float4* a4_out, float4* ab4_out, View lo, View me, View up,
                                int has_lo, int has_up, int zb, int ze, int depth);
__global__ void k_slab_commit(View V, const float4* a4_in, const float4* ab4_in);

struct Lattice {
  int i0, j0, k0, nx, ny, nz;
  long long total;
  double h, band;
};
// Fill of the generated tank: key direction or centre, the liquid cut, the
// per-phase mass, density and temperature, the heater band.
struct FillDev {
  int mode, include_vapor, any_liquid;
  float g[3], c[3];
  double cut;
  float m_liq, m_vap, rho_liq, rho_vap, T_liq, T_vap, T_wall;
  double heater_zmin, heater_zmax;
};
__global__ void k_lattice_classify(const GeomNode* G, int ng, Lattice L, uint8_t* cls, uint32_t* cnt_f,
                                   uint32_t* cnt_w);
__global__ void k_scan_counts(uint32_t* cnt, int n, unsigned long long* total);
__global__ void k_lattice_scatter(Lattice L, const uint8_t* cls, const uint32_t* off_f, const uint32_t* off_w,
                                  long long* fluid_nodes, long long* wall_nodes);
__global__ void k_fill_keys(Lattice L, FillDev F, const long long* fluid_nodes, int nf, uint32_t* keys);
__global__ void k_key_digits(const uint32_t* keys, int n, uint32_t prefix, uint32_t mask, int shift,
                             unsigned int* hist);
__global__ void k_fill_split(Lattice L, FillDev F, const long long* fluid_nodes, int nf, uint8_t* liquid,
                             uint32_t* cnt_keep, uint32_t* cnt_liq);
__global__ void k_emit_walls(const GeomNode* G, int ng, Lattice L, FillDev F, const long long* wall_nodes, int nw,
                             View V);
__global__ void k_jitter_fluid(View V, int n, float amplitude, uint64_t seed);
__global__ void k_emit_fluid(Lattice L, FillDev F, const long long* fluid_nodes, int nf, const uint8_t* liquid,
                             const uint32_t* off_keep, int nw, View V);

}  // namespace cryo
