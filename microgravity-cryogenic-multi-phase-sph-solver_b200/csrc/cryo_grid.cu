// cryo_grid.cu -- uniform-grid neighbour search on the GPU: integer cell keys,
// a stable counting sort by cell, the dense cell table and the reorder gather.
// Replaces SpatialHash::build / reorder_particles (spatial_hash.cu:48-138).
#include <type_traits>

#include "cryo_kernels.cuh"

namespace cryo {

// Cell keys (spatial_hash.cu:61-68): dead particles get the sentinel
// num_cells so they sort to the end.
__global__ void k_keys(Params P, View V, CellSort S) {
  const int n = V.dyn->n;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 xp = V.xp[i];
    count_key(S, i, ph_of(xp) == kDead ? (uint32_t)P.num_cells : (uint32_t)cell_index(P, xyz(xp)));
  }
}

// ------------------------------------------------------------- cell sort
// The stable sort by cell key as a counting sort over the dense cells, whose
// prefix sums are the cell table the passes need anyway:
//   1. the key kernel counts the particles of every cell and notes which
//      number each particle drew (the order of the draws is arbitrary);
//   2. k_cell_scan: exclusive prefix sums of the counts, kScanCells cells per
//      block, and (last block) of the blocks' totals;
//   3. k_cell_scatter: particle index and key to the cell's range, in drawn
//      order; the finished cell table;
//   4. k_cell_order: inside its cell a particle's place is the number of
//      smaller indices there, which makes the result the stable sort whatever
//      the draws were.
// Three launches whatever the number of cells, 24 bytes of traffic and 16 of
// memory per cell: a dam break of 27 k particles steps in 103 us in 5 k cells,
// 114 in 0.9 M, 173 in 5 M, 806 in 35 M, 5.3 ms in 256 M.  A tank's cell holds
// about 18 particles, so step 4 reads one or two cache lines per particle; it
// is quadratic in a cell's particles, as the list build is (8 000 particles
// thrown beyond the domain into its edge cells: the step takes 296 us).
__global__ void __launch_bounds__(kScanThreads) k_cell_scan(Params P, CellSort S, uint32_t* __restrict__ cell_kinds,
                                                            unsigned* ticket) {
  constexpr int kPer = kScanCells / kScanThreads;
  static_assert(kPer == 8, "8 cells per thread");
  __shared__ int wtot[kScanThreads / 32];
  const int cells = P.num_cells + 1;  // the sentinel too
  const int blocks = (cells + kScanCells - 1) / kScanCells;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // exclusive prefix of one value per thread over the block; `total` to all
  auto block_scan = [&](int v, int& total) {
    int incl = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) wtot[warp] = incl;
    __syncthreads();
    int before = 0;
    total = 0;
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; ++w) {
      const int t = wtot[w];
      if (w < warp) before += t;
      total += t;
    }
    __syncthreads();
    return before + incl - v;
  };
  for (int b = blockIdx.x; b < blocks; b += gridDim.x) {
    // the arrays hold a multiple of kPer entries, zero beyond the last cell
    const int base = b * kScanCells + threadIdx.x * kPer;
    int c[kPer], sum = 0;
#pragma unroll
    for (int q = 0; q < kPer; q += 4) {
      const int4 v = base < cells ? *reinterpret_cast<const int4*>(S.count + base + q) : make_int4(0, 0, 0, 0);
      c[q] = v.x; c[q + 1] = v.y; c[q + 2] = v.z; c[q + 3] = v.w;
    }
#pragma unroll
    for (int q = 0; q < kPer; ++q) sum += c[q];
    int total;
    int run = block_scan(sum, total);
    if (base < cells) {
#pragma unroll
      for (int q = 0; q < kPer; q += 4) {
        int4 v;
        v.x = run; v.y = v.x + c[q]; v.z = v.y + c[q + 1]; v.w = v.z + c[q + 2];
        run = v.w + c[q + 3];
        *reinterpret_cast<int4*>(S.local + base + q) = v;
        *reinterpret_cast<int4*>(S.count + base + q) = make_int4(0, 0, 0, 0);  // ready for the next build
        if (P.use_lists) *reinterpret_cast<uint4*>(cell_kinds + base + q) = make_uint4(0u, 0u, 0u, 0u);
      }
    }
    if (threadIdx.x == 0) S.sums[b] = total;
  }
  if (last_block(ticket)) {
    int carry = 0;
    for (int b0 = 0; b0 < blocks; b0 += kScanThreads) {
      const int b = b0 + threadIdx.x;
      const int v = b < blocks ? __ldcg(S.sums + b) : 0;
      int total;
      const int pre = block_scan(v, total);
      if (b < blocks) S.sums[b] = carry + pre;
      carry += total;
    }
  }
}

__global__ void __launch_bounds__(kBlock) k_cell_scatter(Params P, CellSort S, DynState* dyn,
                                                         int* __restrict__ cell_begin) {
  const int n = dyn->n, nc = P.num_cells;
  const int first = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  for (int i = first; i < n; i += step) {
    const uint32_t key = S.key[i];
    const int at = S.local[key] + S.sums[key / kScanCells] + (int)S.slot[i];
    S.drawn[at] = (uint32_t)i;
    S.sorted_key[at] = key;
  }
  for (int c = first; c <= nc; c += step) {
    const int b = S.local[c] + S.sums[c / kScanCells];
    cell_begin[c] = b;
    if (c == nc) dyn->n_alive = b;
  }
}

__global__ void __launch_bounds__(kBlock) k_cell_order(Params P, CellSort S, const DynState* __restrict__ dyn,
                                                       const int* __restrict__ cell_begin) {
  const int n = dyn->n_alive;  // the dead are dropped by the gather
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const uint32_t key = S.sorted_key[p];
    const uint32_t i = S.drawn[p];
    const int b = __ldg(cell_begin + key), e = __ldg(cell_begin + key + 1);
    int smaller = 0;
    for (int q = b; q < e; ++q) smaller += __ldg(S.drawn + q) < i;
    S.perm[b + smaller] = i;
  }
}

// Reorder gather of the persistent arrays (spatial_hash.cu:116-138), fused
// into one pass: dst[i] = src[perm[i]] for i < n_alive; then n = n_alive.
// Also counts the owned fluid and wall particles per chunk (every particle
// unless the context is one slab of a tank); the last block turns the counts
// into the chunk offsets of the ordered phase index lists (partials rows 0
// and 1) and their lengths.
__global__ void __launch_bounds__(kBlock) k_gather(Params P, View src, View dst, const uint32_t* __restrict__ perm,
                                                   const uint32_t* __restrict__ cells, Reduce R, int reset_maxima) {
  __shared__ double sh[2 * kBlock / 32];
  DynState* dyn = src.dyn;
  // the step's maxima start over for the force pass to come (the step size
  // was taken from them by the launch before the sort)
  if (reset_maxima && blockIdx.x == 0 && threadIdx.x == 0) {
    dyn->v_max = 0.0f;
    dyn->a_max = 0.0f;
    dyn->Tv_max = 0.0f;
    dyn->nu_t_max = 0.0f;
    dyn->spacing_ratio = 1.0f;
    if (P.heat_power == 0.0f) dyn->heat_inv_norm = 0.0f;  // no heater: no pass of this step sets it
  }
  const int na = dyn->n_alive;
  const int nch = num_chunks(na);
  int own_lo, own_hi;
  owned_layers(P, src.cell_begin, own_lo, own_hi);
  for (int c = blockIdx.x; c < nch; c += gridDim.x) {
    const int i = c * kChunk + threadIdx.x;
    double cnt[2] = {0.0, 0.0};
    if (i < na) {
      const uint32_t j = perm[i];
      const float4 xp = src.xp[j];
      dst.xp[i] = xp;
      dst.vT[i] = src.vT[j];
      dst.vt[i] = src.vt[j];
      dst.nrm[i] = src.nrm[j];
      dst.mrps[i] = src.mrps[j];
      dst.id[i] = src.id[j];
      const int ph = ph_of(xp);
      const bool own = i >= own_lo && i < own_hi;
      if (is_fluid(ph) && own) cnt[0] = 1.0;
      else if (ph == kWall && own) cnt[1] = 1.0;
      if (P.use_lists && ph <= kWall) reinterpret_cast<uint8_t*>(dst.cell_kinds + cells[i])[ph] = 1;
    }
    publish_chunk<2>(R, c, cnt, sh);
  }
  if (last_block(R.ticket)) {
    const double nf = block_exclusive_scan(R, 0, nch);
    const double nw = block_exclusive_scan(R, 1, nch);
    if (threadIdx.x == 0) {
      dyn->n_fluid_list = (int)nf;
      dyn->n_wall_list = (int)nw;
      dyn->n = na;
    }
  }
}

// Ordered index lists of the owned fluid and wall particles: for the chunk of
// particle `first`, the entries of the particles the block itself handles
// (kBlock / L of them, `first` on), from the gather's chunk offsets and the
// particles' ranks inside the chunk.
template <int L>
__device__ inline void phase_lists(const Params& P, const View& V, const Reduce& R, int n, int first) {
  __shared__ int wcnt[2][kBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = first / kChunk;
  const int p = c * kChunk + threadIdx.x;
  int own_lo, own_hi;
  owned_layers(P, V.cell_begin, own_lo, own_hi);
  const int ph = p < n ? ph_of(V.xp[p]) : kDead;
  const bool own = p >= own_lo && p < own_hi;
  const bool isf = own && is_fluid(ph), isw = own && ph == kWall;
  const unsigned bf = __ballot_sync(0xffffffffu, isf), bw = __ballot_sync(0xffffffffu, isw);
  if (lane == 0) {
    wcnt[0][warp] = __popc(bf);
    wcnt[1][warp] = __popc(bw);
  }
  __syncthreads();
  if (p >= first && p < first + kBlock / L) {
    int pf = 0, pw = 0;
    for (int w = 0; w < warp; ++w) {
      pf += wcnt[0][w];
      pw += wcnt[1][w];
    }
    const unsigned lt = (1u << lane) - 1u;
    if (isf) V.fluid_idx[(int)__ldcg(R.partials + c) + pf + __popc(bf & lt)] = p;
    if (isw) V.wall_idx[(int)__ldcg(R.partials + R.max_chunks + c) + pw + __popc(bw & lt)] = p;
  }
  __syncthreads();
}
__device__ inline uint8_t near_bits(uint32_t kinds) {
  return (uint8_t)((kinds & kCellLiquid ? kNearLiquid : 0) | (kinds & kCellVapor ? kNearVapor : 0) |
                   (kinds & kCellWall ? kNearWall : 0));
}
// The candidates [s, e) of row of cells row9 (0-8, z-major) of the 27-cell
// block, and the kinds of its cells added to `kinds`.  whole: every cell of
// the row (positions that moved after the sort may have left their cell, and
// lanes of one cell then walk the same ranges); otherwise the cells beyond
// the support are dropped, as the cell scan does.  A wall keeps fluid
// neighbours only, so a row of cells without fluid is empty for it.
__device__ inline void list_row(const Params& P, const View& V, const CellWindow& W, int row9, bool whole, bool wall_i,
                                int& s, int& e, uint32_t& kinds) {
  s = e = 0;
  const int z = W.cz + row9 / 3 - 1, y = W.cy + row9 % 3 - 1;
  if (row9 >= 9 || z < W.z0 || z > W.z1 || y < W.y0 || y > W.y1) return;
  int xs = W.x0, xe = W.x1;
  if (!whole && !W.row(P, y, z, xs, xe)) return;
  const int row = (z * P.ny + y) * P.nx;
  uint32_t k = 0;
  for (int x = xs; x <= xe; ++x) k |= __ldg(V.cell_kinds + row + x);
  kinds |= k;
  if (wall_i && !(k & (kCellLiquid | kCellVapor))) return;
  s = __ldg(V.cell_begin + row + xs);
  e = __ldg(V.cell_begin + row + xe + 1);
}

// Neighbour lists of every particle in the reference's iteration order
// (for_each_neighbor filtered by r^2 < support^2, self included), with the
// kinds of cells around each particle.  A wall's list holds its fluid
// neighbours only: every pass that walks a wall's neighbours (the wall
// boundary pass and its reverse) skips the other walls, so the fluid entries
// in their order are all it needs.  mode LISTS_PHASE also fills the ordered
// fluid / wall index lists.
//
// L = 1: a thread per particle, every lane on the same row at the same time.
// An accepted candidate costs no branch: every candidate's index is stored at
// the next place of the thread's ring of sixteen in shared memory (a column
// per thread, no bank conflicts), and acceptance moves the place on.  After
// every eight candidates the threads with a full chunk write it out as one
// 32-byte sector.
// L = LIST_LANES: the lanes share a particle (small tanks, where a thread's
// walk over ~470 candidates sets the time): sixteen candidates per round,
// four consecutive ones per lane, a prefix sum over the lanes for the places,
// the list put together in shared memory and written in whole chunks.
template <int L>
__global__ void __launch_bounds__(kBlock, L == 1 ? 5 : 4) k_build_lists(Params P, View V, Reduce R, int mode) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int kRing = 2 * kNbrChunk;
  constexpr int kStride = kMaxNbr + 4;  // the pad takes what a longer list would add, and spreads the banks
  constexpr int kPer = kBlock / L;  // particles per block
  __shared__ __align__(16) int stage[L == 1 ? kRing * kPer : kPer * kStride];
  DynState* dyn = V.dyn;
  const int n = dyn->n;
  const int lane = threadIdx.x & 31;
  unsigned overflow = 0;
  for (int first = blockIdx.x * kPer; first < n; first += gridDim.x * kPer) {
    if (mode != LISTS_ONLY) phase_lists<L>(P, V, R, n, first);
    const int i = first + threadIdx.x / L;
    const bool valid = i < n;
    const float4 xpi = V.xp[valid ? i : n - 1];
    const V3 xi = xyz(xpi);
    const bool wall_i = ph_of(xpi) == kWall;
    uint32_t kinds = 0;
    int cnt = 0;
    if constexpr (L == 1) {
      if (!valid) continue;
      int* const column = stage + threadIdx.x;
      auto flush = [&](int q) {  // chunk q out of its half of the ring
        if (q >= kMaxNbr / kNbrChunk) return;
        const int* h = column + (q & 1) * kNbrChunk * kPer;
        int4* dst = reinterpret_cast<int4*>(V.nbr + ((size_t)q * V.capacity + i) * kNbrChunk);
        dst[0] = make_int4(h[0], h[kPer], h[2 * kPer], h[3 * kPer]);
        dst[1] = make_int4(h[4 * kPer], h[5 * kPer], h[6 * kPer], h[7 * kPer]);
      };
      int flushed = 0;  // chunks written
      auto scan = [&](auto wall_c) {
        constexpr bool kWallI = decltype(wall_c)::value;
        const CellWindow W(P, xi);
        for (int row9 = 0; row9 < 9; ++row9) {
          int s, e;
          list_row(P, V, W, row9, true, kWallI && wall_i, s, e, kinds);
          for (int j = s; j < e; j += 8) {
            // beyond the row's end: loaded (the array is padded), not accepted
#pragma unroll
            for (int h = 0; h < 8; h += 4) {
              float4 x[4];
#pragma unroll
              for (int u = 0; u < 4; ++u) x[u] = __ldg(V.xp + j + h + u);
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                bool in = norm2(xi - xyz(x[u])) < P.support2 && j + h + u < e;
                if (kWallI) in = in && (!wall_i || is_fluid(ph_of(x[u])));
                column[(cnt & (kRing - 1)) * kPer] = j + h + u;
                cnt += in ? 1 : 0;
              }
            }
            if (cnt - flushed * kNbrChunk >= kNbrChunk) flush(flushed++);
          }
        }
      };
      // a warp with a wall tests the phase for all its particles
      if (__any_sync(__activemask(), wall_i)) scan(std::true_type{});
      else scan(std::false_type{});
      if (cnt > flushed * kNbrChunk) flush(flushed);  // the last, partial chunk
    } else {
      const int sub = lane & (L - 1), lead = lane & ~(L - 1);
      int* const list = stage + (threadIdx.x / L) * kStride;
      constexpr int kRowsPer = (9 + L - 1) / L;
      int rs[kRowsPer], re[kRowsPer];  // rows sub, sub + L, ...: first and end candidate
      {
        const CellWindow W(P, xi);
#pragma unroll
        for (int q = 0; q < kRowsPer; ++q)
          list_row(P, V, W, valid ? q * L + sub : 9, mode == LISTS_ONLY, wall_i, rs[q], re[q], kinds);
      }
#pragma unroll
      for (int row9 = 0; row9 < 9; ++row9) {
        const int s = __shfl_sync(kAll, rs[row9 / L], lead + row9 % L);
        const int e = __shfl_sync(kAll, re[row9 / L], lead + row9 % L);
        for (int f = s; __any_sync(kAll, f < e); f += 4 * L) {
          const int j = f + 4 * sub;
          float4 x[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) x[u] = __ldg(V.xp + min(j + u, n - 1));
          bool in[4];
          int c = 0;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            in[u] = j + u < e && norm2(xi - xyz(x[u])) < P.support2 && (!wall_i || is_fluid(ph_of(x[u])));
            c += in[u];
          }
          int upto = c;  // accepted by the lanes up to this one
#pragma unroll
          for (int o = 1; o < L; o <<= 1) {
            const int t = __shfl_up_sync(kAll, upto, o, L);
            if (sub >= o) upto += t;
          }
          int k = min(cnt + upto - c, kMaxNbr);
          cnt += __shfl_sync(kAll, upto, lead + L - 1);
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (in[u]) list[k++] = j + u;
        }
      }
#pragma unroll
      for (int o = 1; o < L; o <<= 1) kinds |= __shfl_xor_sync(kAll, kinds, o);
      __syncwarp();
      if (valid) {
        const int chunks = (min(cnt, kMaxNbr) + kNbrChunk - 1) / kNbrChunk;
        for (int q = sub; q < chunks; q += L) {
          const int4* src = reinterpret_cast<const int4*>(list + q * kNbrChunk);
          int4* dst = reinterpret_cast<int4*>(V.nbr + ((size_t)q * V.capacity + i) * kNbrChunk);
          dst[0] = src[0];
          dst[1] = src[1];
        }
      }
      __syncwarp();  // the shared list is free again
      if (!valid || sub != 0) continue;
    }
    V.nbr_cnt[i] = cnt;
    if (mode != LISTS_ONLY) V.near_kinds[i] = near_bits(kinds);
    if (cnt > kMaxNbr) overflow = CRYO_DEV_NBR_OVERFLOW;
  }
  if (overflow) atomicOr(&dyn->status, overflow);
}
template __global__ void k_build_lists<1>(Params, View, Reduce, int);
template __global__ void k_build_lists<LIST_LANES>(Params, View, Reduce, int);

// Neighbour list dump (test hook): counts, then the lists at given offsets.
// stored = 0: the cell scan (every neighbour); 1: the lists of the last
// build, as the passes walk them (walls: their fluid neighbours only).
__global__ void k_nbr_count(Params P, View V, int stored, int* __restrict__ counts) {
  const int n = V.dyn->n;
  P.use_lists = stored;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int c = 0;
    for_each_nbr(P, V, i, xyz(V.xp[i]), [&](int, float4, V3, float) { ++c; });
    counts[i] = c;
  }
}
__global__ void k_nbr_fill(Params P, View V, int stored, const long long* __restrict__ offsets,
                           int* __restrict__ list) {
  const int n = V.dyn->n;
  P.use_lists = stored;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    long long o = offsets[i];
    for_each_nbr(P, V, i, xyz(V.xp[i]), [&](int j, float4, V3, float) { list[o++] = j; });
  }
}

}  // namespace cryo
