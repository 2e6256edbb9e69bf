// cryo_grid.cu -- uniform-grid neighbour search on the GPU: integer cell keys,
// a stable counting sort by cell, the dense cell table and the reorder gather.
// Replaces SpatialHash::build / reorder_particles (spatial_hash.cu:48-138).
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
// Three launches whatever the number of cells (the radix sort before it took
// three per 8-bit digit and a fourth kind for the table).  A tank's cell holds
// about 18 particles, so step 4 reads one or two cache lines per particle.
__global__ void __launch_bounds__(kScanThreads) k_cell_scan(Params P, CellSort S, uint8_t* __restrict__ cell_fluid,
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
      }
      if (P.use_lists) *reinterpret_cast<uint2*>(cell_fluid + base) = make_uint2(0u, 0u);
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
                                                   Reduce R, int reset_maxima) {
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
      if (P.use_lists && is_fluid(ph)) dst.cell_fluid[cell_index(P, xyz(xp))] = 1;
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

// Neighbour lists of every particle in the reference's iteration order
// (for_each_neighbor filtered by r^2 < support^2, self included), stored
// transposed so a warp reads consecutive words.  mode LISTS_PHASE also fills
// the ordered fluid / wall index lists from the gather's chunk offsets.
__global__ void __launch_bounds__(kBlock, LIST_MIN_BLOCKS) k_build_lists(Params P, View V, Reduce R, int mode) {
  __shared__ int wcnt[2][kBlock / 32];
  // each thread gathers a chunk of kNbrChunk entries here and stores it as
  // one full 32-byte sector (column per thread: no bank conflicts)
  __shared__ int stage[kNbrChunk][kBlock];
#pragma unroll
  for (int q = 0; q < kNbrChunk; ++q) stage[q][threadIdx.x] = 0;  // the unused tail of a last chunk
  DynState* dyn = V.dyn;
  const int n = dyn->n;
  const int nch = num_chunks(n);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned overflow = 0;
  for (int c = blockIdx.x; c < nch; c += gridDim.x) {
    const int i = c * kChunk + threadIdx.x;
    const bool valid = i < n;
    const float4 xpi = valid ? V.xp[i] : make_float4(0, 0, 0, 0);
    const int ph = valid ? ph_of(xpi) : kDead;
    if (mode != LISTS_ONLY) {
      // ordered phase lists of the owned particles: chunk offset + rank inside the chunk
      int own_lo, own_hi;
      owned_layers(P, V.cell_begin, own_lo, own_hi);
      const bool own = i >= own_lo && i < own_hi;
      const bool isf = valid && own && is_fluid(ph), isw = valid && own && ph == kWall;
      const unsigned bf = __ballot_sync(0xffffffffu, isf), bw = __ballot_sync(0xffffffffu, isw);
      if (lane == 0) {
        wcnt[0][warp] = __popc(bf);
        wcnt[1][warp] = __popc(bw);
      }
      __syncthreads();
      int pf = 0, pw = 0;
      for (int w = 0; w < warp; ++w) {
        pf += wcnt[0][w];
        pw += wcnt[1][w];
      }
      const unsigned lt = (1u << lane) - 1u;
      if (isf) V.fluid_idx[(int)__ldcg(R.partials + c) + pf + __popc(bf & lt)] = i;
      if (isw) V.wall_idx[(int)__ldcg(R.partials + R.max_chunks + c) + pw + __popc(bw & lt)] = i;
      __syncthreads();
    }
    if (!valid) continue;
    const V3 xi = xyz(xpi);
    int cnt = 0;
    const int t = threadIdx.x;
    int4* chunk = reinterpret_cast<int4*>(V.nbr + (size_t)i * kNbrChunk);
    const size_t cstride = (size_t)V.capacity * (kNbrChunk / 4);  // in int4
    auto store_chunk = [&](int q) {
      int4* dst = chunk + (size_t)q * cstride;
      dst[0] = make_int4(stage[0][t], stage[1][t], stage[2][t], stage[3][t]);
      dst[1] = make_int4(stage[4][t], stage[5][t], stage[6][t], stage[7][t]);
    };
    // A wall's list holds its fluid neighbours only: every pass that walks
    // a wall's neighbours (the wall boundary pass and its reverse) skips the
    // other walls, so the fluid entries in their order are all it needs;
    // rows of cells with no fluid are not scanned.
    const bool wall_i = ph == kWall;
    const CellWindow W(P, xi);
    for (int z = W.z0; z <= W.z1; ++z) {
      for (int y = W.y0; y <= W.y1; ++y) {
        // every row of the 27-cell block, whole: lanes in one cell then walk
        // the same ranges (dropping rows beyond the support radius, as the
        // cell scan does, saves candidates but splits the warp more)
        const int xs = W.x0, xe = W.x1;
        const int row = (z * P.ny + y) * P.nx;
        if (wall_i) {
          bool any = false;
          for (int x = xs; x <= xe; ++x) any |= V.cell_fluid[row + x] != 0;
          if (!any) continue;
        }
        const int s = __ldg(V.cell_begin + row + xs);
        const int e = __ldg(V.cell_begin + row + xe + 1);
        // candidates in groups of LIST_GROUP: all loads issued before the
        // tests, so a thread has that many positions in flight
        auto test = [&](const float4& xj, int j) {
          const V3 rij = xi - xyz(xj);
          const float r2 = norm2(rij);
          if (r2 < P.support2 && (!wall_i || is_fluid(ph_of(xj)))) {
            if (cnt < kMaxNbr) {
              stage[cnt & (kNbrChunk - 1)][t] = j;
              if ((cnt & (kNbrChunk - 1)) == kNbrChunk - 1) store_chunk(cnt / kNbrChunk);
            }
            ++cnt;
          }
        };
        int j = s;
        for (; j + LIST_GROUP <= e; j += LIST_GROUP) {
          float4 xg[LIST_GROUP];
#pragma unroll
          for (int u = 0; u < LIST_GROUP; ++u) xg[u] = __ldg(V.xp + j + u);
#pragma unroll
          for (int u = 0; u < LIST_GROUP; ++u) test(xg[u], j + u);
        }
        for (; j < e; ++j) test(__ldg(V.xp + j), j);
      }
    }
    if (cnt < kMaxNbr && (cnt & (kNbrChunk - 1)) != 0) store_chunk(cnt / kNbrChunk);  // partial last chunk
    V.nbr_cnt[i] = cnt;
    if (cnt > kMaxNbr) overflow = CRYO_DEV_NBR_OVERFLOW;
  }
  if (overflow) atomicOr(&dyn->status, overflow);
}

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
