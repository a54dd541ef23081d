// The phases of the one-launch cell-list build (celllist.cu).
#pragma once

#include "uph_internal.cuh"

namespace uph {

template <typename T>
__device__ __forceinline__ T block_exclusive_scan(T v, T *warp_tot, T &total)
{
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  T incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_tot[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    T wv = (lane < (int)(blockDim.x >> 5)) ? warp_tot[lane] : T(0);
    T wi = wv;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      T t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    warp_tot[lane] = wi - wv;  // exclusive prefix of warp totals
    if (lane == 31) warp_tot[32] = wi;
  }
  __syncthreads();
  const T out = incl - v + warp_tot[wid];
  total = warp_tot[32];
  __syncthreads();
  return out;
}


struct CellBuildArgs {
  DevParams P;
  const double *x, *y;
  int first, count;
  CellGrid G;
  unsigned *err;
  int storage_order;
  unsigned *rebuild;  // non-null: skip unless set; clear it and record the binned positions
  double *xbin, *ybin;
  PassStats stats;    // non-null niac: zeroed for the rate pass that follows, built or not
  int *step_counter;  // non-null: advanced by one, built or not
  const int *dyn_count;  // non-null: the ids are [first, first + min(count, *dyn_count))
};

inline CellBuildArgs cell_build_args(const DevParams &P, const double *x, const double *y, int first, int count,
                                     const CellGrid &G, unsigned *err, bool storage_order)
{
  CellBuildArgs A;
  A.P = P;
  A.x = x;
  A.y = y;
  A.first = first;
  A.count = count > 0 ? count : 0;
  A.G = G;
  A.err = err;
  A.storage_order = storage_order ? 1 : 0;
  A.rebuild = nullptr;
  A.xbin = P.xbin;
  A.ybin = P.ybin;
  A.stats = PassStats{nullptr, nullptr};
  A.step_counter = nullptr;
  A.dyn_count = nullptr;
  return A;
}

// Grid-wide barrier over co-resident blocks: arrive on bar[0]; the last
// block resets it and bumps the generation bar[1]; the others wait for the
// bump.  The wait gives up after kWaitNs on the global timer (setting
// ERR_TIMEOUT); the result is uniform over the block.
__device__ __forceinline__ bool cell_grid_barrier(unsigned *bar, unsigned *err)
{
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    volatile unsigned *vgen = bar + 1;
    const unsigned gen = *vgen;
    __threadfence();
    if (atomicAdd(&bar[0], 1u) == gridDim.x - 1) {
      atomicExch(&bar[0], 0u);
      __threadfence();
      atomicAdd(&bar[1], 1u);
    } else {
      const unsigned long long t0 = global_ns();
      long long polls = 0;
      while (*vgen == gen) {
        if ((++polls & 255) == 0 && global_ns() - t0 > kWaitNs) {
          atomicOr(err, ERR_TIMEOUT);
          ok = 0;
          break;
        }
      }
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

__device__ __forceinline__ int cell_of_position(const DevParams &P, double px, double py, unsigned *err,
                                                bool storage_order)
{
  const double fx = (px - P.lo_x) * P.inv_cell;
  const double fy = (py - P.lo_y) * P.inv_cell;
  const bool inside = px >= P.lo_x && py >= P.lo_y && px <= P.hi_x && py <= P.hi_y;
  int cx = 0, cy = 0;
  if (inside) {
    cx = min((int)floor(fx), P.ncx - 1);
    cy = min((int)floor(fy), P.ncy - 1);
  } else {
    atomicOr(err, ERR_OUT_OF_DOMAIN);
    if (fx > 0.0) cx = (int)fmin(fx, (double)(P.ncx - 1));
    if (fy > 0.0) cy = (int)fmin(fy, (double)(P.ncy - 1));
  }
  return storage_order ? storage_key(cx, cy, P.ntx, P.tile) : cy * P.ncx + cx;
}

// How a build's phases are spread over the grid: nb() parts, each phase's
// parts done before the next phase starts anywhere.
// One part per block of a co-resident grid, a grid barrier after each phase
// (no block waits after the last).
struct BarrierPhases {
  unsigned *bar, *err;
  __device__ __forceinline__ int nb() const { return gridDim.x; }
  template <typename Part>
  __device__ __forceinline__ bool run(int phase, Part part) const
  {
    part(blockIdx.x);
    return phase == 3 ? true : cell_grid_barrier(bar, err);
  }
};
// Parts drawn by ticket: a block waits for a phase only when every part of
// it has been drawn, that is by blocks that are running already, so the
// grid need not be co-resident and the launch need not be cooperative.
// words: kPhases tickets, then kPhases counts of finished parts, zero between
// launches.
struct TicketPhases {
  static constexpr int kPhases = 5;  // the build's four, and the pass's recording
  unsigned *words, *err;
  __device__ __forceinline__ int nb() const { return gridDim.x; }
  template <typename Part>
  __device__ __forceinline__ bool run(int phase, Part part) const
  {
    __shared__ unsigned s_word;
    for (;;) {
      if (threadIdx.x == 0) s_word = atomicAdd(words + phase, 1u);
      __syncthreads();
      const unsigned k = s_word;
      if (k >= gridDim.x) break;
      part((int)k);
      __syncthreads();
      if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(words + kPhases + phase, 1u);
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      volatile unsigned *finished = words + kPhases + phase;
      unsigned ok = 1u;
      const unsigned long long t0 = global_ns();
      for (long long polls = 0; *finished < gridDim.x; polls++) {
        if ((polls & 255) == 255 && (global_ns() - t0 > kWaitNs || polls > (1LL << 26))) {
          atomicOr(err, ERR_TIMEOUT);
          ok = 0u;
          break;
        }
      }
      __threadfence();
      s_word = ok;
    }
    __syncthreads();
    const bool ok = s_word != 0u;
    __syncthreads();
    return ok;
  }
};

// Phases:
//   1. cell of every slot, histogram; a slot's rank in its cell is the
//      value its atomic add returned
//   2. each part scans its chunk of cells: local prefixes into fill[],
//      the chunk's total into totals[]; count is zeroed as it is read
//   3. every part scans totals[] in shared memory, writes the final
//      start[] of its chunk and scatters its slots to
//      fill[c] + offset(chunk of c) + rank
//   4. each cell's slots sorted ascending (insertion sort, short cells),
//      so the order does not depend on atomic arrival order; a cell with
//      more than kMaxCellOccupancy slots is left unsorted and flags a
//      neighbour overflow.
// The same formulas as the multi-launch build (k_cell_keys and the rest).
// The build's phases for any block size; s_off: shared memory for
// nb() + 1 ints, s_wt: 33 ints.  False when a wait gave up.  Every block of
// the grid must call it.
template <typename Phases>
__device__ __forceinline__ bool cell_build_phases(const CellBuildArgs &A, const Phases &ph, int *s_off, int *s_wt)
{
  const int nb = ph.nb(), t = threadIdx.x, nt = blockDim.x;
  const int stride = nb * nt;
  const int count = A.dyn_count ? min(A.count, *A.dyn_count) : A.count;
  const int ncell = A.G.ncell;
  int *cnt = A.G.count, *start = A.G.start, *fill = A.G.fill, *list = A.G.list;
  int *cell_of = A.G.cell_of, *rank = A.G.rank;
  // a part's cells, a multiple of four so that four cells move as one word
  const int chunk = ((ncell + nb - 1) / nb + 3) & ~3;
  // Loops over slots take kU of a thread's at a time, every load before its
  // first use, and loops over cells four: a large tank's build waits for
  // memory, not for arithmetic.
  constexpr int kU = 4;

  // 1. keys and histogram
  if (!ph.run(0, [&](int b) {
        for (int k0 = b * nt + t; k0 < count; k0 += kU * stride) {
          double px[kU], py[kU];
          int c[kU], r[kU];
#pragma unroll
          for (int u = 0; u < kU; u++) {
            const int k = k0 + u * stride;
            const int s = A.first + (k < count ? k : k0);
            px[u] = A.x[s];
            py[u] = A.y[s];
          }
#pragma unroll
          for (int u = 0; u < kU; u++) {
            if (k0 + u * stride >= count) continue;
            c[u] = cell_of_position(A.P, px[u], py[u], A.err, A.storage_order != 0);
            r[u] = atomicAdd(&cnt[c[u]], 1);
          }
#pragma unroll
          for (int u = 0; u < kU; u++) {
            const int k = k0 + u * stride, s = A.first + k;
            if (k >= count) continue;
            cell_of[s] = c[u];
            rank[s] = r[u];
            if (A.rebuild) {
              A.xbin[s] = px[u];
              A.ybin[s] = py[u];
            }
          }
        }
      }))
    return false;

  // 2. chunk scans.  Each warp takes a contiguous share of the chunk: it adds
  // the share up, and scans it once the shares before it are known, so that a
  // warp has kU words in flight and never waits for another inside its share.
  // 9.7 million cells over 296 parts of 256 threads: 25 us; 137 with the whole
  // block scanning 2,048 cells at a time.
  if (!ph.run(1, [&](int b) {
        const int c0 = min(b * chunk, ncell), c1 = min(c0 + chunk, ncell);
        const int lane = t & 31, wid = t >> 5, nw = nt >> 5;
        const int share = ((chunk + nw - 1) / nw + 3) & ~3;
        const int w0 = min(c0 + wid * share, c1), w1 = min(w0 + share, c1);
        const int whole = w0 + ((w1 - w0) & ~3);  // the words; what is left is the grid's last cells
        int sum = 0;
        for (int c = w0 + 4 * lane; c < whole; c += 128 * 2 * kU) {
          int4 v[2 * kU];
#pragma unroll
          for (int u = 0; u < 2 * kU; u++)
            v[u] = c + 128 * u < whole ? *reinterpret_cast<const int4 *>(cnt + c + 128 * u) : make_int4(0, 0, 0, 0);
#pragma unroll
          for (int u = 0; u < 2 * kU; u++) sum += v[u].x + v[u].y + v[u].z + v[u].w;
        }
        if (whole + lane < w1) sum += cnt[whole + lane];
        sum = __reduce_add_sync(0xffffffffu, sum);
        if (lane == 0) s_wt[wid] = sum;
        __syncthreads();
        int run = 0, total = 0;
        for (int k = 0; k < nw; k++) {
          const int v = s_wt[k];
          if (k < wid) run += v;
          total += v;
        }
        for (int base = w0; base < whole; base += 128 * kU) {
          int4 v[kU];
#pragma unroll
          for (int u = 0; u < kU; u++) {
            const int c = base + 128 * u + 4 * lane;
            v[u] = c < whole ? *reinterpret_cast<const int4 *>(cnt + c) : make_int4(0, 0, 0, 0);
          }
#pragma unroll
          for (int u = 0; u < kU; u++) {
            const int c = base + 128 * u + 4 * lane;
            const int mine = v[u].x + v[u].y + v[u].z + v[u].w;
            int incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const int up = __shfl_up_sync(0xffffffffu, incl, o);
              if (lane >= o) incl += up;
            }
            const int e0 = run + incl - mine, e1 = e0 + v[u].x, e2 = e1 + v[u].y;
            run += __shfl_sync(0xffffffffu, incl, 31);
            if (c < whole) {
              *reinterpret_cast<int4 *>(fill + c) = make_int4(e0, e1, e2, e2 + v[u].z);
              *reinterpret_cast<int4 *>(cnt + c) = make_int4(0, 0, 0, 0);
            }
          }
        }
        if (lane == 0)
          for (int c = whole; c < w1; c++) {
            fill[c] = run;
            run += cnt[c];
            cnt[c] = 0;
          }
        if (t == 0) A.G.totals[b] = total;
      }))
    return false;

  // 3. chunk offsets, final starts, scatter
  if (!ph.run(2, [&](int b) {
        int run = 0;
        for (int base = 0; base < nb; base += nt) {
          const int i = base + t;
          const int v = i < nb ? A.G.totals[i] : 0;
          int total;
          const int ex = block_exclusive_scan<int>(v, s_wt, total);
          if (i < nb) s_off[i] = ex + run;
          run += total;
        }
        if (t == 0) s_off[nb] = run;
        __syncthreads();
        const int c0 = min(b * chunk, ncell), c1 = min(c0 + chunk, ncell), off = s_off[b];
        for (int base = c0 + 4 * t; base < c1; base += kU * 4 * nt) {
          int4 v[kU];
#pragma unroll
          for (int u = 0; u < kU; u++) {
            const int c = base + u * 4 * nt;
            v[u] = *reinterpret_cast<const int4 *>(fill + (c + 4 <= c1 ? c : c0 & ~3));
          }
#pragma unroll
          for (int u = 0; u < kU; u++) {
            const int c = base + u * 4 * nt;
            if (c + 4 <= c1)
              *reinterpret_cast<int4 *>(start + c) = make_int4(v[u].x + off, v[u].y + off, v[u].z + off, v[u].w + off);
            else
              for (int j = c; j < c1; j++) start[j] = fill[j] + off;
          }
        }
        if (b == nb - 1 && t == 0) start[ncell] = s_off[nb];
        if (b == 0 && t == 0 && A.G.st.live) *A.G.st.nlive = 0;
        for (int k0 = b * nt + t; k0 < count; k0 += kU * stride) {
          int c[kU], at[kU];
#pragma unroll
          for (int u = 0; u < kU; u++) {
            const int k = k0 + u * stride, s = A.first + (k < count ? k : k0);
            c[u] = cell_of[s];
            at[u] = rank[s];
          }
#pragma unroll
          for (int u = 0; u < kU; u++) at[u] += fill[c[u]] + s_off[c[u] / chunk];
#pragma unroll
          for (int u = 0; u < kU; u++) {
            const int k = k0 + u * stride;
            if (k < count) list[at[u]] = A.first + k;
          }
        }
      }))
    return false;

  // 4. per-cell sort by slot; the tiles that hold a particle
  return ph.run(3, [&](int b) {
    if (b == 0 && t == 0 && A.G.gen) {  // no tile of the new list is recorded
      *A.G.st.nstream = 0;
      *A.G.st.nhard = 0;
    }
    for (int c = 4 * (b * nt + t); c < ncell; c += 4 * stride) {
      int s[5], e0[4], e1[4];
      const int n = min(4, ncell - c);
      if (n == 4)
        *reinterpret_cast<int4 *>(s) = *reinterpret_cast<const int4 *>(start + c);
      else
        for (int j = 0; j < 4; j++) s[j] = start[min(c + j, ncell)];
      s[4] = start[c + n];
      // the first two entries of all four cells (most cells hold two), then
      // the rest
#pragma unroll
      for (int j = 0; j < 4; j++) {
        e0[j] = e1[j] = 0;
        if (s[j + 1] - s[j] >= 2) {
          e0[j] = list[s[j]];
          e1[j] = list[s[j] + 1];
        }
      }
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int a0 = s[j], a1 = s[j + 1];
        if (a1 - a0 > kMaxCellOccupancy) {
          atomicOr(A.err, ERR_NEIGHBOR_OVERFLOW);
          continue;
        }
        if (e0[j] > e1[j]) {
          list[a0] = e1[j];
          list[a0 + 1] = e0[j];
        }
        for (int i = a0 + 2; i < a1; i++) {
          const int v = list[i];
          int q = i - 1;
          while (q >= a0 && list[q] > v) {
            list[q + 1] = list[q];
            q--;
          }
          list[q + 1] = v;
        }
      }
    }
    if (A.G.st.live && !A.storage_order) {
      const DevParams &P = A.P;
      const int tiles = P.ntx * (P.ncy / P.tile);
      for (int base = b * nt; base < tiles; base += stride) {
        const int tile = base + t;
        bool any = false;
        if (tile < tiles) {
          const int *row = start + (size_t)(tile / P.ntx) * P.tile * P.ncx + (tile % P.ntx) * P.tile;
          for (int r = 0; r < P.tile; r += 4) {
            int lo[4], hi[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
              const int *q = row + (size_t)min(r + u, P.tile - 1) * P.ncx;
              lo[u] = q[0];
              hi[u] = q[P.tile];
            }
#pragma unroll
            for (int u = 0; u < 4; u++) any |= hi[u] > lo[u];
          }
        }
        const unsigned m = __ballot_sync(0xffffffffu, any);
        int at = 0;
        if ((t & 31) == 0 && m) at = atomicAdd(A.G.st.nlive, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (any) A.G.st.live[at + __popc(m & ((1u << (t & 31)) - 1u))] = tile;
      }
    }
  });
}

}  // namespace uph
