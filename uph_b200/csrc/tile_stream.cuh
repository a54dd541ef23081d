// A leapfrog step's rate pass: persistent CTAs that stream tiles whose
// candidate lists are current.
//
// Between two cell-list builds a tile's block holds the same particles in
// the same order.  So the first pass after a build writes down, per tile
// (stream_record), the slots of the block's records and the records of the
// core's particles, and for every fluid particle its candidate list: the
// block's records within the search radius plus the distance two particles
// can close before the next build, in the stencil walk's order, each with
// what the pair's roles are.  The pair loop needs neither the cell list nor
// a listing phase.  Two CTAs per SM walk the recorded tiles in turn with two
// record buffers each (TileStream): while one tile's pairs are summed, the
// next tile's records arrive by cp.async (8-byte copies straight from the
// state arrays into records).  A thread copies whole records, so it may
// convert its own ones after its own copies landed, before it reports them.
//
// Every candidate is put through the exact pair test inside the pair loop;
// one that fails is summed with a zero kernel, so a warp's lanes stay
// together and no listing is needed.  (Where that gives a sum that is not
// finite, the particle's pairs are summed again without the others.)  Partners are visited in the candidate
// list's order, the stencil walk's, so with one lane per particle the sums
// are those of the other passes.
//
// What bounds it (500,000-particle tank, REF FP64): FP64 arithmetic, about
// 105 operations per pair side, 46 M warp instructions or 79 us of the FP64
// pipe, and beside it the pair loop's shared-memory reads (7.7 wavefronts
// per 16-byte read, 72 us of that pipe) at 16 warps per SM, 128 registers a
// thread (k_ref_step, which holds the build, the recording and the hard tiles
// too, spills 268 bytes of stores and 476 of loads, 424 and 592 in the
// brute-force wall modes; k_wcsph_step none).  Measured: the
// streaming step 0.168 ms in the kernel (0.229 for the pass that staged,
// listed and summed one tile per CTA, plus 8 us for the list launch), the
// recording step 0.285; us per step of 100-step calls, before and after:
// REF 5,000 particles 44 and 22, 61,000 56 and 45, 500,000 253 and 190; WCSPH
// FP64 300,000 in violent motion (a rebuild every third step) 198 and 142,
// FP32 pairs 2,000,000 906 and 556.
//
// Lanes per particle (DevParams::lanes): where the tank is so small that
// its tiles do not fill the machine, a particle's candidates are dealt out to
// 2 or 4 lanes (entry e to lane e mod lanes) of smaller tiles, and the lanes'
// sums are added at the end.
//
// What a pass gives the stream (Pass): kStride (bytes of a record, an odd
// multiple of 16, so that 16-byte reads of eight consecutive records hit
// distinct banks), stage(), convert(), begin() and particle().
#pragma once

#include "cell_build.cuh"
#include "leapfrog.cuh"
#include "tile_pass.cuh"

namespace uph {

// ---- one step, one launch -----------------------------------------------------------
// A step is one ordinary launch: where the skin flag asks for it the cell
// list is rebuilt first (phases drawn by ticket) and the pass is a recording
// one over every tile; else the hard tiles are taken one by one and the
// recorded ones streamed.  What the blocks decide by (the skin flag, the
// list's and the record's generation) changes only when the last block
// finishes, which also publishes the pass's statistics and advances the step
// counter.  (A separate, cooperative list launch that only looks at the flag
// and returns took 8 us of every step.)
struct StepArgs {
  PassStats acc;    // the running sums of this launch, zero between launches
  PassStats out;    // the published statistics
  unsigned *done;   // blocks finished, zero between launches
  unsigned *moved;  // what this launch's blocks raise in place of the skin flag, which blocks of
                    // the same launch may still have to read; zero between launches
  unsigned *ticket;  // the stream's next tile, zero between launches
  unsigned *phases;  // the words of TicketPhases, zero between launches
  int relist;        // record the tiles at every launch (no list outlives its step)
  int *counter;     // the step counter (steps finished when the launch starts)
};

enum StepMode { STEP_STREAM, STEP_RECORD, STEP_FAILED };

// What the launch has to do, and for STEP_RECORD the list built.
__device__ __forceinline__ StepMode step_begin(const CellBuildArgs &C, const StepArgs &A, unsigned char *smem)
{
  const unsigned rebuild = *C.rebuild, recorded = *C.G.st.recorded, gen = *C.G.gen;
  if (!rebuild && recorded == gen) return STEP_STREAM;
  if (rebuild) {
    int *s_off = reinterpret_cast<int *>(smem);
    if (!cell_build_phases(C, TicketPhases{A.phases, C.err}, s_off, s_off + kCellBuildMaxBlocks + 1)) return STEP_FAILED;
  }
  return STEP_RECORD;
}

// The walls' motion into F.D (the counter is one behind: this step has not
// been counted yet).
__device__ __forceinline__ void step_walls(const DevParams &P, const StepOut &F)
{
  if (!F.enabled || !F.walls) return;
  const double t = (*F.d_itime + (F.walls == 2 ? 2 : 1)) * P.dt;
  for (int w = P.nf + blockIdx.x * kTileThreads + threadIdx.x; w < P.n; w += gridDim.x * kTileThreads)
    wall_move_one(P, F.D, F.W, w, t, F.err);
}

__device__ __forceinline__ void step_end(const CellBuildArgs &C, const StepArgs &A, StepMode mode)
{
  const CellGrid &G = C.G;
  __syncthreads();
  if (threadIdx.x != 0) return;
  __threadfence();
  if (atomicAdd(A.done, 1u) != gridDim.x - 1) return;
  __threadfence();
  // every load first: one round of latency
  const unsigned long long niac = *(volatile unsigned long long *)A.acc.niac;
  const int max_nb = *(volatile int *)A.acc.max_nb;
  const unsigned moved = *(volatile unsigned *)A.moved;
  const unsigned rebuild = *(volatile unsigned *)C.rebuild;
  unsigned gen = *(volatile unsigned *)G.gen;
  const int counter = *A.counter;
  *A.done = 0u;
  *A.ticket = 0u;
  *A.acc.niac = 0ull;
  *A.acc.max_nb = 0;
  *A.out.niac = niac;
  *A.out.max_nb = max_nb;
  *A.counter = counter + 1;
  if (mode == STEP_RECORD) {
    for (int k = 0; k < 2 * TicketPhases::kPhases; k++) A.phases[k] = 0u;
    if (rebuild) *G.gen = ++gen;
    *C.rebuild = moved ? 1u : 0u;
    *G.st.recorded = A.relist ? gen - 1u : gen;
    if (A.relist) {
      *G.st.nstream = 0;
      *G.st.nhard = 0;
    }
  } else if (moved) {
    *C.rebuild = 1u;
  }
  *A.moved = 0u;
}

__device__ __forceinline__ uint32_t stream_smem(const void *p)
{
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void *src)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void *src)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void stream_arrive(uint32_t bar)
{
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// true once the barrier's phase `parity` completed; false after kWaitNs on
// the global timer or the poll cap, whichever comes first
__device__ __forceinline__ bool stream_wait(uint32_t bar, uint32_t parity)
{
  unsigned long long t0 = 0;
  for (long long i = 0; i < (1LL << 26); i++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if ((i & 63) == 63) {
      const unsigned long long t = global_ns();
      if (t0 == 0) t0 = t;
      if (t - t0 > kWaitNs) return false;
    }
  }
  return false;
}

// dynamic shared memory: two record buffers, then the four barriers and the
// two next tiles
template <int kStride>
constexpr size_t stream_smem_bytes() { return 2 * (size_t)kStreamCap * kStride + 48; }

// All threads of a 256-thread CTA; smem: stream_smem_bytes<kStride>().
//
// No CTA-wide barrier: a warp that is done with a tile goes on to the next
// one.  Buffer b's two mbarriers are full[b] (every thread's copies of the
// tile have landed and are converted) and empty[b] (every warp has summed
// the tile's pairs).  While a warp sums its it-th tile it refills the other
// buffer: at candidate kIssueAt it waits until tile it - 1 has left that
// buffer and starts its copies of tile it + 1; at candidate kReadyAt, about
// 4 us later on the 500,000-particle tank, it waits for those copies and
// reports them.  (One barrier per tile instead cost the skew between warps,
// 12 of 200 us.)
//
// A CTA's first two tiles are its own, the others are drawn by ticket: the
// first thread draws tile it + 2 while it sums tile it and leaves it in
// shared memory before it reports tile it + 1, where the others find it.
template <typename Pass, int kLanes>
struct TileStream {
  static constexpr int kIssueAt = kLanes == 1 ? 3 : 1, kReadyAt = kLanes == 1 ? 12 : 4;
  static_assert(kStreamCap <= 2 * kTileThreads, "a thread stages at most two records");
  Pass &ps;
  const CellGrid &G;
  unsigned char *smem;
  unsigned *err;
  uint32_t bars;  // full[0], full[1], empty[0], empty[1]
  unsigned *ticket;
  int ntile, cid, nxt, it;  // this CTA's it-th tile, and the one after it
  int drawn;                // thread 0: the tile after that
  int s0, s1;  // the slots this thread copies next, -1 past the block's end
  bool ok;

  __device__ __forceinline__ unsigned char *buffer(int b) const { return smem + (size_t)b * kStreamCap * Pass::kStride; }
  __device__ __forceinline__ uint32_t full(int b) const { return bars + 8 * b; }
  __device__ __forceinline__ uint32_t empty(int b) const { return bars + 16 + 8 * b; }
  __device__ __forceinline__ volatile int &after(int k) const
  {
    return reinterpret_cast<volatile int *>(smem + 2 * (size_t)kStreamCap * Pass::kStride + 32)[k & 1];
  }
  // this thread's slots of tile c
  __device__ __forceinline__ void slots(int c)
  {
    s0 = s1 = -1;
    if (c < ntile) {
      s0 = G.st.slot[(size_t)c * kStreamCap + threadIdx.x];
      if (threadIdx.x + kTileThreads < kStreamCap) s1 = G.st.slot[(size_t)c * kStreamCap + threadIdx.x + kTileThreads];
    }
  }
  __device__ __forceinline__ void issue(int b) const
  {
    unsigned char *p = buffer(b) + (size_t)threadIdx.x * Pass::kStride;
    if (s0 >= 0) ps.stage(s0, stream_smem(p));
    if (s1 >= 0) ps.stage(s1, stream_smem(p + (size_t)kTileThreads * Pass::kStride));
  }
  __device__ __forceinline__ void ready(int c, int b) const
  {
    unsigned char *p = buffer(b) + (size_t)threadIdx.x * Pass::kStride;
    cp_async_wait_all();
    ps.convert(G.st.tile[c], s0 >= 0 ? p : nullptr, s1 >= 0 ? p + (size_t)kTileThreads * Pass::kStride : nullptr);
    stream_arrive(full(b));
  }
  // the refill of the other buffer, called before candidate e of every warp
  // (all lanes), e = 0, 1, ... at least up to kReadyAt
  __device__ __forceinline__ void refill(int e)
  {
    if (e != kIssueAt && e != kReadyAt) return;
    if (nxt >= ntile || !ok) return;
    const int b = (it + 1) & 1;
    if (e == kIssueAt) {
      // tile it - 1 was the ((it - 1) / 2 + 1)-th to leave that buffer
      if (it > 0) ok = __all_sync(0xffffffffu, stream_wait(empty(b), ((it - 1) >> 1) & 1));
      if (threadIdx.x == 0) drawn = 2 * gridDim.x + atomicAdd(ticket, 1u);
      if (ok) issue(b);
    } else {
      if (threadIdx.x == 0) after(it) = drawn;
      ready(nxt, b);
    }
  }

  __device__ __forceinline__ void run(const DevParams &P, int nstream)
  {
    ntile = nstream;
    cid = blockIdx.x;
    nxt = blockIdx.x + gridDim.x;
    it = 0;
    drawn = 0;
    ok = true;
    bars = stream_smem(smem + 2 * (size_t)kStreamCap * Pass::kStride);
    if (cid >= ntile) return;
    if (threadIdx.x == 0) {
      for (int b = 0; b < 2; b++) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(full(b)), "r"(kTileThreads));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(empty(b)), "r"(kTileThreads / 32));
      }
    }
    slots(cid);
    issue(0);
    int2 core = G.st.core[(size_t)cid * kTileThreads + threadIdx.x];
    __syncthreads();
    ready(cid, 0);
    while (cid < ntile) {
      const int b = it & 1;
      const int a = core.x, rec = core.y;
      CandReader<kLanes> rd;
      const int n = rd.init(G, P.nf, a);
      ps.begin(a);
      ok = __all_sync(0xffffffffu, ok && stream_wait(full(b), (it >> 1) & 1));
      if (!ok) break;
      if (it > 0) nxt = after(it - 1);
      slots(nxt);
      core = make_int2(-1, 0);
      if (nxt < ntile) core = G.st.core[(size_t)nxt * kTileThreads + threadIdx.x];
      ps.particle(buffer(b), rec, a, n, rd, *this);
      cid = nxt;
      it++;
    }
    if (!ok) {
      // a wait gave up: let this thread's copies land and stop
      cp_async_wait_all();
      atomicOr(err, ERR_TIMEOUT);
    }
  }
  // the warp has read the last record of its tile
  __device__ __forceinline__ void done_reading() const
  {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) stream_arrive(empty(it & 1));
  }
};

// Shared memory of stream_record, one per group.
struct RecordSmem {
  int gs[kTileRowsMax], roff[kTileRowsMax + 1];  // as TileBlock's
  int tab[kTileTabMax];
  float2 posf[kStreamCap];  // relative to the block's origin
  unsigned who[kStreamCap];  // reference index; kWhoWall (itype >= 2), kWhoBoundary
  int slot[kStreamCap];
  int cid;
};
constexpr unsigned kWhoWall = 0x80000000u, kWhoBoundary = 0x40000000u, kWhoIndex = 0x3fffffffu;
// Entries a lane has not written out yet: a ring of 16 (a 40-byte stride
// spreads the lanes over the banks), each full eight leaving as one word.
struct RecordRing {
  unsigned short e[kTileThreads][20];
};
constexpr size_t kRecordSmemBytes = sizeof(RecordRing) + sizeof(RecordSmem) * (kTileThreads / 32);

// A group of kGroup threads (a warp, or the CTA) writes the candidate lists
// and the record of tile `tile`; a tile that does not fit the stream (more
// records than a buffer, more core particles than lanes for them, a list that
// overflowed, no room in the stream's arrays) goes onto the list of hard
// tiles.  Only FP32 distances are computed: a candidate within the list
// radius (F32Test::vl, rounding included) is listed, and the pair loop
// decides.  The distances are those of the positions the list binned
// (DevParams::xbin), which the skin bounds the motion from: a pass that
// records later than it was built (walls may have moved meanwhile) writes the
// same lists, as does one that records at every launch, so which lanes and
// which tiles a pair falls to, and with them every rounding, do not depend on
// when lists are written.
template <bool kBrute, int kGroup>
__device__ __forceinline__ void stream_record(const DevParams &P, const SlotArrays &S, const CellGrid &G, int tile,
                                              RecordSmem &R, RecordRing &ring)
{
  auto sync = [] {
    if constexpr (kGroup == 32)
      __syncwarp();
    else
      __syncthreads();
  };
  auto any_of = [](bool v) {
    if constexpr (kGroup == 32)
      return __any_sync(0xffffffffu, v) != 0;
    else
      return __syncthreads_or(v) != 0;
  };
  const int lane = threadIdx.x & 31, tid = threadIdx.x & (kGroup - 1);
  const int T = P.tile, reach = P.reach;
  const int cx0 = (tile % P.ntx) * T, cy0 = (tile / P.ntx) * T;
  const int bx0 = max(cx0 - reach, 0), by0 = max(cy0 - reach, 0);
  const int W = min(cx0 + T - 1 + reach, P.ncx - 1) - bx0 + 1, H = min(cy0 + T - 1 + reach, P.ncy - 1) - by0 + 1;
  const int stride = W + 1, lc0 = cx0 - bx0;
  sync();
  for (int e = tid; e < stride * H; e += kGroup) {
    const int r = e / stride, c = e - r * stride;
    R.tab[e] = G.start[(size_t)(by0 + r) * P.ncx + bx0 + c];
  }
  sync();
  // row lengths of the block and of the core, and their prefixes (every
  // warp of the group for itself)
  int len = 0, clen = 0, gs = 0;
  if (lane < H) {
    const int *row = R.tab + lane * stride;
    gs = row[0];
    len = row[W] - gs;
    const int cr = by0 + lane - cy0;
    if (cr >= 0 && cr < T) clen = row[lc0 + T] - row[lc0];
  }
  int il = len, ic = clen;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, il, o), c = __shfl_up_sync(0xffffffffu, ic, o);
    if (lane >= o) {
      il += a;
      ic += c;
    }
  }
  const int nrec = __shfl_sync(0xffffffffu, il, 31), ncore = __shfl_sync(0xffffffffu, ic, 31);
  const int coff = ic - clen;  // core particles before this row
  if (tid < 32) {
    R.gs[lane] = gs;
    R.roff[lane] = il - len;
    if (lane == 31) R.roff[32] = il;
  }
  const bool fits = nrec <= kStreamCap && ncore * P.lanes <= kTileThreads;
  bool overflow = false, fluid = !fits;
  int c = -1;
  sync();
  if (fits) {
    // list positions -> record indices of the block
    for (int e = tid; e < stride * H; e += kGroup) {
      const int r = e / stride;
      R.tab[e] = R.roff[r] + (R.tab[e] - R.gs[r]);
    }
    sync();
    const double ox = fma((double)bx0, P.cell, P.lo_x), oy = fma((double)by0, P.cell, P.lo_y);
    constexpr int kU = kGroup == 32 ? 4 : 2;  // records of a thread in flight
    for (int k0 = tid; k0 < nrec; k0 += kU * kGroup) {
      int s[kU], r[kU];
      double x[kU], y[kU];
      unsigned who[kU];
#pragma unroll
      for (int u = 0; u < kU; u++) {
        const int k = min(k0 + kGroup * u, nrec - 1);
        r[u] = tile_row_of(R.roff, k);
        s[u] = G.list[R.gs[r[u]] + k - R.roff[r[u]]];
      }
#pragma unroll
      for (int u = 0; u < kU; u++) {
        x[u] = P.xbin[s[u]];
        y[u] = P.ybin[s[u]];
        const int o = S.orig[s[u]];
        who[u] = (unsigned)o | (S.itype[s[u]] >= 2 ? kWhoWall : 0u) | (o >= P.b0 && o < P.b1 ? kWhoBoundary : 0u);
      }
#pragma unroll
      for (int u = 0; u < kU; u++) {
        const int k = k0 + kGroup * u;
        if (k >= nrec) continue;
        const int *rt = R.tab + r[u] * stride + lc0;
        const int cr = by0 + r[u] - cy0;
        fluid |= s[u] < P.nf && cr >= 0 && cr < T && k >= rt[0] && k < rt[T];
        R.posf[k] = make_float2((float)(x[u] - ox), (float)(y[u] - oy));
        R.who[k] = who[u];
        R.slot[k] = s[u];
      }
    }
    fluid = any_of(fluid);
    if (fluid) {
      if (tid == 0) R.cid = atomicAdd(G.st.nstream, 1);
      sync();
      c = R.cid;
      if (c >= G.st.cap) c = -1;
    }
  }
  if (c >= 0) {
    int *slot = G.st.slot + (size_t)c * kStreamCap;
    for (int k = tid; k < kStreamCap; k += kGroup) slot[k] = k < nrec ? R.slot[k] : -1;
    const float vl = make_f32_test(P, max(W, H), 0.f, 0.f).vl;
    unsigned short *mine = ring.e[threadIdx.x];
    for (int k0 = 0; k0 < kTileThreads / P.lanes; k0 += kGroup) {
      const int k = k0 + tid;
      // the k-th core particle: the row with coff <= k, its record there
      int row = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1)
        if (__shfl_sync(0xffffffffu, coff, row + step) <= k) row += step;
      const int first = __shfl_sync(0xffffffffu, coff, row);
      int kr = 0, a = -1;
      if (k < ncore) {
        kr = R.tab[row * stride + lc0] + k - first;
        a = R.slot[kr];
        if (a >= P.nf) a = -1;
      }
      if (a >= 0) {
        const float2 of = R.posf[kr];
        const int oa = (int)(R.who[kr] & kWhoIndex);
        const unsigned role_i = kCandI | (S.itype[a] == 1 ? kCandWall : 0u), base = oa >= P.pb ? kCandNoPair : 0u;
        // the column of the particle's cell: the largest whose first record
        // is not past it
        const int *rt = R.tab + row * stride;
        int col = 0;
#pragma unroll
        for (int step = 16; step > 0; step >>= 1)
          if (col + step < W && rt[col + step] <= kr) col += step;
        const int c0 = max(col - reach, 0), c1 = min(col + reach, W - 1);
        uint4 *out = reinterpret_cast<uint4 *>(G.vl) + a;
        int cnt = 0, gone = 0;
        auto flush = [&] {
          const uint2 *h = reinterpret_cast<const uint2 *>(mine + (gone & 8));
          const uint2 w0 = h[0], w1 = h[1];
          if (gone < G.vl_cap) *out = make_uint4(w0.x, w0.y, w1.x, w1.y);
          out += P.nf;
          gone += 8;
        };
        for (int r = max(row - reach, 0); r <= min(row + reach, H - 1); r++) {
          const int kend = R.tab[r * stride + c1 + 1];
          for (int q = R.tab[r * stride + c0]; q < kend; q += 4) {
#pragma unroll
            for (int u = 0; u < 4; u++) {
              const int kk = min(q + u, kend - 1);
              const float2 f = R.posf[kk];
              const unsigned who = R.who[kk];
              const float dx = of.x - f.x, dy = of.y - f.y;
              const bool in = q + u < kend && kk != kr && fmaf(dx, dx, dy * dy) < vl;
              const int ob = (int)(who & kWhoIndex);
              unsigned e = (unsigned)kk | base;
              if (ob > oa) e |= role_i & ((who & kWhoWall) ? (kCandI | kCandWall) : kCandI);
              if (ob >= P.pb) e |= kCandNoPair;
              if (kBrute && (who & kWhoBoundary)) e |= kCandBoundary;
              if (in) mine[cnt & 15] = (unsigned short)e;
              cnt += in;
            }
            if (cnt - gone >= 8) flush();
          }
        }
        if (cnt > gone) flush();
        const bool over = cnt > G.vl_cap;
        overflow |= over;
        G.vl_n[a] = over ? kVlOverflow : (unsigned char)cnt;
      }
      if (k * P.lanes < kTileThreads)
        for (int l = 0; l < P.lanes; l++)
          G.st.core[(size_t)c * kTileThreads + k * P.lanes + l] = make_int2(a, kr);
    }
    overflow = any_of(overflow);
    // a tile whose lists do not fit is hard: its place in the stream is left
    // empty
    if (overflow) {
      for (int k = tid; k < kTileThreads; k += kGroup) G.st.core[(size_t)c * kTileThreads + k] = make_int2(-1, 0);
      for (int k = tid; k < kStreamCap; k += kGroup) slot[k] = -1;
    }
  }
  if (tid == 0) {
    if (c >= 0) G.st.tile[c] = tile;
    if (fluid && (c < 0 || overflow)) G.st.hard[atomicAdd(G.st.nhard, 1)] = tile;
  }
}

// The recording of every tile that holds a particle: a warp per tile, for the
// more tiles in flight, in whole rounds of the grid's warps, and a CTA per
// tile, for the shorter chain, where what is left is few rounds of the grid.
// us on a stirred dam break: 61,000 particles (390 tiles, 296 CTAs) 25 by
// CTAs, 84 by warps; 300,000 (1,600 tiles) 100 against 72; 2,000,000 (9,600
// tiles, four rounds of warps and 130 tiles) 285 with the last ones by CTAs,
// 327 without.
template <bool kBrute>
__device__ __forceinline__ bool step_record(const CellBuildArgs &C, const SlotArrays &S, const StepArgs &A,
                                            unsigned char *smem)
{
  const CellGrid &G = C.G;
  RecordRing &ring = *reinterpret_cast<RecordRing *>(smem);
  RecordSmem *R = reinterpret_cast<RecordSmem *>(smem + sizeof(RecordRing));
  const int nlive = *(volatile int *)G.st.nlive;
  const volatile int *live = G.st.live;
  const TicketPhases ph{A.phases, C.err};
  constexpr int kWarps = kTileThreads / 32;
  const int round = (int)gridDim.x * kWarps, rest = nlive % round;
  const int by_warps = rest <= 4 * (int)gridDim.x ? nlive - rest : nlive;
  return ph.run(4, [&](int b) {
    const int w = threadIdx.x >> 5;
    for (int t = b * kWarps + w; t < by_warps; t += round)
      stream_record<kBrute, 32>(C.P, S, G, live[t], R[w], ring);
    if (by_warps < nlive) __syncthreads();
    for (int t = by_warps + b; t < nlive; t += gridDim.x)
      stream_record<kBrute, kTileThreads>(C.P, S, G, live[t], R[0], ring);
  });
}

// The whole step of a pass (launch_step).  hard_tile(t) takes one hard tile,
// ps streams the others.
template <bool kBrute, int kLanes, typename Pass, typename HardTile>
__device__ __forceinline__ void step_run(const CellBuildArgs &C, const SlotArrays &S, const StepOut &F,
                                         const StepArgs &A, Pass &ps, unsigned char *smem, HardTile hard_tile)
{
  const DevParams &P = C.P;
  const CellGrid &G = C.G;
  // nothing of the launch before is read or overwritten above this line; the
  // next launch's blocks may take the places that this one's blocks leave
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  StepMode mode = step_begin(C, A, smem);
  step_walls(P, F);
  if (mode == STEP_RECORD && !step_record<kBrute>(C, S, A, smem)) mode = STEP_FAILED;
  if (mode != STEP_FAILED) {
    const int nhard = *(volatile int *)G.st.nhard;
    const int nstream = min(*(volatile int *)G.st.nstream, G.st.cap);
    for (int k = blockIdx.x; k < nhard; k += gridDim.x) {
      hard_tile(*(volatile int *)&G.st.hard[k]);
      __syncthreads();
    }
    TileStream<Pass, kLanes> t{ps, G, smem, C.err};
    t.ticket = A.ticket;
    t.run(P, nstream);
  }
  pass_stats(A.acc, ps.my_pairs, ps.my_nb);
  step_end(C, A, mode);
}

// The launch of a step.  kStep: the pass's kernel, with `smem` bytes of
// dynamic shared memory.
template <auto kStep>
uph_status launch_step(size_t smem, const DevParams &P, const SlotArrays &S, const CellGrid &G, const StepOut &F,
                       const StepArgs &A, unsigned *err, cudaStream_t s)
{
  static int resident[64] = {};  // blocks that fit the device at once
  int dev = 0;
  UPH_CUDA(cudaGetDevice(&dev));
  int most = dev >= 0 && dev < 64 ? resident[dev] : 0;
  if (most == 0) {
    int sms = 0, per_sm = 0;
    UPH_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    UPH_CUDA(cudaFuncSetAttribute(kStep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    UPH_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kStep, kTileThreads, smem));
    most = std::min(per_sm * sms, kCellBuildMaxBlocks);
    if (most < 1) return fail(UPH_CUDA_ERROR, "the rate pass's kernel cannot be resident");
    if (dev >= 0 && dev < 64) resident[dev] = most;
  }
  CellBuildArgs C = cell_build_args(P, S.x, S.y, 0, P.n, G, err, false);
  C.rebuild = P.rebuild;
  C.P.rebuild = A.moved;
  // The next step's blocks are set up while this one's last blocks run
  // (step_run waits for the launch before it): 22.3 against 23.1 us a
  // step of 5,000 particles, 45 against 47 of 61,000.  In a captured graph,
  // whose nodes follow each other faster, plain edges are the better ones:
  // 18.3 against 18.8 us a step of 5,000.
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  UPH_CUDA(cudaStreamIsCapturing(s, &capturing));
  cudaLaunchAttribute early{};
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(std::max(1, std::min(most, P.ntx * (P.ncy / P.tile))));
  cfg.blockDim = dim3(kTileThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &early;
  cfg.numAttrs = capturing == cudaStreamCaptureStatusNone ? 1 : 0;
  UPH_CUDA(cudaLaunchKernelEx(&cfg, kStep, C, S, F, A));
  return UPH_OK;
}

}  // namespace uph
