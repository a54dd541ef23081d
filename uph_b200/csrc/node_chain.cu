// Fused node-side layers of the surrogate network on the tcgen05 tensor cores.
//
// Between two edge layers every layer of the network is node-local, so a
// 128-row tile of nodes can run through all of them without leaving the SM:
//   encoder: F -> relu(E1 F + b) -> h0 = E2 (.) + b -> [P | Q] = W_pq h0 + b
//   round:   S, h -> m = W2 S -> u = relu(N1 [h ; m] + b) -> h' = h + N2 u + b
//            -> [P | Q]' = W_pq' h' + b        (or, in the last round,
//            -> relu(Dec1 h' + b) -> out = Dec2 (.) + b)
// Every weight is cut into 128 x 128 pieces (N1 into its two K halves, which
// accumulate into one TMEM tile; W_pq into its P and Q rows, which fill
// TMEM columns 0..127 and 128..255), each a K = 128, N = 128 UMMA.
//
// Two persistent CTAs per SM, 96 KiB of shared memory each:
//   X  2 atoms   the tile's first operand (F or S), then m, u, ... and P
//   H  2 atoms   h, updated in place by the residual layer, at last Q
//   W  2 atoms   one weight piece
// (an atom = 128 rows x 64 BF16 columns in the 128-byte-swizzled K-major
// layout of the UMMA descriptors).  Inputs arrive by TMA (2-D tensor maps
// with 128-byte swizzle, no multicast), weight pieces as pre-swizzled images
// by bulk copies, all completing on mbarriers; h and [P | Q] leave the SM as
// TMA tensor stores of swizzled atoms.
//
// One thread of a ninth warp produces: it fetches, issues every piece's MMAs,
// refills the weight slot as soon as a piece is done, and stores.  Eight warps
// run the epilogues (TMEM lane = row, a warp takes 64 of a layer's 128 columns):
// bias, residual, ReLU, BF16 into shared memory.  Layers alternate between the
// two 128-column halves of the CTA's TMEM, so a piece that needs nothing of
// the running epilogue (N1's h half, W_Q, the next tile's first) is multiplied
// beside it.
//
// Bound by the chain of a tile (a layer's MMA some 1,200 cycles, its epilogue
// 3,000, then [P | Q] out and the next operand in, 4,000), which the SM's two
// CTAs overlap; the tensor pipe is busy for some 20 us of a round at 207,000
// nodes.  A round there: 88 us (encoder 69, last round 76), against 114 (90,
// 91) with four warps that waited for every load, MMA and store in turn, and
// 89 (66, 86) with one CTA per SM whose two tiles share a ring of three weight
// pieces: both tiles then end together.
//
// The arithmetic is that of the unfused path (tc_gemm.cu) step for step --
// the same K order of MMAs, FP32 bias then residual, the same BF16 rounding
// points -- so both give the same network.
//
// Every mbarrier wait is bounded; a wait that gives up sets ERR_TIMEOUT, the
// CTA stops, waits (bounded) for its copies, stores and MMAs in flight, frees
// its TMEM and returns.
#include <cudaTypedefs.h>

#include <cute/arch/mma_sm100_desc.hpp>
#include <cute/numeric/numeric_types.hpp>

#include "node_chain.cuh"

namespace uph {
namespace {

constexpr int kAtom = 16384;           // 128 rows x 128 bytes
constexpr int kOffX = 0;               // 2 atoms: the tile's working activations
constexpr int kOffH = 2 * kAtom;       // 2 atoms: h
constexpr int kOffW = 4 * kAtom;       // 2 atoms: one weight piece (128 x 128)
constexpr int kSmemUsed = 6 * kAtom;   // 96 KiB: two CTAs per SM
constexpr int kSmemBytes = kSmemUsed + 1024;
constexpr int kEpiWarps = 8;
constexpr int kThreads = 32 * (kEpiWarps + 1);
constexpr int kMaxLayers = 5;
constexpr int kPieceBytes = 2 * kAtom;
constexpr long long kWaitLimit = 1LL << 26;

enum Buf : int { BUF_X = 0, BUF_H = 1 };

// what a layer's epilogue does with its accumulator
enum Epi : int {
  EPI_X = 0,         // (+ bias) (ReLU) -> BF16 into X
  EPI_H = 1,         // + bias -> BF16 into H (the encoder's h0; Q)
  EPI_RESIDUAL = 2,  // + bias + h -> BF16 into H
  EPI_OUT = 3,       // columns 0..15 + bias -> FP32 to out
};

struct LayerSpec {
  int epi;
  int relu;
};

struct PieceSpec {
  int a;      // A operand buffer
  int first;  // starts its layer's accumulator
  int last;   // completes it
  int after;  // reads what the layer before left in shared memory
};

__host__ __device__ inline int piece_count(int mode) { return mode == CHAIN_ENCODER ? 4 : 6; }
__host__ __device__ inline int layer_count(int mode) { return mode == CHAIN_ENCODER ? 4 : 5; }

// encoder: E1 | E2 | W_P | W_Q;  round: W2 | N1a N1b | N2 | W_P | W_Q;
// last round: W2 | N1a N1b | N2 | Dec1 | Dec2
__device__ __forceinline__ PieceSpec piece_of(int mode, int p)
{
  if (mode == CHAIN_ENCODER) {
    if (p == 0) return PieceSpec{BUF_X, 1, 1, 0};
    if (p == 1) return PieceSpec{BUF_X, 1, 1, 1};
    if (p == 2) return PieceSpec{BUF_H, 1, 1, 1};
    return PieceSpec{BUF_H, 1, 1, 0};
  }
  if (p == 0) return PieceSpec{BUF_X, 1, 1, 0};
  if (p == 1) return PieceSpec{BUF_H, 1, 0, 0};
  if (p == 2) return PieceSpec{BUF_X, 0, 1, 1};
  if (p == 3) return PieceSpec{BUF_X, 1, 1, 1};
  if (p == 4) return PieceSpec{BUF_H, 1, 1, 1};
  return mode == CHAIN_ROUND ? PieceSpec{BUF_H, 1, 1, 0} : PieceSpec{BUF_X, 1, 1, 1};
}

__device__ __forceinline__ LayerSpec layer_of(int mode, int l)
{
  if (mode == CHAIN_ENCODER) {
    if (l == 0) return LayerSpec{EPI_X, 1};
    return l == 2 ? LayerSpec{EPI_X, 0} : LayerSpec{EPI_H, 0};
  }
  if (l == 0) return LayerSpec{EPI_X, 0};
  if (l == 1) return LayerSpec{EPI_X, 1};
  if (l == 2) return LayerSpec{EPI_RESIDUAL, 0};
  if (mode == CHAIN_ROUND) return l == 3 ? LayerSpec{EPI_X, 0} : LayerSpec{EPI_H, 0};
  return l == 3 ? LayerSpec{EPI_X, 1} : LayerSpec{EPI_OUT, 0};
}

// a layer's bias: that of its last piece, W_P and W_Q sharing W_Q's 256 values
__device__ __forceinline__ const float *bias_of(const ChainArgs &a, int l)
{
  const int np = piece_count(a.mode);
  if (a.mode != CHAIN_LAST && l == layer_count(a.mode) - 2) return a.piece[np - 1].bias;
  if (a.mode != CHAIN_LAST && l == layer_count(a.mode) - 1) return a.piece[np - 1].bias + 128;
  return a.piece[a.mode == CHAIN_ENCODER || l == 0 ? l : l + 1].bias;
}

__device__ __forceinline__ uint32_t su32(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr)
{
  cute::UMMA::SmemDescriptor d;
  d.desc_ = 0;
  d.start_address_ = static_cast<uint16_t>(addr >> 4);
  d.leading_byte_offset_ = 1;
  d.stride_byte_offset_ = 1024 >> 4;
  d.version_ = 1;
  d.base_offset_ = 0;
  d.lbo_mode_ = 0;
  d.layout_type_ = static_cast<uint8_t>(cute::UMMA::LayoutType::SWIZZLE_128B);
  return d.desc_;
}

// true once the barrier's phase `parity` completed; false after kWaitNs on
// the global timer or kWaitLimit polls, whichever comes first
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity)
{
  const unsigned long long t0 = global_ns();
  for (long long i = 0; i < kWaitLimit; i++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if ((i & 63) == 63 && global_ns() - t0 > kWaitNs) return false;
  }
  return false;
}

__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// one 128-row x 64-column box of a 2-D tensor map (x = column, y = row)
__device__ __forceinline__ void tma_load_box(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar)
{
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// one 128-row x 64-column box from shared memory to a 2-D tensor map (x, y
// are non-negative and x * 2 bytes is a multiple of 16)
__device__ __forceinline__ void tma_store_box(const CUtensorMap *map, uint32_t src, int x, int y)
{
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(src), "r"(x), "r"(y)
               : "memory");
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t addr, float v[16])
{
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 16; j++) v[j] = __uint_as_float(r[j]);
}

// 64 consecutive TMEM columns of this warp's 32 lanes, waited for inside the
// same asm statement so no use of the registers can be scheduled before
// the load completes
__device__ __forceinline__ void tmem_ld64(uint32_t addr, float v[64])
{
  uint32_t r[64];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x64.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, %48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%64];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]), "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]), "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]), "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]), "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
      : "r"(addr)
      : "memory");
#pragma unroll
  for (int j = 0; j < 64; j++) v[j] = __uint_as_float(r[j]);
}

// row r, columns [c0, c0 + 16) of a swizzled K-major buffer of 128-row atoms
__device__ __forceinline__ void smem_put16(uint8_t *buf, int r, int c0, const float v[16])
{
  __align__(16) __nv_bfloat162 h[8];
#pragma unroll
  for (int j = 0; j < 8; j++) h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
  uint8_t *row = buf + (c0 >> 6) * kAtom + r * 128;
  const int q = (c0 & 63) >> 3;
  *reinterpret_cast<uint4 *>(row + ((q ^ (r & 7)) << 4)) = *reinterpret_cast<uint4 *>(&h[0]);
  *reinterpret_cast<uint4 *>(row + (((q + 1) ^ (r & 7)) << 4)) = *reinterpret_cast<uint4 *>(&h[4]);
}

__device__ __forceinline__ void smem_get16(const uint8_t *buf, int r, int c0, float v[16])
{
  const uint8_t *row = buf + (c0 >> 6) * kAtom + r * 128;
  const int q = (c0 & 63) >> 3;
  __align__(16) __nv_bfloat162 h[8];
  *reinterpret_cast<uint4 *>(&h[0]) = *reinterpret_cast<const uint4 *>(row + ((q ^ (r & 7)) << 4));
  *reinterpret_cast<uint4 *>(&h[4]) = *reinterpret_cast<const uint4 *>(row + (((q + 1) ^ (r & 7)) << 4));
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const float2 f = __bfloat1622float2(h[j]);
    v[2 * j] = f.x;
    v[2 * j + 1] = f.y;
  }
}

// issue the K = 128 MMA of one 128 x 128 weight piece
__device__ __forceinline__ void issue_piece(uint32_t tmem, uint32_t a, uint32_t w, uint32_t idesc, int accumulate,
                                            uint32_t bar)
{
#pragma unroll
  for (int ka = 0; ka < 2; ka++)
#pragma unroll
    for (int kk = 0; kk < 4; kk++) {
      const uint64_t da = desc_sw128(a + ka * kAtom + kk * 32);
      const uint64_t db = desc_sw128(w + ka * kAtom + kk * 32);
      const uint32_t acc = (accumulate || ka || kk) ? 1u : 0u;
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "setp.ne.b32 p, %4, 0;\n\t"
          "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
          "l"(da), "l"(db), "r"(idesc), "r"(acc));
    }
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

struct ChainBars {
  uint64_t x, h, w;    // the tile's first operand, h and the weight piece have arrived
  uint64_t part;       // an MMA that does not complete its layer is done
  uint64_t layer[2];   // the MMAs of layer number g (counted over the tiles) are done: [g % 2]
  uint64_t epi[2];     // its epilogue is done: [g % 2], one arrival per warp
};

__global__ void __launch_bounds__(kThreads, 2) k_node_chain(const __grid_constant__ ChainArgs a)
{
  extern __shared__ uint8_t smem_raw[];
  __shared__ ChainBars bars;
  __shared__ uint32_t tmem_slot;
  __shared__ int s_mma_pending;  // set by the final drain: an MMA never completed
  __shared__ float s_bias[kMaxLayers][128];
  uint8_t *sm = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sb = su32(sm);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int NP = piece_count(a.mode), NL = layer_count(a.mode);
  const int stride = gridDim.x, first_tile = blockIdx.x;
  auto tile_of = [&](int it) { return first_tile + it * stride; };

  if (warp == kEpiWarps) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&tmem_slot)), "r"(256));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  if (tid == 0) {
    auto init = [](uint64_t *b, int count) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(b)), "r"(count));
    };
    init(&bars.x, 1);
    init(&bars.h, 1);
    init(&bars.w, 1);
    init(&bars.part, 1);
    for (int k = 0; k < 2; k++) {
      init(&bars.layer[k], 1);
      init(&bars.epi[k], kEpiWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_mma_pending = 0;
  }
  for (int l = 0; l < NL; l++) {
    const float *bias = bias_of(a, l);
    const int ncol = layer_of(a.mode, l).epi == EPI_OUT ? 16 : 128;
    if (bias && tid < ncol) s_bias[l][tid] = bias[tid];
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;

  if (warp == kEpiWarps) {
    if (lane == 0) {
      const uint32_t bar_x = su32(&bars.x), bar_h = su32(&bars.h), bar_w = su32(&bars.w), bar_part = su32(&bars.part);
      const uint32_t idesc = static_cast<uint32_t>(
          cute::UMMA::make_instr_desc<cute::bfloat16_t, cute::bfloat16_t, float, 128, 128, cute::UMMA::Major::K,
                                      cute::UMMA::Major::K>());
      // barrier phases; a wait that gave up leaves its phase pending, and the
      // drain below waits for that same phase again
      uint32_t ph_x = 0, ph_h = 0, ph_w = 0, ph_part = 0;
      bool pend_x = false, pend_h = false, pend_w = false, pend_part = false, pend_layer = false;
      auto wait_on = [&](uint32_t bar, uint32_t &ph, bool &pend) {
        const bool ok = mbar_wait(bar, ph);
        if (ok) {
          ph ^= 1u;
          pend = false;
        }
        return ok;
      };
      int g = 0;     // the layer at work, counted over the tiles
      int done = 0;  // epilogues seen done
      auto wait_epilogues = [&](int count) {
        bool ok = true;
        while (ok && done < count) {
          ok = mbar_wait(su32(&bars.epi[done & 1]), (done >> 1) & 1);
          if (ok) done++;
        }
        return ok;
      };
      // the weight piece into its slot: one contiguous image of two atoms
      auto issue_weight = [&](int p) {
        mbar_expect(bar_w, kPieceBytes);
        bulk_load(sb + kOffW, a.piece[p].img, kPieceBytes, bar_w);
        pend_w = true;
      };
      auto issue_x = [&](int tile) {
        if (tile >= a.ntiles) return;
        mbar_expect(bar_x, 2 * kAtom);
        tma_load_box(sb + kOffX, &a.tm_a, 0, tile * 128, bar_x);
        tma_load_box(sb + kOffX + kAtom, &a.tm_a, 64, tile * 128, bar_x);
        pend_x = true;
      };
      auto issue_h = [&](int tile) {
        if (tile >= a.ntiles || a.mode == CHAIN_ENCODER) return;
        mbar_expect(bar_h, 2 * kAtom);
        tma_load_box(sb + kOffH, &a.tm_h, 0, tile * 128, bar_h);
        tma_load_box(sb + kOffH + kAtom, &a.tm_h, 64, tile * 128, bar_h);
        pend_h = true;
      };
      auto store = [&](const CUtensorMap *map, int off, int x, int row) {
        tma_store_box(map, sb + off, x, row);
        tma_store_box(map, sb + off + kAtom, x + 64, row);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      };
      // the stores so far have read shared memory
      auto stores_read = [] { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); };

      issue_weight(0);
      issue_x(first_tile);
      issue_h(first_tile);
      const bool pq = a.mode != CHAIN_LAST;  // the chain ends in [P | Q]
      const int h_piece = NP - 2;            // the first to read the finished h
      bool ok = true;
      for (int it = 0; ok && tile_of(it) < a.ntiles; it++) {
        const int row0 = tile_of(it) * 128;
        for (int p = 0; p < NP; p++) {
          const PieceSpec ps = piece_of(a.mode, p);
          ok = wait_on(bar_w, ph_w, pend_w);
          if (ok && p == 0) ok = wait_on(bar_x, ph_x, pend_x);
          if (ok && p == 1 && a.mode != CHAIN_ENCODER) ok = wait_on(bar_h, ph_h, pend_h);
          // the operand is the last layer's result, or else the accumulator
          // is that of the layer before it
          if (ok) ok = wait_epilogues(ps.after ? g : g - 1);
          if (!ok) break;
          if (p == h_piece && a.store_h) store(&a.tm_hout, kOffH, 0, row0);
          if (p == NP - 1 && pq) stores_read();  // Q will overwrite h
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          issue_piece(tmem + 128 * (g & 1), sb + (ps.a == BUF_X ? kOffX : kOffH), sb + kOffW, idesc, !ps.first,
                      ps.last ? su32(&bars.layer[g & 1]) : bar_part);
          (ps.last ? pend_layer : pend_part) = true;
          if (p == 0 && it > 0 && pq) {
            stores_read();  // the last tile's Q
            issue_h(tile_of(it));
          }
          if (ps.last) {
            ok = mbar_wait(su32(&bars.layer[g & 1]), (g >> 1) & 1);
            if (!ok) break;
            pend_layer = false;
            g++;
          } else {
            ok = wait_on(bar_part, ph_part, pend_part);
            if (!ok) break;
          }
          if (p + 1 < NP)
            issue_weight(p + 1);
          else if (tile_of(it + 1) < a.ntiles)
            issue_weight(0);
          if (!pq && p == 4) issue_h(tile_of(it + 1));
          if (!pq && p == 5) issue_x(tile_of(it + 1));
        }
        if (ok && pq) {
          ok = wait_epilogues(g - 1);
          if (!ok) break;
          store(&a.tm_pq, kOffX, 0, row0);
          stores_read();
          issue_x(tile_of(it + 1));
          ok = wait_epilogues(g);
          if (!ok) break;
          store(&a.tm_pq, kOffH, 128, row0);
        }
      }
      // normal end or a failed wait: let every copy, store or MMA in flight
      // land (bounded again).  An MMA that still has not completed may write
      // the accumulator: its TMEM is then left allocated rather than freed
      // under it.
      bool mma_done = true;
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
      if (pend_x) mbar_wait(bar_x, ph_x);
      if (pend_h) mbar_wait(bar_h, ph_h);
      if (pend_w) mbar_wait(bar_w, ph_w);
      if (pend_part && !mbar_wait(bar_part, ph_part)) mma_done = false;
      if (pend_layer && !mbar_wait(su32(&bars.layer[g & 1]), (g >> 1) & 1)) mma_done = false;
      if (!ok || !mma_done) atomicOr(a.err, ERR_TIMEOUT);
      if (!mma_done) s_mma_pending = 1;
    }
    __syncwarp();
  } else {
    const int r = (warp & 3) * 32 + lane;  // tile row = TMEM lane of this thread
    const int half = warp >> 2;            // columns [64 half, 64 half + 64): one atom
    bool ok = true;
    int g = 0;
    for (int it = 0; ok && tile_of(it) < a.ntiles; it++) {
      const int row0 = tile_of(it) * 128;
      for (int l = 0; l < NL; l++, g++) {
        const LayerSpec ls = layer_of(a.mode, l);
        ok = mbar_wait(su32(&bars.layer[g & 1]), (g >> 1) & 1);
        // h was written by TMA: its readers wait for its barrier themselves
        if (ok && ls.epi == EPI_RESIDUAL) ok = mbar_wait(su32(&bars.h), it & 1);
        // Each thread polls on its own clock, so a wait can give up in some
        // threads only; the warp-wide TMEM loads below need the whole warp.
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t taddr = tmem + 128 * (g & 1) + (static_cast<uint32_t>((warp & 3) * 32) << 16);
        const bool biased = bias_of(a, l) != nullptr;
        if (ls.epi == EPI_OUT) {
          if (half == 0) {
            float v[16];
            tmem_ld16(taddr, v);
            const int grow = row0 + r;
#pragma unroll
            for (int j = 0; j < 16; j++) v[j] += s_bias[l][j];
            if (grow < a.n) {
              float4 *dst = reinterpret_cast<float4 *>(a.out + (size_t)grow * 128);
#pragma unroll
              for (int j = 0; j < 4; j++) dst[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            }
          }
        } else {
          float v[64];
          tmem_ld64(taddr + 64 * half, v);
          if (biased)
#pragma unroll
            for (int j = 0; j < 64; j++) v[j] += s_bias[l][64 * half + j];
          uint8_t *buf = sm + (ls.epi == EPI_X ? kOffX : kOffH);
#pragma unroll
          for (int q = 0; q < 4; q++) {
            float *w = v + 16 * q;
            const int c0 = 64 * half + 16 * q;
            if (ls.epi == EPI_RESIDUAL) {
              float h[16];
              smem_get16(buf, r, c0, h);
#pragma unroll
              for (int j = 0; j < 16; j++) w[j] += h[j];
            }
            if (ls.relu)
#pragma unroll
              for (int j = 0; j < 16; j++) w[j] = fmaxf(w[j], 0.0f);
            smem_put16(buf, r, c0, w);
          }
        }
        // results -> visible to the next MMA and the TMA stores
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(su32(&bars.epi[g & 1]));
      }
    }
    if (!ok) atomicOr(a.err, ERR_TIMEOUT);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kEpiWarps && !s_mma_pending)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256));
}

__global__ void k_swizzle_image(const __nv_bfloat16 *__restrict__ W, int N, int K, uint8_t *__restrict__ img)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // one 16-byte chunk
  const int chunks = K / 8;
  if (i >= N * chunks) return;
  const int row = i / chunks, c = i % chunks;
  const int ka = c / 8, cc = c % 8;
  const uint4 v = *reinterpret_cast<const uint4 *>(W + (size_t)row * K + c * 8);
  *reinterpret_cast<uint4 *>(img + (size_t)ka * N * 128 + row * 128 + ((cc ^ (row & 7)) << 4)) = v;
}

}  // namespace

namespace {
uph_status encode_map(CUtensorMap *map, CUtensorMapDataType type, int elem, const void *base, int rows, int cols,
                      int row_bytes, int box_rows)
{
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  if (!encode) {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    const cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q);
    if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn)
      return fail(UPH_CUDA_ERROR, "cuTensorMapEncodeTiled is not available from the driver");
    encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (row_bytes & 15) || rows < 1 || cols < 1 || (cols * elem) % 16)
    return fail(UPH_BAD_ARG, "tensor map: base, row stride and columns must be whole 16-byte words");
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(row_bytes)};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(128 / elem), static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  const CUresult r = encode(map, type, 2, const_cast<void *>(base), dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(UPH_CUDA_ERROR, "cuTensorMapEncodeTiled failed");
  return UPH_OK;
}
}  // namespace

uph_status make_tensor_map(CUtensorMap *map, const void *base, int rows, int cols, int row_bytes, int box_rows)
{
  return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, rows, cols, row_bytes, box_rows);
}

uph_status make_f32_map(CUtensorMap *map, const void *base, int rows, int cols, int row_bytes)
{
  return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, rows, cols, row_bytes, 128);
}

uph_status make_row_tensor_map(CUtensorMap *map, const void *base, int rows, int cols, int row_bytes)
{
  if (cols % 64) return fail(UPH_BAD_ARG, "tensor map: columns must be whole boxes");
  return make_tensor_map(map, base, rows, cols, row_bytes, 128);
}

void launch_swizzle_image(const __nv_bfloat16 *W, int N, int K, uint8_t *img, cudaStream_t s)
{
  const int chunks = N * (K / 8);
  k_swizzle_image<<<(chunks + 255) / 256, 256, 0, s>>>(W, N, K, img);
}

uph_status launch_node_chain(const ChainArgs &a, cudaStream_t s)
{
  if (a.n < 1 || a.ntiles != (a.n + 127) / 128) return fail(UPH_BAD_ARG, "node chain: bad tile count");
  for (int p = 0; p < (a.mode == CHAIN_ENCODER ? 4 : 6); p++)
    if (!a.piece[p].img || (reinterpret_cast<uintptr_t>(a.piece[p].img) & 15))
      return fail(UPH_BAD_ARG, "node chain: missing or misaligned weight piece");
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    UPH_CUDA(cudaGetDevice(&dev));
    UPH_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    UPH_CUDA(cudaFuncSetAttribute(k_node_chain, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
  }
  const int grid = a.ntiles < 2 * sms ? a.ntiles : 2 * sms;
  k_node_chain<<<grid, kThreads, kSmemBytes, s>>>(a);
  UPH_CUDA(cudaGetLastError());
  return UPH_OK;
}

}  // namespace uph
