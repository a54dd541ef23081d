// BF16 tensor-core GEMM on sm_100a (tcgen05), FP32 accumulation in TMEM.
//
//   C[M x N] = A[M x K] . B[N x K]^T  (+ bias[N], optional ReLU)
//
// An operand is row-major with K contiguous ("K-major") or stored transposed
// ([K x rows], rows contiguous, "MN-major"); K a multiple of 64, N of 128.
// One CTA of 128 threads computes a 128 x 128 tile of C over a K range (the
// whole K, or one split of it):
//   - one thread fetches slices of 64 K by TMA (2-D tensor maps, 128-byte
//     swizzle, no multicast; rows beyond the matrix read as zero) into a ring
//     of stages, each with an mbarrier that counts its bytes.  A K-major
//     slice is one box of 128 rows x 64 K; an MN-major slice two boxes of 64 K
//     x 64 rows, which the UMMA reads as they lie;
//   - the same thread issues four tcgen05.mma per slice (M = 128, N = 128,
//     K = 16 each, kind::f16 with BF16 inputs) into a 128-column FP32
//     accumulator in TMEM and commits them to the stage's second mbarrier,
//     after which the stage is refilled;
//   - after the last slice, what the epilogue reads (a residual, a mask, the
//     old result) arrives by TMA in the stages' memory, each warp reads its 32
//     TMEM lanes (one output row per thread) with tcgen05.ld, and the results
//     leave as TMA tensor stores of swizzled boxes.  (Rows stored and read by
//     their threads, 32 bytes at a time, took 33 us where this takes 19.)
// Split-K launches write FP32 partial tiles that k_splitk_reduce sums in a
// fixed order (deterministic), and with them, where asked for, the column
// sums of a transposed A (a bias gradient beside its weight gradient), taken
// from the staged slices.
//
// Bound by memory and latency (K is 128 or 256): two stages hold a whole K of
// 128, so a row GEMM's CTA waits once for its loads, and three CTAs per SM
// (64 KB each) overlap their phases; a split-K CTA streams four stages.
// At 83,000 rows, N = K = 128, cold caches: 19 us a row GEMM and 15 + 7 us a
// split-K product and its sum, against 67 and up to 131 + 15 with the same tiles fed
// by 16-byte (for transposed operands 2-byte) stores of the threads, one slice
// at a time, and column sums as passes of their own.
//
// Every mbarrier wait is bounded; a wait that gives up sets ERR_TIMEOUT in the
// error word, and the CTA still frees its TMEM before returning.
#include <cuda_bf16.h>

#include <cute/arch/mma_sm100_desc.hpp>
#include <cute/numeric/numeric_types.hpp>

#include "node_chain.cuh"
#include "uph_internal.cuh"
#include "uph_surrogate.h"

namespace uph {

constexpr int kTcM = 128;       // rows of C per CTA (UMMA M)
constexpr int kTcN = 128;       // columns of C per CTA (UMMA N)
constexpr int kTcBK = 64;       // K per shared-memory slice: one 128-byte swizzle atom row
constexpr int kTcUmmaK = 16;    // K of one tcgen05.mma of kind::f16
constexpr int kTcRowStages = 2, kTcSplitStages = 4;
constexpr int kTcTileBytes = kTcM * kTcBK * 2;  // 16 KiB, same for the B slice (kTcN rows)
constexpr int kTcBoxBytes = kTcTileBytes / 2;   // one box of an MN-major slice
constexpr int kTcExtraBytes = kTcM * kTcN * 2;  // the BF16 result beside an FP32 one
constexpr int tc_smem_bytes(int stages, bool extra) { return stages * 2 * kTcTileBytes + (extra ? kTcExtraBytes : 0) + 1024; }
constexpr long long kWaitLimit = 1LL << 26;     // poll cap; the time bound is kWaitNs

struct TcGemmArgs {
  CUtensorMap tm_a, tm_b;
  // the FP32 result (or its partials), the BF16 result and the BF16 matrix
  // the epilogue reads (the residual, else the mask)
  CUtensorMap tm_c32, tm_c16, tm_e16;
  int a_trans, b_trans;      // operand stored as [K x rows] (rows contiguous) instead of [rows x K]
  int M, N, K;               // K multiple of 64, N multiple of 128
  int k_per_split;           // multiple of 64
  const float *bias;         // [N] or null
  int relu;
  int masked;                // zero the result where tm_e16 <= 0
  int residual;              // add tm_e16 after the bias
  const __nv_bfloat16 *mask;  // the mask beside a residual, read by the threads, or null
  int ldm;
  int accumulate;            // add the result to tm_c32's contents
  int c32, c16;              // write tm_c32 / tm_c16
  float *partials;           // split-K whose tiles are not whole boxes: [splits][M][N] FP32 stored by the threads
  int split_rows;            // split-K: rows of tm_c32 per split (M), else 0
  float *col_partials;       // split-K, A transposed: [splits][M] sums of A over the split's K, or null
  unsigned *err;
  int stall;                 // self-test of the bounded waits (GemmCall::stall)
};

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory descriptor of a slice's 16 K from `smem_addr`, 128-byte
// swizzle (PTX ISA, tcgen05 shared memory descriptor).  K-major: rows of 128
// bytes, 8-row groups 1024 bytes apart (SBO), unit leading offset.  MN-major:
// K rows of 64 elements (128 bytes), groups of 8 K 1024 bytes apart (SBO), the
// next 64 elements of the rows one box further (LBO).
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr, bool mn_major)
{
  cute::UMMA::SmemDescriptor d;
  d.desc_ = 0;
  d.start_address_ = static_cast<uint16_t>(smem_addr >> 4);
  d.leading_byte_offset_ = mn_major ? kTcBoxBytes >> 4 : 1;
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

// one slice of an operand into the 16 KiB at `dst`: rows r0 .., K k0 ..
__device__ __forceinline__ void tma_slice(uint32_t dst, const CUtensorMap *map, bool trans, int r0, int k0, uint32_t bar)
{
#pragma unroll
  for (int c = 0; c < 2; c++) {
    if (c == 1 && !trans) break;
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            dst + c * kTcBoxBytes),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(trans ? r0 + 64 * c : k0), "r"(trans ? k0 : r0), "r"(bar)
        : "memory");
  }
}

__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar)
{
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_store(const CUtensorMap *map, uint32_t src, int x, int y)
{
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(src), "r"(x), "r"(y)
               : "memory");
}

// 32 consecutive TMEM columns of this warp's 32 lanes, waited for inside the
// same asm statement so that no use of the registers precedes the load
__device__ __forceinline__ void tmem_ld32(uint32_t addr, float v[32])
{
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr)
      : "memory");
#pragma unroll
  for (int j = 0; j < 32; j++) v[j] = __uint_as_float(r[j]);
}

// row r, columns [c0, c0 + 32) of a BF16 tile of two 64-column boxes, 128-byte
// swizzle
__device__ __forceinline__ void get32_bf16(const uint8_t *tile, int r, int c0, float v[32])
{
  const uint8_t *row = tile + (c0 >> 6) * kTcTileBytes + r * 128;
  const int q0 = (c0 & 63) >> 3;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const uint4 w = *reinterpret_cast<const uint4 *>(row + (((q0 + q) ^ (r & 7)) << 4));
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      v[8 * q + 2 * j] = __uint_as_float(u[j] << 16);
      v[8 * q + 2 * j + 1] = __uint_as_float(u[j] & 0xffff0000u);
    }
  }
}
__device__ __forceinline__ void put32_bf16(uint8_t *tile, int r, int c0, const float v[32])
{
  uint8_t *row = tile + (c0 >> 6) * kTcTileBytes + r * 128;
  const int q0 = (c0 & 63) >> 3;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    __align__(16) __nv_bfloat162 h[4];
#pragma unroll
    for (int j = 0; j < 4; j++) h[j] = __floats2bfloat162_rn(v[8 * q + 2 * j], v[8 * q + 2 * j + 1]);
    *reinterpret_cast<uint4 *>(row + (((q0 + q) ^ (r & 7)) << 4)) = *reinterpret_cast<uint4 *>(&h[0]);
  }
}

template <cute::UMMA::Major A, cute::UMMA::Major B>
__device__ __forceinline__ uint32_t tc_idesc()
{
  return static_cast<uint32_t>(
      cute::UMMA::make_instr_desc<cute::bfloat16_t, cute::bfloat16_t, float, kTcM, kTcN, A, B>());
}

// kBoth: the old result and a BF16 matrix are read, or a residual and a mask
// (forms that no layer of the network needs: in the layers' own kernel their
// checks and addresses would cost 0.6 us a product)
template <int kStages, bool kBoth>
__global__ void __launch_bounds__(128) k_tc_gemm(const __grid_constant__ TcGemmArgs g)
{
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full[kStages], freed[kStages];
  __shared__ uint64_t stall_bar;  // the self-test's barrier: initialised, never arrived at
  __shared__ uint64_t epi_bar;    // what the epilogue reads
  __shared__ uint32_t tmem_base_slot;
  __shared__ float s_bias[kTcN];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int m0 = blockIdx.x * kTcM, n0 = blockIdx.y * kTcN;
  const int kbeg = blockIdx.z * g.k_per_split;
  const int kend = min(g.K, kbeg + g.k_per_split);
  const int nslices = max(0, (kend - kbeg) / kTcBK);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool sums = g.col_partials && blockIdx.y == 0;

  if (warp == 0) {  // TMEM: 128 FP32 columns for the 128 x 128 accumulator
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)),
                 "r"(kTcN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  if (tid == 0) {
    for (int s = 0; s < kStages; s++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[s])));
      // the MMAs' commit, and every thread's reads of the slice for the sums
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&freed[s])), "r"(sums ? 129 : 1));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&stall_bar)));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&epi_bar)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (g.bias) s_bias[tid] = g.bias[n0 + tid];
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_slot;
  const bool at = g.a_trans != 0, bt = g.b_trans != 0;
  using cute::UMMA::Major;
  const uint32_t idesc = at ? (bt ? tc_idesc<Major::MN, Major::MN>() : tc_idesc<Major::MN, Major::K>())
                            : (bt ? tc_idesc<Major::K, Major::MN>() : tc_idesc<Major::K, Major::K>());
  // bytes of 16 K inside a slice
  const uint32_t astep = at ? 2 * 1024 : kTcUmmaK * 2, bstep = bt ? 2 * 1024 : kTcUmmaK * 2;
  auto fetch = [&](int s) {  // thread 0
    const int st = s % kStages;
    const uint32_t bar = smem_u32(&full[st]), ta = smem_u32(smem + st * 2 * kTcTileBytes);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(2 * kTcTileBytes) : "memory");
    tma_slice(ta, &g.tm_a, at, m0, kbeg + s * kTcBK, bar);
    tma_slice(ta + kTcTileBytes, &g.tm_b, bt, n0, kbeg + s * kTcBK, bar);
  };

  // the self-test waits for a phase that never completes: the bounded wait
  // gives up, no copy or MMA has been issued, and the CTA goes straight to
  // freeing its TMEM.  Every thread polls on its own clock, so a wait that
  // gives up near the limit can give up in some threads only: the outcome is
  // made uniform over the block before anyone acts on it.
  bool ok = g.stall ? mbar_wait(smem_u32(&stall_bar), 0u) : true;
  ok = __syncthreads_and(ok) != 0;
  int fetched = 0, issued = 0;  // slices whose copies / MMAs were issued (thread 0)
  if (tid == 0 && ok)
    for (; fetched < min(kStages, nslices); fetched++) fetch(fetched);
  float colsum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (tid == 0 || sums) {
    for (int s = 0; s < nslices && ok; s++) {
      const int st = s % kStages;
      const uint32_t parity = (uint32_t)((s / kStages) & 1);
      ok = mbar_wait(smem_u32(&full[st]), parity);
      if (!ok) break;
      const uint8_t *ta = smem + st * 2 * kTcTileBytes;
      if (tid == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a_addr = smem_u32(ta), b_addr = a_addr + kTcTileBytes;
#pragma unroll
        for (int kk = 0; kk < kTcBK / kTcUmmaK; kk++) {
          const uint64_t da = umma_desc_sw128(a_addr + kk * astep, at);
          const uint64_t db = umma_desc_sw128(b_addr + kk * bstep, bt);
          const uint32_t accumulate = (s > 0 || kk > 0) ? 1u : 0u;
          asm volatile(
              "{\n\t.reg .pred p;\n\t"
              "setp.ne.b32 p, %4, 0;\n\t"
              "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
              :
              : "r"(tmem), "l"(da), "l"(db), "r"(idesc), "r"(accumulate));
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_u32(&freed[st]))
                     : "memory");
        issued = s + 1;
      }
      if (sums) {
        // eight columns of A (16-byte chunk tid % 16 of a K row, which lies at
        // chunk ^ (k % 8) of its box) over the K rows tid / 16, + 8, ...
        const int cg = tid & 15, kr = tid >> 4;
        const uint8_t *col = ta + (cg >> 3) * kTcBoxBytes + kr * 128 + (((cg & 7) ^ kr) << 4);
#pragma unroll
        for (int k = 0; k < kTcBK / 8; k++) {
          const uint4 w = *reinterpret_cast<const uint4 *>(col + k * 1024);
          const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int j = 0; j < 4; j++) {
            colsum[2 * j] += __uint_as_float(u[j] << 16);
            colsum[2 * j + 1] += __uint_as_float(u[j] & 0xffff0000u);
          }
        }
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&freed[st])) : "memory");
      }
      // refill the stage of the slice before this one
      if (tid == 0 && s > 0 && fetched < nslices) {
        const int pr = (s - 1) % kStages;
        ok = mbar_wait(smem_u32(&freed[pr]), (uint32_t)(((s - 1) / kStages) & 1));
        if (ok) fetch(fetched++);
      }
    }
  }
  // Drain: thread 0 waits for every slice's copies and for every MMA, on the
  // normal path and after a failed wait alike, so that nothing still writes
  // shared memory or the accumulator when the CTA ends.  Waiting on a phase
  // that already completed returns at once.
  bool drained = true;
  if (tid == 0) {
    for (int s = max(0, fetched - kStages); s < fetched; s++)
      if (s >= issued && !mbar_wait(smem_u32(&full[s % kStages]), (uint32_t)((s / kStages) & 1))) drained = false;
    // a stage with the sums' arrivals missing (a failed wait elsewhere)
    // completes no phase: the last commits are then waited for below only on
    // the normal path, and the TMEM is left allocated
    for (int s = max(0, issued - kStages); s < issued; s++)
      if (!mbar_wait(smem_u32(&freed[s % kStages]), (uint32_t)((s / kStages) & 1))) drained = false;
  }
  drained = __syncthreads_and(drained) != 0;
  ok = __syncthreads_and(ok) != 0 && drained;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (ok && sums) {
    // the eight K groups of every column, added in order
    float *red = reinterpret_cast<float *>(smem);
    for (int j = 0; j < 8; j++) red[(tid >> 4) * kTcM + (tid & 15) * 8 + j] = colsum[j];
    __syncthreads();
    float t = red[tid];
    for (int k = 1; k < 8; k++) t += red[k * kTcM + tid];
    if (m0 + tid < g.M) g.col_partials[(size_t)blockIdx.z * g.M + m0 + tid] = t;
    __syncthreads();  // the epilogue reuses the memory
  }

  if (!ok) {
    if (threadIdx.x == 0) atomicOr(g.err, ERR_TIMEOUT);
  } else {
    // Regions of the stages' memory, free now.  FP32 (result, old result): 4
    // boxes of 32 columns, 64 KiB; BF16: 2 boxes of 64 columns, 32 KiB: the
    // result in the first half, or past the stages beside an FP32 result; the
    // matrix that is read in the second half (a row's FP32 result overwrites
    // there what its thread has used), or past the stages where the old result
    // arrives in both halves (a BF16 result then takes its place column by
    // column, as it is used).
    uint8_t *past = smem + kStages * 2 * kTcTileBytes;
    uint8_t *r32 = smem, *e16 = kBoth && g.accumulate ? past : smem + kTcM * kTcN * 2;
    uint8_t *r16 = g.c32 ? past : smem;
    const bool reads16 = g.masked || g.residual;
    if (reads16 || g.accumulate) {
      if (tid == 0) {
        const uint32_t bar = smem_u32(&epi_bar);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                     "r"((reads16 ? kTcM * kTcN * 2 : 0) + (g.accumulate ? kTcM * kTcN * 4 : 0))
                     : "memory");
        if (reads16)
          for (int c = 0; c < 2; c++) tma_load(smem_u32(e16) + c * kTcTileBytes, &g.tm_e16, n0 + 64 * c, m0, bar);
        if (g.accumulate)
          for (int c = 0; c < 4; c++) tma_load(smem_u32(r32) + c * kTcTileBytes, &g.tm_c32, n0 + 32 * c, m0, bar);
      }
      ok = mbar_wait(smem_u32(&epi_bar), 0u);
      if (!ok) atomicOr(g.err, ERR_TIMEOUT);
      // a wait that gave up: thread 0 lets the copies land (bounded again)
      if (!ok && tid == 0) mbar_wait(smem_u32(&epi_bar), 0u);
      ok = __syncthreads_and(ok) != 0;
    }
    // warp w owns TMEM lanes [32w, 32w + 32) = rows m0 + 32w + lane
    const int r = warp * 32 + lane, row = m0 + r;
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    if (ok) {
#pragma unroll 1
      for (int c0 = 0; c0 < kTcN; c0 += 32) {
        float v[32];
        tmem_ld32(lane_addr + c0, v);
        if (g.bias)
#pragma unroll
          for (int j = 0; j < 32; j++) v[j] += s_bias[c0 + j];
        if (g.residual) {
          float e[32];
          get32_bf16(e16, r, c0, e);
#pragma unroll
          for (int j = 0; j < 32; j++) v[j] += e[j];
        }
        uint8_t *f32row = r32 + (c0 >> 5) * kTcTileBytes + r * 128;
        if (g.accumulate)
#pragma unroll
          for (int q = 0; q < 8; q++) {
            const float4 o = *reinterpret_cast<const float4 *>(f32row + ((q ^ (r & 7)) << 4));
            v[4 * q] += o.x;
            v[4 * q + 1] += o.y;
            v[4 * q + 2] += o.z;
            v[4 * q + 3] += o.w;
          }
        if (g.relu)
#pragma unroll
          for (int j = 0; j < 32; j++) v[j] = fmaxf(v[j], 0.0f);
        if (g.masked) {
          float e[32];
          get32_bf16(e16, r, c0, e);
#pragma unroll
          for (int j = 0; j < 32; j++)
            if (!(e[j] > 0.0f)) v[j] = 0.0f;
        }
        if (kBoth && g.mask && row < g.M) {
          const __nv_bfloat16 *mk = g.mask + (size_t)row * g.ldm + n0 + c0;
#pragma unroll
          for (int j = 0; j < 32; j++)
            if (!(__bfloat162float(mk[j]) > 0.0f)) v[j] = 0.0f;
        }
        if (g.partials) {
          if (row < g.M) {
            float *dst = g.partials + ((size_t)blockIdx.z * g.M + row) * g.N + n0 + c0;
#pragma unroll
            for (int q = 0; q < 8; q++)
              *reinterpret_cast<float4 *>(dst + 4 * q) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
          }
          continue;
        }
        if (g.c32)
#pragma unroll
          for (int q = 0; q < 8; q++)
            *reinterpret_cast<float4 *>(f32row + ((q ^ (r & 7)) << 4)) =
                make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        if (g.c16) put32_bf16(r16, r, c0, v);
      }
      // generic-proxy shared stores -> visible to the TMA stores
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    if (tid == 0 && ok) {
      const int row0 = m0 + blockIdx.z * g.split_rows;
      if (g.c32)
        for (int c = 0; c < 4; c++) tma_store(&g.tm_c32, smem_u32(r32) + c * kTcTileBytes, n0 + 32 * c, row0);
      if (g.c16)
        for (int c = 0; c < 2; c++) tma_store(&g.tm_c16, smem_u32(r16) + c * kTcTileBytes, n0 + 64 * c, m0);
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  // an MMA that never completed may still write the accumulator: its TMEM
  // is then left allocated rather than freed under it (the error word
  // already says the tensor core stopped answering)
  if (warp == 0 && drained)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcN));
}

// out[i] (+)= sum over splits of partials[s][i], and the same for the column
// sums: groups of 8 threads take every 8th split of four values and are added
// in group order (a fixed order: deterministic).
constexpr int kReduceGroups = 8;
__global__ void __launch_bounds__(256) k_splitk_reduce(const float *__restrict__ partials, int splits, int count,
                                                       float *out, int accumulate,
                                                       const float *__restrict__ col_partials, int cols, float *col_out)
{
  __shared__ float4 red[kReduceGroups][256 / kReduceGroups];
  const int l = threadIdx.x & 31, grp = threadIdx.x >> 5;
  const int main_blocks = (count / 4 + 31) / 32;
  const bool is_col = (int)blockIdx.x >= main_blocks;
  const float *src = is_col ? col_partials : partials;
  const int n = is_col ? cols : count;
  const int i = (((int)blockIdx.x - (is_col ? main_blocks : 0)) * 32 + l) * 4;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (i < n)
    for (int s = grp; s < splits; s += kReduceGroups) {
      const float4 v = *reinterpret_cast<const float4 *>(src + (size_t)s * n + i);
      acc.x += v.x;
      acc.y += v.y;
      acc.z += v.z;
      acc.w += v.w;
    }
  red[grp][l] = acc;
  __syncthreads();
  if (grp != 0 || i >= n) return;
  float *dst = (is_col ? col_out : out) + i;
  // the caller's result need not lie on a 16-byte boundary
  const bool words = (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
  float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
  if (!is_col && accumulate) t = words ? *reinterpret_cast<const float4 *>(dst) : make_float4(dst[0], dst[1], dst[2], dst[3]);
#pragma unroll
  for (int k = 0; k < kReduceGroups; k++) {
    t.x += red[k][l].x;
    t.y += red[k][l].y;
    t.z += red[k][l].z;
    t.w += red[k][l].w;
  }
  if (words) {
    *reinterpret_cast<float4 *>(dst) = t;
  } else {
    dst[0] = t.x;
    dst[1] = t.y;
    dst[2] = t.z;
    dst[3] = t.w;
  }
}

uph_status launch_tc_gemm(const GemmCall &c, cudaStream_t s)
{
  if (!c.A || !c.B || !c.err || c.M <= 0 || c.N <= 0 || c.K <= 0) return fail(UPH_BAD_ARG, "tc_gemm: bad arguments");
  if (c.K % kTcBK || c.N % kTcN) return fail(UPH_BAD_ARG, "tc_gemm: K must be a multiple of 64, N of 128");
  const int ldc16 = c.ldc16 > 0 ? c.ldc16 : c.ldc;
  if (c.lda % 8 || c.ldb % 8 || c.ldc % 8 || ldc16 % 8 || (c.mask && c.ldm % 8) || (c.residual && c.ldr % 8))
    return fail(UPH_BAD_ARG, "tc_gemm: leading dimensions must be multiples of 8");
  if ((c.a_trans && c.M % 8) || (c.b_trans && c.N % 8))
    return fail(UPH_BAD_ARG, "tc_gemm: a transposed operand needs a multiple of 8 rows");
  int splits = c.splits < 1 ? 1 : c.splits;
  if (splits > 1 && (!c.partials || !c.c_f32 || c.bias || c.relu || c.c_bf16 || c.mask || c.residual || c.ldc != c.N))
    return fail(UPH_BAD_ARG, "tc_gemm: split-K writes a dense FP32 result only, without bias, ReLU or mask");
  if (splits == 1 && !c.c_f32 && !c.c_bf16) return fail(UPH_BAD_ARG, "tc_gemm: no output");
  if (splits == 1 && c.accumulate && !c.c_f32) return fail(UPH_BAD_ARG, "tc_gemm: accumulate needs c_f32");
  if (c.col_sums && (!c.a_trans || splits <= 1 || !c.col_partials || c.M % 4))
    return fail(UPH_BAD_ARG, "tc_gemm: column sums go with a split-K product of a transposed A");
  static bool configured = false;
  if (!configured) {
    UPH_CUDA(cudaFuncSetAttribute(k_tc_gemm<kTcRowStages, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  tc_smem_bytes(kTcRowStages, true)));
    UPH_CUDA(cudaFuncSetAttribute(k_tc_gemm<kTcRowStages, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  tc_smem_bytes(kTcRowStages, true)));
    UPH_CUDA(cudaFuncSetAttribute(k_tc_gemm<kTcSplitStages, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  tc_smem_bytes(kTcSplitStages, false)));
    configured = true;
  }
  TcGemmArgs g;
  const int kv = c.k_valid > 0 ? c.k_valid : c.K;
  auto map_of = [&](CUtensorMap *m, const void *base, int ld, int trans, int rows) {
    return trans ? make_tensor_map(m, base, kv, rows, ld * 2, 64) : make_tensor_map(m, base, rows, c.K, ld * 2, kTcM);
  };
  uph_status tr = map_of(&g.tm_a, c.A, c.lda, c.a_trans, c.M);
  if (tr == UPH_OK) tr = map_of(&g.tm_b, c.B, c.ldb, c.b_trans, c.N);
  if (tr != UPH_OK) return tr;
  g.a_trans = c.a_trans;
  g.b_trans = c.b_trans;
  g.M = c.M;
  g.N = c.N;
  g.K = c.K;
  int kps = c.K;
  if (splits > 1) kps = ((c.K / kTcBK + splits - 1) / splits) * kTcBK;
  g.k_per_split = kps;
  splits = (c.K + kps - 1) / kps;
  g.bias = c.bias;
  g.relu = c.relu;
  g.masked = c.mask && !c.residual;
  g.mask = c.residual ? (const __nv_bfloat16 *)c.mask : nullptr;
  g.ldm = c.ldm;
  g.residual = c.residual != nullptr;
  g.accumulate = splits > 1 ? 0 : c.accumulate;
  // split-K partials leave by TMA where a split's tiles are whole boxes
  const bool split = splits > 1, boxed = !split || c.M % kTcM == 0;
  g.partials = split && !boxed ? c.partials : nullptr;
  g.split_rows = split ? c.M : 0;
  g.c32 = split ? boxed : c.c_f32 != nullptr;
  g.c16 = !split && c.c_bf16;
  if (g.c32) {
    tr = split ? make_f32_map(&g.tm_c32, c.partials, splits * c.M, c.N, c.N * 4)
               : make_f32_map(&g.tm_c32, c.c_f32, c.M, c.N, c.ldc * 4);
    if (tr != UPH_OK) return tr;
  }
  if (g.c16) tr = make_tensor_map(&g.tm_c16, c.c_bf16, c.M, c.N, ldc16 * 2, kTcM);
  if (tr == UPH_OK && g.masked) tr = make_tensor_map(&g.tm_e16, c.mask, c.M, c.N, c.ldm * 2, kTcM);
  if (tr == UPH_OK && c.residual) tr = make_tensor_map(&g.tm_e16, c.residual, c.M, c.N, c.ldr * 2, kTcM);
  if (tr != UPH_OK) return tr;
  const bool both = (c.mask && c.residual) || (g.accumulate && (c.mask || c.residual));
  g.col_partials = splits > 1 && c.col_sums ? c.col_partials : nullptr;
  g.err = c.err;
  g.stall = c.stall;
  dim3 grid((c.M + kTcM - 1) / kTcM, c.N / kTcN, splits);
  if (splits > 1)
    k_tc_gemm<kTcSplitStages, false><<<grid, 128, tc_smem_bytes(kTcSplitStages, false), s>>>(g);
  else if (both)
    k_tc_gemm<kTcRowStages, true><<<grid, 128, tc_smem_bytes(kTcRowStages, true), s>>>(g);
  else
    k_tc_gemm<kTcRowStages, false><<<grid, 128, tc_smem_bytes(kTcRowStages, g.c32 && g.c16), s>>>(g);
  if (splits > 1) {
    const int count = c.M * c.N, cols = c.col_sums ? c.M : 0;
    const int blocks = (count / 4 + 31) / 32 + (cols / 4 + 31) / 32;
    k_splitk_reduce<<<blocks, 256, 0, s>>>(c.partials, splits, count, c.c_f32, c.accumulate, c.col_partials, cols,
                                           c.col_sums);
  }
  UPH_CUDA(cudaGetLastError());
  return UPH_OK;
}

}  // namespace uph

using namespace uph;

// C ABI for tests: device pointers, both operands K-major.  splits > 1
// requires `partials` of splits * M * N floats and writes the sum into c_f32
// (accumulated onto its contents when accumulate != 0).
extern "C" uph_status uph_tc_gemm_bf16(const void *A, int32_t lda, const void *B, int32_t ldb, int32_t M, int32_t N,
                                       int32_t K, const float *bias, int32_t relu, float *c_f32, void *c_bf16,
                                       int32_t ldc, int32_t splits, float *partials, int32_t accumulate,
                                       unsigned *err, void *stream)
{
  GemmCall c;
  c.A = A;
  c.lda = lda;
  c.B = B;
  c.ldb = ldb;
  c.M = M;
  c.N = N;
  c.K = K;
  c.bias = bias;
  c.relu = relu;
  c.c_f32 = c_f32;
  c.c_bf16 = c_bf16;
  c.ldc = ldc;
  c.splits = splits;
  c.partials = partials;
  c.accumulate = accumulate;
  c.err = err;
  return launch_tc_gemm(c, (cudaStream_t)stream);
}

// C ABI for tests: a row product with the whole epilogue (GemmCall); mask and
// residual are BF16 [M x ldc] or null.
extern "C" uph_status uph_tc_gemm_bf16_epilogue(const void *A, int32_t lda, const void *B, int32_t ldb, int32_t M,
                                                int32_t N, int32_t K, const float *bias, const void *residual,
                                                int32_t accumulate, int32_t relu, const void *mask, float *c_f32,
                                                void *c_bf16, int32_t ldc, unsigned *err, void *stream)
{
  GemmCall c;
  c.A = A;
  c.lda = lda;
  c.B = B;
  c.ldb = ldb;
  c.M = M;
  c.N = N;
  c.K = K;
  c.bias = bias;
  c.residual = residual;
  c.ldr = ldc;
  c.accumulate = accumulate;
  c.relu = relu;
  c.mask = mask;
  c.ldm = ldc;
  c.c_f32 = c_f32;
  c.c_bf16 = c_bf16;
  c.ldc = ldc;
  c.err = err;
  return launch_tc_gemm(c, (cudaStream_t)stream);
}

// Failure-detection self test: one tile whose CTA waits on a barrier nothing
// arrives at.  The bounded wait gives up, the kernel sets ERR_TIMEOUT, frees
// its TMEM and returns; the context stays usable.
extern "C" uph_status uph_tc_wait_selftest(const void *A, const void *B, float *c_f32, unsigned *err, void *stream)
{
  if (!A || !B || !c_f32 || !err) return fail(UPH_BAD_ARG, "uph_tc_wait_selftest: NULL argument");
  cudaStream_t q = (cudaStream_t)stream;
  GemmCall c;
  c.A = A;
  c.lda = kTcBK;
  c.B = B;
  c.ldb = kTcBK;
  c.M = kTcM;
  c.N = kTcN;
  c.K = kTcBK;
  c.c_f32 = c_f32;
  c.ldc = kTcN;
  c.err = err;
  c.stall = 1;
  UPH_CUDA(cudaMemsetAsync(err, 0, sizeof(unsigned), q));
  uph_status r = launch_tc_gemm(c, q);
  if (r != UPH_OK) return r;
  unsigned e = 0;
  UPH_CUDA(cudaMemcpyAsync(&e, err, sizeof e, cudaMemcpyDeviceToHost, q));
  UPH_CUDA(cudaStreamSynchronize(q));
  if (e & ERR_TIMEOUT) return fail(UPH_TIMEOUT, "uph_tc_wait_selftest: the wait gave up as intended");
  return UPH_OK;
}
