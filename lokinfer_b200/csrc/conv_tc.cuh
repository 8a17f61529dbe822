// Device code and types shared by the tensor-core convs (conv_tc.cu, conv_pair.cu): constants of their common structure, PTX
// wrappers, bounded waits, descriptors, the activation prologue.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>

#include "lkc_common.h"

#ifndef LKC_TC_PROF
#define LKC_TC_PROF 0  // 1: role-level cycle counters (lkc_conv1d_tc_profile); a build option, off in the product
#endif

namespace lkc {
namespace tc {

constexpr bool kProf = LKC_TC_PROF != 0;
constexpr int NT = 256;         // time columns per tile (= UMMA N)
constexpr int NTS = 128;        // time columns per tile of the split form: one statistics chunk
constexpr int NTS2 = 64;        // the same for rows of no more columns
constexpr int MT = 128;         // output channels per tile (= UMMA M)
constexpr int KC = 16;          // input channels per staged chunk (one weight stage, two K8 steps)
constexpr int MAX_NB = 4;       // most activation (hi / lo) buffers
constexpr int NRAW = 2;         // raw-input staging buffers, filled one chunk ahead
constexpr int EPI_WARPS = 8, PRO_WARPS = 8;
constexpr int W_WARP = EPI_WARPS + PRO_WARPS, MMA_WARP = W_WARP + 1, RAW_WARP = W_WARP + 2;
constexpr int NWARPS = EPI_WARPS + PRO_WARPS + 4;
constexpr int NTHREADS = NWARPS * 32;  // 640
// setmaxnreg takes one value per warpgroup: 0-1 epilogue, 2-3 producers, 4 control
constexpr int LAUNCH_REGS = 96, EPI_REGS = 160, PRO_REGS = 56, CTL_REGS = 48;
static_assert(NTHREADS * LAUNCH_REGS <= 65536, "launch register budget");
// setmaxnreg moves registers inside the CTA's own launch allocation (NTHREADS * LAUNCH_REGS); an increase beyond what
// the decreases release would block forever.
static_assert(EPI_WARPS * 32 * EPI_REGS + PRO_WARPS * 32 * PRO_REGS + (NWARPS - EPI_WARPS - PRO_WARPS) * 32 * CTL_REGS <=
                  NTHREADS * LAUNCH_REGS,
              "register pool");
// Operand formats (template parameter F16 of the kernel):
//   tf32 split (F16 = false): hi = tf32(v), lo = v - hi, both stored as f32; per tap and 16 channels 6 MMAs of
//     kind::tf32 (K8): 2 x hi*hi into Dhi, 2 x (lo*hi + hi*lo) into Dlo.
//   f16 split (F16 = true): hi = f16(v), lo = f16((v - hi) * 2^11), both with the same 11-bit significand as tf32;
//     per tap and 16 channels 3 MMAs of kind::f16 (K16): hi*hi into Dhi, lo*hi + hi*lo into Dlo, which is folded in
//     with the factor 2^-11. Products are exact and accumulate in f32 as before, so the accuracy is that of the
//     tf32 split at half the tensor time, half the staged bytes and half the weight traffic. Values beyond the f16
//     range (|v| > 65504) are flagged in the status word: an activation becomes an infinite f16 operand (the output
//     of that launch is then not finite; kStatusF16Range), a weight is clamped at pack time (kStatusF16Weights).
constexpr float kLoScale = 2048.f;  // 2^11
constexpr int kStatusF16Range = 0x10000, kStatusF16Weights = 0x20000, kStatusWaitMask = 0xffff;
template <bool F16>
struct Fmt {
  static constexpr int W_STAGE_BYTES = F16 ? 2 * MT * KC * 2 : 2 * MT * KC * 4;  // hi + lo of [128 co x 16 ci]
  static constexpr int W_STAGE_FLOATS = W_STAGE_BYTES / 4;
  static constexpr int NB = F16 ? 3 : 2;  // activation (hi / lo) buffers; the f16 ones are half the size
  static constexpr int ACT_BYTES_PER_ROW = F16 ? 2 * KC * 2 : 2 * KC * 4;  // hi + lo of one time row, 16 channels
};
constexpr int STAGE_PITCH = 33;  // floats per row of an epilogue transpose tile (unaligned route)
constexpr int STAGE_FLOATS = 32 * STAGE_PITCH;
constexpr int BOX = 32, BOX_BYTES = BOX * BOX * 4;  // residual / output boxes of the aligned route: 32 co x 32 t
static_assert(BOX_BYTES <= STAGE_FLOATS * 4, "a swizzled box fits in a warp's tile");
// Floats per row of a split tile's partial: rows 16-byte aligned, 4 banks apart.
__host__ __device__ constexpr int partPitch(int cols) { return cols + 4; }
// A split tile's memory behind its MMAs, over the operand buffers: this CTA's partial tile, then the rows that the CTAs of the
// cluster send it. Those are at most split * (rows a CTA owns, rounded up; 2 channels of 10 rows and a gap of 2 over 8 CTAs).
constexpr int PART_ROWS = 176;
__host__ __device__ constexpr int partBytes(int cols) { return MT * partPitch(cols) * 4; }
__host__ __device__ constexpr int recvBytes(int cols) { return PART_ROWS * partPitch(cols) * 4; }
constexpr size_t SPLIT_SMEM = 120 * 1024;  // more than half an SM's: one CTA per SM, for whose TMEM two would compete
constexpr int MAX_SPLIT = 8;     // CTAs of a split tile (the portable cluster size)
static_assert(MAX_SPLIT <= EPI_WARPS, "an epilogue warp per receiver");
constexpr int MAX_HALO = 50;     // (K - 1) * dilation of the widest Kokoro conv (K 11, dilation 5)
constexpr int MAX_W_STAGES = 4, MIN_W_STAGES = 2, PREF_W_STAGES = 2;  // weight ring slots
constexpr int TAP_GROUP = 6;  // most taps per weight slot: one bulk copy, one wait, MMAs back to back, one release
constexpr int MAX_CHAIN = 24;  // most chained hi MMAs between two drains of Dhi
// The same of a pointwise conv with tf32 halves, whose alternative is one f32 sum over the channels on the CUDA cores.
// The drift of a chain of 24 made it the less exact of the two below about 700 channels. Error against float64 (1e-7 of
// the result) of the decoder's 528- and 512-channel convs over 8..1040 columns: CUDA cores 1.2-2.8 and 3.8-4.2, chains of
// 24: 1.5-3.2 and 4.5-4.7, of 12: 1.1-2.0 and 2.6-2.7, of 8: 0.9-1.6 and 1.9-2.2; of its 1104-channel convs: CUDA cores
// 4.3-5.4, chains of 24: 3.5-4.4, of 8: 1.6-1.9. 528 -> 1024 channels at 320 columns: 42.9 us at 24, 43.5 at 8.
constexpr int MAX_CHAIN_POINT32 = 8;
constexpr uint32_t SPIN_LIMIT = 1u << 24;
constexpr uint32_t SLEEP_EPI_NS = 256, SLEEP_EPI_SPLIT_NS = 64, SLEEP_PRO_NS = 128, SLEEP_W_NS = 64, SLEEP_MMA_NS = 32;
constexpr uint64_t WAIT_LIMIT_NS = 200ull * 1000 * 1000;  // 0.2 s: a healthy wait is tens of microseconds
constexpr int kMaxSmem = 232448;  // 227 KB per CTA on sm_100

struct TcArgs {
  const float *x, *wp, *bias, *affine, *alpha, *residual;
  const float *statsIn, *gb;  // split form: the AdaIN affine of x is computed here from its chunk statistics (null: `affine`)
  float eps;
  float *out, *stats;
  int ci, co, k, dilation, padding;
  int64_t l, lo, nchunks;
  int64_t validLo, validHi;            // x columns outside [validLo, validHi) are zero padding (after the activation)
  int64_t xPitch, resPitch, outPitch;  // row pitches in floats
  int padLeft;       // ConvTranspose: 1 = one-sample left reflect pad
  float slope, outScale;
  int delta;       // columns between the 16-byte boundary a tile's window is loaded from and its first column (0: 4-byte route)
  int tileCols;    // time columns per tile: NTS or NTS2 split, 160 or NTS in pairs, else 160 .. NT in steps of 32 (see tileColsFor)
  int mainRows;    // staged rows that every lane has a slot for: the window up to NT (split: tileCols) rows, a multiple of 64
  int rows;        // staged time rows per buffer: at least tileCols + (k-1)*dilation + delta and mainRows
  int ext;         // raw staging: [16][NT, split: tileCols], then [16][ext] with the rows beyond them (two TMA boxes)
  int wStages;     // weight ring depth (slots)
  int nb;          // activation buffers
  int wG;          // taps per weight slot: the k taps of a chunk go in ceil(k / wG) groups of near-equal size
  int drainN;      // 16-channel chunks accumulated in Dhi between two drains into the running sums
  int tmaIn;       // 1: x rows are 16-byte aligned, the raw windows come by tiled TMA loads
  int tmaOut;      // 1: out (and residual) rows are 16-byte aligned, boxes go by TMA
  int numTTiles, numCoBlk;
  int split;       // 0 = a persistent CTA per SM over tiles of tileCols columns; else the CTAs that share one such tile
  int pair;        // 1: tiles of CTA pairs (conv_pair.cu)
  int nRaw;        // CTA pairs: raw-input staging buffers
  int early;       // the launch may overlap the end of the one before it (programmatic dependent launch)
  int* status;
  long long* prof;  // null, or 16 cycle counters summed over CTAs (see convTcProfile)
};

// ---------------------------------------------------------------------------------------------- PTX helpers

__device__ __forceinline__ uint32_t smemAddr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbarInit(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smemAddr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbarArrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smemAddr(bar)) : "memory");
}
__device__ __forceinline__ void mbarArriveExpectTx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smemAddr(bar)), "r"(bytes) : "memory");
}
// One poll. Without a suspend-time hint the hardware parks the thread only briefly, which keeps the wake-up latency of
// the hand-offs low (a 1 ms hint measured 3-7 % slower end to end).
__device__ __forceinline__ bool mbarTryWait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smemAddr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ uint64_t globalTimerNs() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// One poll that never parks the thread.
__device__ __forceinline__ bool mbarTestWait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smemAddr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: gives up (false) after SPIN_LIMIT polls or WAIT_LIMIT_NS of wall time, whichever comes first, or as
// soon as another role has aborted. Between polls the warp sleeps `sleepNs`: the warp scheduler issues greedily from
// a ready warp, so a tight spin loop starves the producer warps that share its scheduler (measured: the producers
// ran at a tenth of their instruction rate next to spinning epilogue warps). Latency-critical waiters pass 0.
__device__ __forceinline__ bool mbarWait(uint64_t* bar, uint32_t parity, volatile int* abortFlag, uint32_t sleepNs) {
  if (mbarTryWait(bar, parity)) return true;
  const uint64_t t0 = globalTimerNs();
  for (uint32_t spins = 0; !mbarTryWait(bar, parity); ++spins) {
    if (sleepNs) __nanosleep(sleepNs);
    if (*abortFlag || spins >= SPIN_LIMIT) return false;
    if ((spins & 63) == 63 && globalTimerNs() - t0 > WAIT_LIMIT_NS) return false;
  }
  return true;
}
// Wait without the abort check, for draining copies in flight after an abort (bounded all the same).
__device__ __forceinline__ void mbarWaitQuiet(uint64_t* bar, uint32_t parity) {
  const uint64_t t0 = globalTimerNs();
  uint32_t spins = 0;
  while (!mbarTryWait(bar, parity) && ++spins < SPIN_LIMIT && globalTimerNs() - t0 < WAIT_LIMIT_NS) {
  }
}
__device__ __forceinline__ void fenceProxyAsync() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fenceBarrierInit() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void tcFenceBefore() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcFenceAfter() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void bulkCopyG2S(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smemAddr(dst)),
               "l"(src), "r"(bytes), "r"(smemAddr(bar))
               : "memory");
}
// Tiled TMA copies of a rank-2 tensor (coordinates: x = innermost = time, y = channel). x * 4 bytes must be a
// multiple of 16; a load may start outside the tensor (the missing part is filled with zeros), a store is clipped behind the 16 bytes
// that the last column is in.
__device__ __forceinline__ void tmaLoad2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smemAddr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smemAddr(bar))
      : "memory");
}
__device__ __forceinline__ void tmaStore2d(const CUtensorMap* map, int x, int y, const void* src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(x), "r"(y), "r"(smemAddr(src))
               : "memory");
}
__device__ __forceinline__ void bulkCommit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// Until the bulk stores of this thread have read their shared-memory source / have completed.
__device__ __forceinline__ void bulkWaitRead() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulkWaitAll() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ void cpAsync4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smemAddr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cpAsyncCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpAsyncWait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void tmemAlloc(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(slot)), "r"(cols)
               : "memory");
}
__device__ __forceinline__ void tmemRelinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmemDealloc(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
// Clusters: this CTA's rank, the two halves of the barrier of all threads of all its CTAs, and the address of another CTA's copy of
// this CTA's shared memory.
// The arrivals are relaxed: they order nothing in front of them. What the CTAs send each other, rows or signals, is waited for
// at an mbarrier, whose initialisation has its own fence; the cluster barriers only say that operand buffers are read and that nobody
// needs this CTA any more. As releases they waited for every store in flight, spills and output rows included: us per forward
// 313 -> 299 at T = 24, 551 -> 540 at T = 121, the decoder at F = 8 / 61 / 160 / 1040 177 -> 171, 183 -> 177, 260 -> 254, 570 -> 561.
__device__ __forceinline__ uint32_t clusterRank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void clusterArrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}
__device__ __forceinline__ void clusterWait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t peerAddr(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// Bulk copy into another CTA's shared memory, counted by a barrier there (both as peerAddr gives them).
__device__ __forceinline__ void bulkCopyPeer(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "r"(smemAddr(src)), "r"(bytes), "r"(bar)
               : "memory");
}
// D[tmem] (+)= A[smem desc] * B[smem desc], kind::tf32, issued by one thread.
__device__ __forceinline__ void mmaTf32(uint32_t dTmem, uint64_t descA, uint64_t descB, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(dTmem),
      "l"(descA), "l"(descB), "r"(idesc), "r"(accum)
      : "memory");
}
// kind::f16 with the descriptors given as (low word, high word): only the low word (address and leading-dimension
// fields) changes between taps, so the issuing thread does its descriptor arithmetic in 32 bits.
__device__ __forceinline__ void mmaF16W(uint32_t dTmem, uint32_t aLo, uint32_t aHi, uint32_t bLo, uint32_t bHi,
                                        uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "mov.b64 da, {%1, %2};\n\t"
      "mov.b64 db, {%3, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}" ::"r"(dTmem),
      "r"(aLo), "r"(aHi), "r"(bLo), "r"(bHi), "r"(idesc), "r"(accum)
      : "memory");
}
// One lane of a converged warp, for the MMA and commit instructions, which one thread issues. Measured against a test on the
// lane number: 1.3 k clocks per 16-channel chunk less in the issuing thread (role counters), the library 13.6 -> 8.7 MB.
__device__ __forceinline__ bool electOne() {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(ok));
  return ok != 0;
}
__device__ __forceinline__ void mmaCommit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smemAddr(bar))
               : "memory");
}
// tcgen05.ld 32x32b: thread i of the warp gets TMEM lane (base lane + i), registers = consecutive columns.
__device__ __forceinline__ void tmemLoad16Async(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmemWaitLoads() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor, K-major, no swizzle: core matrix = 8 rows x 16 bytes stored contiguously (rows at
// 16-byte pitch), `sbo` = byte distance between 8-row groups, `lbo` = byte distance between the two 16-byte K chunks
// of one K8 step. Bits: [0,14) address >> 4, [16,30) lbo >> 4, [32,46) sbo >> 4, [46,48) version = 1, [61,64) layout 0.
__device__ __forceinline__ uint64_t makeDesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return uint64_t((addr >> 4) & 0x3FFFu) | (uint64_t((lbo >> 4) & 0x3FFFu) << 16) |
         (uint64_t((sbo >> 4) & 0x3FFFu) << 32) | (uint64_t(1) << 46);
}
// Instruction descriptor of an M128 x N `n` MMA: D f32 (bits 4-5 = 1), both operands K-major, N >> 3 at bit 17, M >> 4 at
// bit 24, A and B f16 (format 0) or tf32 (bits 7-9 / 10-12 = 2).
__host__ __device__ constexpr uint32_t idescOf(bool f16, int n) {
  return (1u << 4) | (f16 ? 0u : (2u << 7) | (2u << 10)) | (uint32_t(n >> 3) << 17) | (uint32_t(MT >> 4) << 24);
}

// hi half of the tf32 split. Saturating: a value next to the largest float, or infinite, gets the largest finite hi, so that
// lo = v - hi stays finite resp. infinite and the products keep the sum's value; rounded up to infinity, hi would make
// lo = -inf and the sum NaN.
__device__ __forceinline__ float tf32Round(float v) {
  uint32_t r;
  asm("cvt.rna.satfinite.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
  return __uint_as_float(r);
}

// sin(u)^2 for any finite u, absolute error ~1.5e-7: u = n pi/2 + r with |r| <= pi/4 (three-term Cody-Waite),
// sin^2(u) = sin^2(r) for even n and 1 - sin^2(r) for odd n.
// Two elements at a time on the packed f32x2 pipe (fma.rn.f32x2 and friends: one instruction, two lanes of math),
// two independent lanes of the same operation sequence.
__device__ __forceinline__ float2 sinSq2(float2 u) {
  const float2 kMagic = make_float2(12582912.f, 12582912.f);
  const float2 t = __ffma2_rn(u, make_float2(0.6366197723675814f, 0.6366197723675814f), kMagic);
  const float2 n = __fadd2_rn(t, make_float2(-12582912.f, -12582912.f));
  float2 r = __ffma2_rn(n, make_float2(-1.5703125f, -1.5703125f), u);
  r = __ffma2_rn(n, make_float2(-4.837512969970703125e-4f, -4.837512969970703125e-4f), r);
  r = __ffma2_rn(n, make_float2(-7.54978995489188216e-8f, -7.54978995489188216e-8f), r);
  const float2 s2 = __fmul2_rn(r, r);
  float2 p = __ffma2_rn(s2, make_float2(2.7557319e-6f, 2.7557319e-6f), make_float2(-1.9841270e-4f, -1.9841270e-4f));
  p = __ffma2_rn(p, s2, make_float2(8.3333333e-3f, 8.3333333e-3f));
  p = __ffma2_rn(p, s2, make_float2(-1.6666667e-1f, -1.6666667e-1f));
  p = __ffma2_rn(p, s2, make_float2(1.f, 1.f));
  const float2 sn = __fmul2_rn(r, p);
  const float2 q = __fmul2_rn(sn, sn);
  return make_float2((__float_as_int(t.x) & 1) ? 1.f - q.x : q.x, (__float_as_int(t.y) & 1) ? 1.f - q.y : q.y);
}

// Prologue with per-channel constants folded once per launch (sPar rows -mean, a, b, inv):
//   Snake: u = (x - mean) * (alpha scale) + alpha beta; result = (u + sin^2(u)) / alpha  (= v + sin^2(alpha v) / alpha)
//   leaky / none: v = (x - mean) * scale + beta
// Centering first keeps the precision when the variance is tiny next to the mean, as in the reference.
template <int ACT>
__device__ __forceinline__ float2 activate2(float2 x, float2 negm, float2 a, float2 b, float2 inv, float slope) {
  const float2 v = __ffma2_rn(__fadd2_rn(x, negm), a, b);
  if (ACT == 1) return __fmul2_rn(__fadd2_rn(v, sinSq2(v)), inv);
  if (ACT == 2) return make_float2(v.x >= 0.f ? v.x : v.x * slope, v.y >= 0.f ? v.y : v.y * slope);
  return v;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

template <int N>
__device__ __forceinline__ void regInc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void regDec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

// Tensor maps of a launch.
struct TcMaps {
  CUtensorMap x, ext, res, out;
  CUtensorMap w, w1;  // CTA pairs: the weights of a tap group of wG and of wG - 1 taps
};

}  // namespace tc

// CTA pairs (conv_pair.cu): the buffers of a launch (activations, raw input, weight slots, taps per slot) with its shared memory, or
// 0 where they do not fit; the launch.
size_t pairSmem(int ci, int rows, int rawPitch, int k, int* nb, int* nRaw, int* wStages, int* wG);
int convPair(const tc::TcArgs& a, const tc::TcMaps& m, Act act, int grid, size_t smem, cudaStream_t s);

}  // namespace lkc
