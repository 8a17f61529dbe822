// Tensor-core fused conv1d on CTA pairs (tcgen05.mma.cta_group::2): the form of conv_tc.cu's conv for whole pairs of output-channel
// blocks and 16-byte aligned rows. Same operands (f16 halves), same drains, same prologue; see there. What differs:
//
//   D[256 co, W t] += Wtap[256 co, 16 ci] * Ashift[16 ci, W t]: each CTA of a pair has 128 of the output channels and stages half
//   of the tile's columns, of which an MMA reads both halves.
//
// W is 160 columns, or 128 where the chunk statistics have to be of 128 columns: Dhi then fits twice beside Dlo into tensor memory,
// and the hi MMAs of a drain group need not wait for the drain of the one before, nor for the final phase of the tile before. At 128
// columns the sums are added in the same order too, bit for bit; at 160 a residual is added behind another drain, and statistics are
// those of narrow tiles.
// What bounds it: an M128 N256 MMA of the other form reads 96 B/clk of shared memory, an M128 N160 one 115, which leaves the other
// roles (weights, windows, residual, output: about 50 B/clk at K = 11) too little. A pair reads 83 at W = 160, 66 with the weights
// of two of a tap's three MMAs in the collector, and stages half as many window columns for an output channel.
//
// One thread of the pair's first CTA issues the MMAs of both. Hand-offs that it waits for are barriers of that CTA, at which both
// CTAs arrive; those that it signals are committed to both. Every wait is bounded, in both CTAs. They set up and leave together (a
// cluster barrier at either end), and a CTA arrives at the last one only when every signal that is for it has come: neither signals
// into shared memory that is gone. Where a wait has run out, and that cannot be waited for, a fence stands in front of the arrival.
#include <algorithm>
#include <type_traits>

#include "conv_tc.cuh"

namespace lkc {
using namespace tc;

namespace {

constexpr int ACT_ROW = Fmt<true>::ACT_BYTES_PER_ROW;
constexpr int MAX_RAW = 4;     // raw-input staging buffers
constexpr int ACC_COLS = 160;  // tensor memory columns of an accumulator, and widest tile
constexpr int TAP_BYTES = Fmt<true>::W_STAGE_BYTES;

struct PairLayout {
  uint32_t act, raw, w, par, stat, bar, total;
};
__host__ __device__ inline PairLayout pairLayout(int ci, int rows, int rawPitch, int nb, int nRaw, int wStages, int wG) {
  PairLayout s;
  s.act = EPI_WARPS * BOX_BYTES;  // boxes: [0, act)
  s.raw = (s.act + uint32_t(nb) * ACT_ROW * rows + 127u) & ~127u;
  s.w = (s.raw + uint32_t(nRaw) * KC * rawPitch * 4 + 1023u) & ~1023u;  // (a raw buffer is a multiple of 128: rawPitch is of 4)
  s.par = s.w + uint32_t(wStages) * wG * TAP_BYTES;
  s.stat = s.par + uint32_t(4) * ci * 4;
  s.bar = s.stat + 2 * 128 * 16;
  s.total = s.bar + 512;
  return s;
}

// ---------------------------------------------------------------------------------------------- PTX helpers

// Arrival at a barrier of either CTA. What it reports stays in this SM: operands that a proxy fence has handed to the tensor core,
// accumulators that are read. (As a release at cluster scope it waited for this thread's stores: 2.9 k instead of 2.1 k clocks per
// staged chunk.)
__device__ __forceinline__ void mbarArriveAt(uint32_t clusterAddr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(clusterAddr) : "memory");
}
// Tiled load into this CTA's shared memory, counted by a barrier of either CTA of the pair.
__device__ __forceinline__ void tmaLoad2dPair(void* dst, const CUtensorMap* map, int x, int y, uint32_t clusterBar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smemAddr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(clusterBar)
      : "memory");
}
__device__ __forceinline__ void storePeer(uint32_t clusterAddr, int v) {
  asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(clusterAddr), "r"(v) : "memory");
}
__device__ __forceinline__ void fenceCluster() { asm volatile("fence.acq_rel.cluster;" ::: "memory"); }
// What the A collector does with the operand: nothing, keep it, use what it has for the last time.
enum class Coll { None, Fill, Last };
template <Coll C>
__device__ __forceinline__ void mmaPair(uint32_t dTmem, uint32_t aLo, uint32_t aHi, uint32_t bLo, uint32_t bHi, uint32_t idesc,
                                        uint32_t accum) {
#define LKC_MMA_PAIR(suffix)                                           \
  asm volatile(                                                        \
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"                    \
      "setp.ne.b32 p, %6, 0;\n\t"                                      \
      "mov.b64 da, {%1, %2};\n\t"                                      \
      "mov.b64 db, {%3, %4};\n\t"                                      \
      "tcgen05.mma.cta_group::2.kind::f16" suffix " [%0], da, db, %5, p;\n\t}" ::"r"(dTmem), \
      "r"(aLo), "r"(aHi), "r"(bLo), "r"(bHi), "r"(idesc), "r"(accum)   \
      : "memory")
  if constexpr (C == Coll::None) LKC_MMA_PAIR("");
  if constexpr (C == Coll::Fill) LKC_MMA_PAIR(".collector::a::fill");
  if constexpr (C == Coll::Last) LKC_MMA_PAIR(".collector::a::lastuse");
#undef LKC_MMA_PAIR
}
// Arrives at the barrier of this offset in both CTAs when the MMAs issued so far are done.
__device__ __forceinline__ void mmaCommitPair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                   smemAddr(bar)),
               "h"(uint16_t(3))
               : "memory");
}
__device__ __forceinline__ void tmemAllocPair(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(slot)), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmemRelinquishPair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmemDeallocPair(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}

template <int ACT>
__global__ void __launch_bounds__(NTHREADS, 1)
    convPairKernel(const TcArgs a, const __grid_constant__ CUtensorMap mapX,
                   const __grid_constant__ CUtensorMap mapRes, const __grid_constant__ CUtensorMap mapOut,
                   const __grid_constant__ CUtensorMap mapW, const __grid_constant__ CUtensorMap mapW1) {
  const uint32_t W = a.tileCols, kIdesc = (1u << 4) | ((W >> 3) << 17) | (uint32_t(256 >> 4) << 24);  // M 256, N W, f16
  extern __shared__ __align__(1024) unsigned char smemRaw[];
  const int rows = a.rows, rawPitch = a.ext;
  const int NB = a.nb, NRAWB = a.nRaw;
  const PairLayout lay = pairLayout(a.ci, rows, rawPitch, NB, NRAWB, a.wStages, a.wG);
  const int actBufFloats = ACT_ROW / 4 * rows;  // hi + lo
  const int rawBufFloats = KC * rawPitch;
  float* const sAct = reinterpret_cast<float*>(smemRaw + lay.act);   // NB buffers of [2 (hi, lo)][16-byte K chunks][rows]
  float* const sRaw = reinterpret_cast<float*>(smemRaw + lay.raw);   // buffers of [KC][rawPitch] raw input
  unsigned char* const sW = smemRaw + lay.w;                         // slots of wG taps of [2 (hi, lo)][16-byte K chunks][128]
  float* const sPar = reinterpret_cast<float*>(smemRaw + lay.par);   // [4][ci]: folded prologue constants
  float4* const sStat = reinterpret_cast<float4*>(smemRaw + lay.stat);  // per tile parity, epilogue warp of the first half and lane
  uint64_t* const bars = reinterpret_cast<uint64_t*>(smemRaw + lay.bar);
  constexpr int B_EMPTY = MAX_NB, W_FULL = B_EMPTY + MAX_NB, W_EMPTY = W_FULL + MAX_W_STAGES, HI_FULL = W_EMPTY + MAX_W_STAGES,
                HI_EMPTY = HI_FULL + 2, LO_FULL = HI_EMPTY + 2, LO_EMPTY = LO_FULL + 1, RAW_FULL = LO_EMPTY + 1,
                RAW_EMPTY = RAW_FULL + MAX_RAW, RES_BAR = RAW_EMPTY + MAX_RAW, STAT_FULL = RES_BAR + EPI_WARPS,
                NUM_BARS = STAT_FULL + 8;
  static_assert(NUM_BARS * 8 + 8 <= 512, "barriers");
  uint64_t* const bFull = bars;               // (first CTA) both CTAs' windows staged
  uint64_t* const bEmpty = bars + B_EMPTY;
  uint64_t* const wFull = bars + W_FULL;      // (first CTA) both CTAs' weights
  uint64_t* const wEmpty = bars + W_EMPTY;
  uint64_t* const hiFull = bars + HI_FULL;
  uint64_t* const hiEmpty = bars + HI_EMPTY;  // (first CTA)
  uint64_t* const loFull = bars + LO_FULL;
  uint64_t* const loEmpty = bars + LO_EMPTY;  // (first CTA)
  uint64_t* const rawFull = bars + RAW_FULL;
  uint64_t* const rawEmpty = bars + RAW_EMPTY;
  uint64_t* const resBar = bars + RES_BAR;    // one per epilogue warp
  uint64_t* const statFull = bars + STAT_FULL;  // per tile parity and quarter of the channels
  uint32_t* const tmemSlot = reinterpret_cast<uint32_t*>(bars + NUM_BARS);
  volatile int* const abortFlag = reinterpret_cast<int*>(tmemSlot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (smemAddr(smemRaw) & 1023u) {  // the 128-byte swizzle of the boxes assumes it (the same in both CTAs)
    if (threadIdx.x == 0) atomicOr(a.status, (6 << 8) | 1);
    return;
  }
  const uint32_t rank = clusterRank();
  const int pair = int(blockIdx.x) >> 1, pairStep = int(gridDim.x) >> 1;
  const int numTiles = a.numTTiles * a.numCoBlk;  // pair tiles
  // tile t of the pair: columns of pair tile tt, channel block cb; the next one is stepT, stepC further
  const int n0 = a.numCoBlk, stepT = pairStep / n0, stepC = pairStep - stepT * n0, tt0 = pair / n0, cb0 = pair - tt0 * n0;
  auto advance = [&](int& tt, int& cb) {
    tt += stepT, cb += stepC;
    if (cb >= n0) cb -= n0, ++tt;
  };
  const int lo = int(a.lo);
  const int nChunks16 = a.ci / KC;
  const int nGroups = (nChunks16 + a.drainN - 1) / a.drainN;  // Dhi drains per tile
  // tap groups of a chunk: the first tgExtra groups have tgBase + 1 taps, the others tgBase
  const int nTapGroups = (a.k + a.wG - 1) / a.wG, tgBase = a.k / nTapGroups, tgExtra = a.k % nTapGroups;

  if (threadIdx.x < NUM_BARS) {  // a thread per barrier: one copy of the code
    const int i = threadIdx.x;
    const int arrivals = i < B_EMPTY                      ? PRO_WARPS      // bFull: four warps of either CTA
                         : i >= HI_EMPTY && i < LO_FULL   ? 2 * EPI_WARPS  // hiEmpty
                         : i == LO_EMPTY                  ? 2 * EPI_WARPS
                         : i >= RAW_EMPTY && i < RES_BAR  ? PRO_WARPS / 2  // rawEmpty
                                                          : 1;
    mbarInit(bars + i, arrivals);
    fenceBarrierInit();
  }
  if (threadIdx.x == 0) *abortFlag = 0;
  if (warp == MMA_WARP) {  // the MMA warps own the TMEM allocation
    tmemAllocPair(tmemSlot, 512);
    tmemRelinquishPair();
  }
  tcFenceBefore();
  __syncthreads();
  clusterArrive(), clusterWait();  // the peer's barriers are there (their fence is above; its flag is older than any wait that gives up)
  tcFenceAfter();
  const uint32_t tmemHi = *tmemSlot, tmemLo = tmemHi + 2 * ACC_COLS;

  // mbarWait that adds the cycles it spent to acc in the profiling build
  auto waitT = [&](uint64_t* bar, uint32_t parity, long long& acc, uint32_t sleepNs) -> bool {
    if constexpr (!kProf) {
      return mbarWait(bar, parity, abortFlag, sleepNs);
    } else {
      const long long t0 = clock64();
      const bool ok = mbarWait(bar, parity, abortFlag, sleepNs);
      acc += clock64() - t0;
      return ok;
    }
  };
  auto profAddIf = [&](bool mine, int slot, long long v) {
    if (kProf && a.prof && mine) atomicAdd(reinterpret_cast<unsigned long long*>(a.prof + slot), (unsigned long long)v);
  };
  auto profAdd = [&](int slot, long long v) { profAddIf(lane == 0, slot, v); };
  // What this role gave up waiting for, role << 8 | code, or 0. Reported once, behind the roles (a report at each of twenty waits is
  // 9 KB of code).
  int dead = 0;
  // One arrival of this CTA at a barrier of the first.
  auto arriveFirst = [&](uint64_t* bar) {
    if (rank == 0) mbarArrive(bar);
    else mbarArriveAt(peerAddr(smemAddr(bar), 0));
  };

  if (warp < EPI_WARPS) {
    // ------------------------------------------------------------------ accumulate + epilogue (see conv_tc.cu)
    regInc<EPI_REGS>();
    dependenciesWait();
    constexpr int NBAT = 3;  // most 32-column batches of a warp
    const int q = warp & 3, g = warp >> 2;  // TMEM lane quarter (32 channels), half of the tile
    const int nb0 = int((W >> 5) + 1) >> 1, nbat = g ? int(W >> 5) - nb0 : nb0, gcol = g * nb0 * 32;
    unsigned char* const box = smemRaw + warp * BOX_BYTES;  // 32 channels x 32 columns, 128-byte swizzle
    unsigned char* const boxRow = box + lane * 128;         // this lane's channel
    const int swz = lane & 7;
    uint64_t* const myRes = &resBar[warp];
    const uint32_t tmemMine = (uint32_t(q * 32) << 16) + gcol;
    uint32_t groupIt = 0, tileIt = 0, resIt = 0;
    bool resInFlight = false;
    long long wHi = 0, wLo = 0, cPre = 0, cFin = 0;
    const long long tStart = kProf ? clock64() : 0;
    int tt = tt0, cb = cb0;
    for (int t = pair; t < numTiles && !dead; t += pairStep, ++tileIt, advance(tt, cb)) {
      const long long tPre = kProf ? clock64() : 0;
      const int t0 = tt * int(W) + gcol;  // first column of this warp
      const int nValid = lo <= t0 ? 0 : lo - t0 < nbat * 32 ? lo - t0 : nbat * 32;
      const int coBase = (2 * cb + int(rank)) * MT + q * 32, co = coBase + lane;
      const float bias = a.bias ? a.bias[co] : 0.f;
      float S[NBAT * 32];
#pragma unroll
      for (int j = 0; j < NBAT * 32; ++j) S[j] = bias;
      const bool hasRes = a.residual != nullptr;
      auto fetchResidual = [&](int b) {
        if (lane == 0) {
          bulkWaitRead();  // the stores of the previous tile have read the box
          mbarArriveExpectTx(myRes, BOX_BYTES);
          tmaLoad2d(box, &mapRes, t0 + b * BOX, coBase, myRes);
        }
        resInFlight = true;
      };
      auto addResidual = [&](int b) {  // with a constant b
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float4 v = *reinterpret_cast<const float4*>(boxRow + ((c ^ swz) << 4));
          S[b * 32 + 4 * c] += v.x, S[b * 32 + 4 * c + 1] += v.y, S[b * 32 + 4 * c + 2] += v.z, S[b * 32 + 4 * c + 3] += v.w;
        }
      };
      if (kProf) cPre += clock64() - tPre;
      // wait for the group's hi chain, add it to the running sums, hand Dhi back
      auto drainGroup = [&] {
        const uint32_t hb = groupIt & 1;
        if (!waitT(&hiFull[hb], groupIt >> 1 & 1, wHi, SLEEP_EPI_NS)) {
          dead = 1 << 8 | 1;
          return;
        }
        tcFenceAfter();
#pragma unroll
        for (int b = 0; b < 2 * NBAT; ++b) {
          if (b >= 2 * nbat) break;
          uint32_t v[16];
          tmemLoad16Async(tmemHi + hb * ACC_COLS + tmemMine + b * 16, v);
          tmemWaitLoads();
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            const float2 sum = __fadd2_rn(make_float2(S[b * 16 + j], S[b * 16 + j + 1]),
                                          make_float2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])));
            S[b * 16 + j] = sum.x, S[b * 16 + j + 1] = sum.y;
          }
        }
        tcFenceBefore();
        __syncwarp();
        if (lane == 0) arriveFirst(&hiEmpty[hb]);
        ++groupIt;
      };
      // Residual batches ride behind the drains, as in conv_tc.cu. A column's is added behind the same drain as there, so that the bits
      // do not depend on the form: at W = 128 the two halves of the tile are the batches 0, 1 and 2, 3 of a warp there.
      const int nPlan = W == 128 ? 4 : nbat, rb0 = W == 128 ? 2 * g : 0;
      const int nPre = hasRes && nGroups < nPlan ? nPlan - nGroups : 0;
      const int nSteps = nPre + nGroups, preAt = nGroups == 1 ? 0 : 1;  // first step without a drain
      int rb = -rb0;  // next residual batch of this warp
#pragma unroll 1
      for (int c = 0; c < nSteps && !dead; ++c) {
        const bool doRes = hasRes && rb >= 0 && rb < nbat;
        if (doRes) fetchResidual(rb);
        if (c == nSteps - 1) {
          // Last step of the tile (always a drain): Dlo first, so that the next tile's lo MMAs need not wait for the drain.
          if (!waitT(loFull, tileIt & 1, wLo, SLEEP_EPI_NS)) {
            dead = 1 << 8 | 2;
            break;
          }
          tcFenceAfter();
#pragma unroll
          for (int b = 0; b < NBAT; ++b) {  // two 16-column loads in flight per wait
            if (b >= nbat) break;
            uint32_t va[16], vb[16];
            tmemLoad16Async(tmemLo + tmemMine + b * 32, va);
            tmemLoad16Async(tmemLo + tmemMine + b * 32 + 16, vb);
            tmemWaitLoads();
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              S[b * 32 + j] = fmaf(__uint_as_float(va[j]), 1.f / kLoScale, S[b * 32 + j]);
              S[b * 32 + 16 + j] = fmaf(__uint_as_float(vb[j]), 1.f / kLoScale, S[b * 32 + 16 + j]);
            }
          }
          tcFenceBefore();
          __syncwarp();
          if (lane == 0) arriveFirst(loEmpty);
        }
        if (c < preAt || c >= preAt + nPre) drainGroup();
        if (doRes && !dead) {
          if (!mbarWait(myRes, resIt & 1, abortFlag, 32)) {
            dead = 1 << 8 | 3;
            break;
          }
          ++resIt, resInFlight = false;
          switch (rb) {
            case 0: addResidual(0); break;
            case 1: addResidual(1); break;
            default: addResidual(2); break;
          }
          __syncwarp();
        }
        ++rb;
      }
      if (dead) break;
      const long long tFin = kProf ? clock64() : 0;
      if (hasRes && a.outScale != 1.f) {
#pragma unroll
        for (int j = 0; j < NBAT * 32; ++j) S[j] *= a.outScale;
      }
      // Per 32-column batch: the registers to the warp's box, which one lane sends, and the batch's statistics meanwhile.
      float pMean[NBAT], pM2[NBAT];
#pragma unroll
      for (int b = 0; b < NBAT; ++b) {
        const int nb = nValid - b * 32 <= 0 ? 0 : nValid - b * 32 < 32 ? nValid - b * 32 : 32;  // valid columns
        if (nb > 0) {  // warp-uniform
          if (lane == 0) bulkWaitRead();  // the previous store has read the box
          __syncwarp();
#pragma unroll
          for (int c = 0; c < 8; ++c)
            *reinterpret_cast<float4*>(boxRow + ((c ^ swz) << 4)) =
                make_float4(S[b * 32 + 4 * c], S[b * 32 + 4 * c + 1], S[b * 32 + 4 * c + 2], S[b * 32 + 4 * c + 3]);
          fenceProxyAsync();  // generic-proxy stores -> visible to the TMA unit
          __syncwarp();
          if (lane == 0) {
            tmaStore2d(&mapOut, t0 + b * BOX, coBase, box);
            bulkCommit();
          }
        }
        float m = 0.f, q0 = 0.f, q1 = 0.f, q2 = 0.f, q3 = 0.f, s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
        if (nb == 32) {
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            s0 += S[b * 32 + j], s1 += S[b * 32 + j + 1], s2 += S[b * 32 + j + 2], s3 += S[b * 32 + j + 3];
          m = ((s0 + s1) + (s2 + s3)) * (1.f / 32.f);
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const float d0 = S[b * 32 + j] - m, d1 = S[b * 32 + j + 1] - m, d2 = S[b * 32 + j + 2] - m, d3 = S[b * 32 + j + 3] - m;
            q0 = fmaf(d0, d0, q0), q1 = fmaf(d1, d1, q1), q2 = fmaf(d2, d2, q2), q3 = fmaf(d3, d3, q3);
          }
        } else if (nb > 0) {  // ragged end of a row
          auto at = [&](int j) { return *reinterpret_cast<const float*>(boxRow + (((j >> 2) ^ swz) << 4) + ((j & 3) << 2)); };
#pragma unroll 1
          for (int j = 0; j < nb; ++j) s0 += at(j);
          m = s0 / float(nb);
#pragma unroll 1
          for (int j = 0; j < nb; ++j) q0 = fmaf(at(j) - m, at(j) - m, q0);
        }
        pMean[b] = m, pM2[b] = (q0 + q1) + (q2 + q3);
      }
      if (a.stats && W != 128) {  // a pair per 32 columns
        float2* const st = reinterpret_cast<float2*>(a.stats) + int64_t(co) * a.nchunks + (t0 >> 5);
#pragma unroll
        for (int b = 0; b < NBAT; ++b)
          if (b * 32 < nValid) st[b] = make_float2(pMean[b], pM2[b]);
      } else if (a.stats) {
        // The tile is one 128-column chunk: the warp of the first 64 columns leaves its two pairs to the one of the others. (Neither
        // can be two tiles ahead: the MMAs need both.)
        float4* const mail = sStat + (tileIt & 1) * 128 + q * 32 + lane;
        uint64_t* const bar = &statFull[(tileIt & 1) * 4 + q];
        if (g == 0) {
          *mail = make_float4(pMean[0], pM2[0], pMean[1], pM2[1]);
          __syncwarp();
          if (lane == 0) mbarArrive(bar);
        } else if (!mbarWait(bar, tileIt >> 1 & 1, abortFlag, 0)) {
          dead = 1 << 8 | 4;
          break;
        } else {
          const float4 f = *mail;
          const int left = lo - tt * 128;  // > 0
          // exact combine: mean = sum n_b m_b / n, M2 = sum M2_b + sum n_b (m_b - mean)^2
          const float m[4] = {f.x, f.z, pMean[0], pMean[1]}, m2[4] = {f.y, f.w, pM2[0], pM2[1]};
          float n[4], sum = 0.f, sq = 0.f;
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            n[b] = float(left <= b * 32 ? 0 : left - b * 32 < 32 ? left - b * 32 : 32);
            sum = fmaf(n[b], m[b], sum);
          }
          const float mean = left < 128 ? sum / float(left) : sum * (1.f / 128.f);
#pragma unroll
          for (int b = 0; b < 4; ++b) sq += m2[b] + n[b] * (m[b] - mean) * (m[b] - mean);
          float* const st = a.stats + (int64_t(co) * a.nchunks + tt) * 2;
          if ((reinterpret_cast<uintptr_t>(a.stats) & 7) == 0) *reinterpret_cast<float2*>(st) = make_float2(mean, sq);
          else st[0] = mean, st[1] = sq;
        }
      }
      if (kProf) cFin += clock64() - tFin;
    }
    // Copies of this warp still in flight must end before the CTA may exit: a residual box after an abort, and the output boxes
    // on every path.
    if (resInFlight) mbarWaitQuiet(myRes, resIt & 1);
    if (lane == 0) bulkWaitAll();
    if (kProf && warp == 0) profAdd(5, wHi), profAdd(6, wLo), profAdd(7, cPre), profAdd(8, cFin), profAdd(9, clock64() - tStart);
  } else if (warp < EPI_WARPS + PRO_WARPS) {
    // ------------------------------------------------------------------ activation producers (see conv_tc.cu)
    regDec<PRO_REGS>();
    dependenciesWait();
    // Four warps stage a chunk, four channels each, the other four the next one: the two of a scheduler are then at different
    // points, one computing while the other waits, loads or hands over.
    const int pw = warp - EPI_WARPS, cg = pw & 3, grp = pw >> 2;
    for (int c = pw * 32 + lane; c < a.ci; c += PRO_WARPS * 32) {
      const float al = ACT == 1 ? a.alpha[c] : 1.f;
      sPar[c] = a.affine ? -a.affine[c] : 0.f;
      sPar[a.ci + c] = (a.affine ? a.affine[a.ci + c] : 1.f) * al;
      sPar[2 * a.ci + c] = (a.affine ? a.affine[2 * a.ci + c] : 0.f) * al;
      sPar[3 * a.ci + c] = 1.f / al;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(PRO_WARPS * 32) : "memory");  // producer warps only
    int buf = grp, rawBuf = grp, lastBuf = -1;  // NB, NRAWB >= 2
    uint32_t bufPar = 1, rawPar = 0, lastPar = 0;
    long long wB = 0, wCp = 0, cTr = 0;
    const long long tStart = kProf ? clock64() : 0;
    int c = grp, t = pair, tt = tt0, cb = cb0;
    while (c >= nChunks16) c -= nChunks16, t += pairStep, advance(tt, cb);
    const int validLo = int(a.validLo), validHi = int(a.validHi);
    while (t < numTiles && !dead) {
      // rows [okLo, okHi) of the window are inside the valid range, the others are zero padding (after the activation)
      const int x0 = tt * int(W) + int(rank * W / 2) - a.padding - a.delta;
      const int okLo = validLo - x0, okHi = validHi - x0;
      for (; c < nChunks16; c += 2) {
        if (!waitT(&rawFull[rawBuf], rawPar, wCp, SLEEP_PRO_NS)) {
          dead = 2 << 8 | 2;
          break;
        }
        if (!waitT(&bEmpty[buf], bufPar, wB, SLEEP_PRO_NS)) {
          dead = 2 << 8 | 1;
          break;
        }
        const long long tTr = kProf ? clock64() : 0;
        // [cg / 2][rows][8 f16], this thread's 4 channels = half of a 16-byte K chunk
        float* const hiAt = sAct + buf * actBufFloats + (cg >> 1) * rows * 4 + (cg & 1) * 2;
        float* const loAt = hiAt + actBufFloats / 2;
        const float* const raw = sRaw + rawBuf * rawBufFloats;
        const float* par = sPar + c * KC + cg * 4;
        const float4 nm = *reinterpret_cast<const float4*>(par), pa = *reinterpret_cast<const float4*>(par + a.ci),
                     pb = *reinterpret_cast<const float4*>(par + 2 * a.ci), pi = *reinterpret_cast<const float4*>(par + 3 * a.ci);
        float big = 0.f;  // largest |value| this thread staged in the chunk (f16 range check)
        auto stage = [&](auto edge, int r, const float* sp, int pitch) {
          float2 v01 = activate2<ACT>(make_float2(sp[0], sp[pitch]), make_float2(nm.x, nm.y), make_float2(pa.x, pa.y),
                                      make_float2(pb.x, pb.y), make_float2(pi.x, pi.y), a.slope);
          float2 v23 = activate2<ACT>(make_float2(sp[2 * pitch], sp[3 * pitch]), make_float2(nm.z, nm.w), make_float2(pa.z, pa.w),
                                      make_float2(pb.z, pb.w), make_float2(pi.z, pi.w), a.slope);
          if constexpr (decltype(edge)::value) {
            const bool ok = r >= okLo && r < okHi;
            v01.x = ok ? v01.x : 0.f, v01.y = ok ? v01.y : 0.f, v23.x = ok ? v23.x : 0.f, v23.y = ok ? v23.y : 0.f;
          }
          big = max3(max3(big, fabsf(v01.x), fabsf(v01.y)), fabsf(v23.x), fabsf(v23.y));
          const __half2 h01 = __float22half2_rn(v01), h23 = __float22half2_rn(v23);
          const float2 sc = make_float2(kLoScale, kLoScale);
          const float2 f01 = __half22float2(h01), f23 = __half22float2(h23);
          const __half2 l01 = __float22half2_rn(__fmul2_rn(__fadd2_rn(v01, make_float2(-f01.x, -f01.y)), sc));
          const __half2 l23 = __float22half2_rn(__fmul2_rn(__fadd2_rn(v23, make_float2(-f23.x, -f23.y)), sc));
          uint2 hw, lw;
          hw.x = *reinterpret_cast<const uint32_t*>(&h01), hw.y = *reinterpret_cast<const uint32_t*>(&h23);
          lw.x = *reinterpret_cast<const uint32_t*>(&l01), lw.y = *reinterpret_cast<const uint32_t*>(&l23);
          *reinterpret_cast<uint2*>(hiAt + r * 4) = hw;
          *reinterpret_cast<uint2*>(loAt + r * 4) = lw;
        };
        const float* const sp = raw + cg * 4 * rawPitch;
        if (okLo <= 0 && okHi >= rows) {  // all but the tiles at the ends of the valid range
#pragma unroll 1
          for (int r = lane; r < rows; r += 32) stage(std::false_type{}, r, sp + r, rawPitch);
        } else {
#pragma unroll 1
          for (int r = lane; r < rows; r += 32) stage(std::true_type{}, r, sp + r, rawPitch);
        }
        if (big > 65504.f) atomicOr(a.status, kStatusF16Range);
        fenceProxyAsync();  // generic-proxy stores -> visible to the tensor core (async proxy)
        __syncwarp();
        if (lane == 0) {
          arriveFirst(&bFull[buf]);
          mbarArrive(&rawEmpty[rawBuf]);  // the raw buffer may be refilled
        }
        if (kProf) cTr += clock64() - tTr;
        lastBuf = buf, lastPar = bufPar;
        if ((rawBuf += 2) >= NRAWB) rawBuf -= NRAWB, rawPar ^= 1;
        if ((buf += 2) >= NB) buf -= NB, bufPar ^= 1;
      }
      while (c >= nChunks16) c -= nChunks16, t += pairStep, advance(tt, cb);
    }
    // The releases of the last NB chunks' buffers are signals to this CTA: they have to be here before it may leave. A group waits for
    // its last chunk's and for the buffer that it would take next, whose last chunk is NB before that one.
    if (lastBuf >= 0 && !dead && (!mbarWait(&bEmpty[buf], bufPar, abortFlag, SLEEP_PRO_NS) ||
                                  !mbarWait(&bEmpty[lastBuf], lastPar ^ 1, abortFlag, SLEEP_PRO_NS)))
      dead = 2 << 8 | 3;
    if (kProf && pw == 0) profAdd(10, wB), profAdd(11, wCp), profAdd(12, cTr), profAdd(13, clock64() - tStart);
  } else {
    regDec<CTL_REGS>();
    if (warp == W_WARP) {
      // ---------------------------------------------------------------- weight producer, of this CTA's half of the channels
      dependenciesWait();
      uint32_t ws = 0, wPh = 1;
      long long wW = 0;
      const long long tStart = kProf ? clock64() : 0;
      const int slotBytes = a.wG * TAP_BYTES;
      constexpr int tapRows = TAP_BYTES / 1024;  // rows of the maps are 1 KB
      const uint32_t wFull0 = peerAddr(smemAddr(wFull), 0);
      int tt = tt0, cb = cb0;
      for (int t = pair; t < numTiles && !dead; t += pairStep, advance(tt, cb)) {
        int y = (2 * cb + int(rank)) * nChunks16 * a.k * tapRows;
        for (int c = 0; c < nChunks16 && !dead; ++c) {
          for (int gi = 0; gi < nTapGroups; ++gi) {
            const int n = tgBase + (gi < tgExtra ? 1 : 0);
            if (!waitT(&wEmpty[ws], wPh, wW, SLEEP_W_NS)) {
              dead = 3 << 8 | 1;
              break;
            }
            if (lane == 0) {
              if (rank == 0) mbarArriveExpectTx(&wFull[ws], 2 * n * TAP_BYTES);
              tmaLoad2dPair(sW + ws * slotBytes, n == a.wG ? &mapW : &mapW1, 0, y, wFull0 + ws * 8);
            }
            __syncwarp();
            y += n * tapRows;
            if (++ws == uint32_t(a.wStages)) ws = 0, wPh ^= 1;
          }
        }
      }
      // The releases of the last slots are signals to this CTA: they have to be here before it may leave.
      for (int i = 0; i < a.wStages && !dead; ++i) {
        if (!mbarWait(&wEmpty[ws], wPh, abortFlag, SLEEP_W_NS)) dead = 3 << 8 | 2;
        if (++ws == uint32_t(a.wStages)) ws = 0, wPh ^= 1;
      }
      if (kProf) profAdd(14, wW), profAdd(15, clock64() - tStart);
      // After an abort copies may be in flight whose barrier is the other CTA's: give them far longer than they take.
      if (dead || *abortFlag)
        for (const uint64_t tEnd = globalTimerNs() + 1000 * 1000; globalTimerNs() < tEnd;) __nanosleep(1000);
      __syncwarp();
      if (rank != 0) dependentsLaunch();  // the first CTA's signal comes from its MMA warp
    } else if (warp == RAW_WARP) {
      // ---------------------------------------------------------------- raw-window loader (see conv_tc.cu)
      if (lane == 0) {
        dependenciesWait();
        uint32_t rb = 0, ph = 1, issued = 0;
        long long wR = 0;
        const uint32_t bytes = uint32_t(rawBufFloats) * 4;
        int tt = tt0, cb = cb0;
        for (int t = pair; t < numTiles && !dead; t += pairStep, advance(tt, cb)) {
          const int x0 = tt * int(W) + int(rank * W / 2) - a.padding - a.delta;
          for (int c = 0; c < nChunks16; ++c, ++issued) {
            if (!waitT(&rawEmpty[rb], ph, wR, SLEEP_W_NS)) {
              dead = 5 << 8 | 1;
              break;
            }
            float* dst = sRaw + rb * rawBufFloats;
            mbarArriveExpectTx(&rawFull[rb], bytes);
            tmaLoad2d(dst, &mapX, x0, c * KC, &rawFull[rb]);
            if (++rb == uint32_t(NRAWB)) rb = 0, ph ^= 1;
          }
        }
        if (dead || *abortFlag) {
          for (uint32_t i = issued > uint32_t(NRAWB) ? issued - NRAWB : 0; i < issued; ++i)
            mbarWaitQuiet(&rawFull[i % NRAWB], (i / NRAWB) & 1);
        }
      }
    } else if (warp == MMA_WARP && rank == 0) {
      // ---------------------------------------------------------------- MMA issuer of the pair
      // As in conv_tc.cu: one wait per weight slot, its MMAs back to back, one release. Of a tap's three MMAs the two with the hi
      // weights are neighbours, the second of which finds them in the collector.
      const uint64_t dA0 = makeDesc(smemAddr(sW), MT * 16, 128);
      const uint64_t dB0 = makeDesc(smemAddr(sAct), rows * 16, 128) + uint32_t(a.delta);
      constexpr uint32_t kTapU = TAP_BYTES >> 4, kLoAU = kTapU / 2;
      const uint32_t bufU = uint32_t(actBufFloats * 4) >> 4, loBU = bufU >> 1, slotU = uint32_t(a.wG) * kTapU;
      const int dil = a.dilation, wStages = a.wStages, drainN = a.drainN;
      int slot = 0, buf = 0, g = 0;
      uint32_t slotPh = 0, bufPh = 0, hb = 0, hiPar = 1, loPar = 1;
      bool ready = false;  // the next round's weight slot is already known to be full
      long long wBf = 0, wHe = 0, wWf = 0, wLe = 0;
      const long long tStart = kProf ? clock64() : 0;
      const bool leader = electOne();
      for (int tile = pair; leader && tile < numTiles && !dead; tile += pairStep) {
        for (int c = 0; c < nChunks16 && !dead; ++c) {
          if (!waitT(&bFull[buf], bufPh, wBf, SLEEP_MMA_NS)) {
            dead = 4 << 8 | 2;
            break;
          }
          const bool lastChunk = c == nChunks16 - 1, groupEnd = g == drainN - 1 || lastChunk;
          const uint64_t dBc = dB0 + uint32_t(buf) * bufU;
          const uint32_t dHi = tmemHi + hb * ACC_COLS;
          int kk = 0;
          for (int gi = 0; gi < nTapGroups; ++gi) {
            const int gN = tgBase + (gi < tgExtra ? 1 : 0);
            if (!ready && !waitT(&wFull[slot], slotPh, wWf, SLEEP_MMA_NS)) {
              dead = 4 << 8 | 3;
              break;
            }
            const uint64_t dA = dA0 + uint32_t(slot) * slotU, dB = dBc + uint32_t(kk * dil);
            const uint32_t aHi = uint32_t(dA >> 32), bHi = uint32_t(dB >> 32);
            uint32_t aj = uint32_t(dA), bj = uint32_t(dB);
            uint32_t accHi = (kk | g) == 0 ? 0u : 1u, accLo = (kk | c) == 0 ? 0u : 1u;
            int nslot = slot + 1;
            uint32_t nph = slotPh;
            if (nslot == wStages) nslot = 0, nph ^= 1;
            if (accLo == 0u && !waitT(loEmpty, loPar, wLe, SLEEP_MMA_NS)) {
              dead = 4 << 8 | 4;
              break;
            }
            if (accHi == 0u && !waitT(&hiEmpty[hb], hiPar, wHe, SLEEP_MMA_NS)) {
              dead = 4 << 8 | 1;
              break;
            }
            tcFenceAfter();
#pragma unroll 1
            for (int j = 0; j < gN; ++j, aj += kTapU, bj += uint32_t(dil), accHi = accLo = 1u) {
              mmaPair<Coll::None>(tmemLo, aj + kLoAU, aHi, bj, bHi, kIdesc, accLo);
              mmaPair<Coll::Fill>(dHi, aj, aHi, bj, bHi, kIdesc, accHi);
              mmaPair<Coll::Last>(tmemLo, aj, aHi, bj + loBU, bHi, kIdesc, 1u);
            }
            // first poll of the next slot's barrier, with the whole round queued behind it
            ready = mbarTestWait(&wFull[nslot], nph);
            mmaCommitPair(&wEmpty[slot]);  // weight slots free once the MMAs have read them
            kk += gN;
            slot = nslot, slotPh = nph;
          }
          if (dead) break;
          if (lastChunk) mmaCommitPair(loFull);
          if (groupEnd) mmaCommitPair(&hiFull[hb]);
          mmaCommitPair(&bEmpty[buf]);  // activation buffers free once the MMAs have read them
          if (++buf == NB) buf = 0, bufPh ^= 1;
          ++g;
          if (groupEnd) g = 0, hiPar ^= hb, hb ^= 1;
        }
        loPar ^= 1;
      }
      __syncwarp();
      dependentsLaunch();
      // The epilogues' last releases of the accumulators are signals to this CTA, the second CTA's too: no MMA waits for them.
      if (leader && !dead && !mbarWait(loEmpty, loPar, abortFlag, SLEEP_EPI_NS)) dead = 4 << 8 | 5;
      for (int i = 0; i < 2 && leader && !dead; ++i, hiPar ^= hb, hb ^= 1)
        if (!mbarWait(&hiEmpty[hb], hiPar, abortFlag, SLEEP_EPI_NS)) dead = 4 << 8 | 6;
      if (kProf)
        profAddIf(leader, 0, wBf), profAddIf(leader, 1, wHe), profAddIf(leader, 2, wWf), profAddIf(leader, 3, wLe),
            profAddIf(leader, 4, clock64() - tStart);
    }
  }

  if (dead && (lane == 0 || warp == MMA_WARP)) {  // first timeout wins the low 16 bits; the flag bits above them are kept
    int old = *a.status;
    while ((old & kStatusWaitMask) == 0) {
      const int seen = atomicCAS(a.status, old, old | dead);
      if (seen == old) break;
      old = seen;
    }
    *abortFlag = 1;  // both CTAs of the pair stop
    storePeer(peerAddr(smemAddr(const_cast<int*>(abortFlag)), rank ^ 1), 1);
    fenceCluster();  // that store and the arrivals that nobody waits for now (releases on every path cost 0.3 to 0.6 us per launch)
  }
  tcFenceBefore();
  clusterArrive(), clusterWait();  // nothing is under way to either CTA's shared memory or TMEM any more
  if (warp == MMA_WARP) {
    tcFenceAfter();
    tmemDeallocPair(tmemHi, 512);
  }
}

template <int ACT>
int launchPair(const TcArgs& a, const TcMaps& m, int grid, size_t smem, cudaStream_t s) {
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  const auto kernel = convPairKernel<ACT>;
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    if (e != cudaSuccess) return failCuda("conv (CTA pairs): cudaFuncSetAttribute", e);
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cfg.gridDim = dim3(unsigned(grid)), cfg.blockDim = dim3(NTHREADS), cfg.dynamicSmemBytes = smem, cfg.stream = s, cfg.attrs = attr;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
  cfg.numAttrs = 1;
  if (a.early) {
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
  }
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, a, m.x, m.res, m.out, m.w, m.w1);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return failCuda("conv (CTA pairs)", e);
  }
  return launched("conv (CTA pairs)");
}

}  // namespace

// Fewer rounds (weight slots of more taps) first, as each costs the issuing thread about 270 clocks: two slots where one holds a
// chunk's taps, else three, as a slot of 48 KB takes longer to refill than the other one's MMAs. Four of either kind of
// activation buffer where they fit beside them, else three and two.
size_t pairSmem(int ci, int rows, int rawPitch, int k, int* nb, int* nRaw, int* wStages, int* wG) {
  for (int g = std::min(8, k); g >= 1; --g) {
    const int groups = (k + g - 1) / g, gmax = (k + groups - 1) / groups;
    for (int n = 4; n >= 3; --n) {
      const int raws = n == 4 ? 4 : 2;
      const size_t base = pairLayout(ci, rows, rawPitch, n, raws, 0, 0).total;
      if (base > size_t(kMaxSmem)) continue;
      const int ws = int(std::min<size_t>(MAX_W_STAGES, (size_t(kMaxSmem) - base) / (size_t(gmax) * TAP_BYTES)));
      if (ws < (groups == 1 ? 2 : 3)) continue;
      *nb = n, *nRaw = raws, *wStages = ws, *wG = gmax;
      return pairLayout(ci, rows, rawPitch, n, raws, ws, gmax).total;
    }
  }
  return 0;
}

int convPair(const TcArgs& a, const TcMaps& m, Act act, int grid, size_t smem, cudaStream_t s) {
  switch (act) {
    case Act::None: return launchPair<0>(a, m, grid, smem, s);
    case Act::Snake: return launchPair<1>(a, m, grid, smem, s);
    case Act::Leaky: return launchPair<2>(a, m, grid, smem, s);
  }
  return fail("conv (CTA pairs): bad activation");
}

}  // namespace lkc
