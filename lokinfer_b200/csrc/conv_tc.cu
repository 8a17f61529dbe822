// Tensor-core fused conv1d for sm_100a: implicit GEMM on tcgen05 with TMEM accumulators and split operands.
//
//   out[co, t] = sum_{ci, kk} W[co, ci, kk] * A[ci, t + kk d - pad],  A = act((x - mean) * scale + beta), zero outside
//   [0, L); epilogue + bias [+ residual] [* oscale] and the per-(channel, 128-column chunk) (mean, M2).
//
// GEMM view: D[128 co, 256 t] += Wtap[128 co, 16 ci] * Ashift[16 ci, 256 t] for every 16-channel chunk and tap. Some launches
// take narrower tiles (tileColsFor: 160, 192 or 224 columns; 128 or 64 in the split form).
// f32 accuracy comes from splitting both operands, v = hi + lo with an 11-bit hi and an 11-bit lo:
// out = sum Whi Ahi + (sum Wlo Ahi + Whi Alo); the lo*lo term, 2^-22 relative, is dropped. Two operand formats
// (see Fmt below): f16 halves (default; 3 kind::f16 K16 MMAs per tap and 16 channels) or tf32 halves (6 kind::tf32
// K8 MMAs).
//
// The tensor core adds into its f32 accumulator with truncation, so a long accumulation chain drifts towards zero by
// about 1.5e-8 of the result per MMA (measured: the error grows linearly with the chain length). Two accumulators
// keep that out of the result: Dhi (TMEM columns 0-255) takes only the hi*hi products of a short run of MMAs (a drain
// group: as many whole 16-channel chunks as fit in 24 chained MMAs, at least one chunk), is then drained by the
// epilogue warps into f32 registers (round-to-nearest adds on the CUDA cores) and restarted; Dlo (columns 256-511)
// takes every lo product of the tile, where the same drift is scaled by 2^-11.
//
// Global memory traffic goes through the TMA unit whenever the rows of a tensor are 16-byte aligned (base pointer and
// row pitch; the entry points take a row pitch for every [C, L] activation tensor, so a caller that owns its
// intermediates can pad the rows): the raw input window of a 16-channel chunk is one pair of tiled bulk loads, the
// residual arrives as 32 x 32 boxes in the 128-byte swizzle, and the output leaves as 32 x 32 boxes of the same
// swizzle (bulk tensor stores). Tensors whose rows are not aligned (the reference's contiguous [C, L] with an odd L)
// take 4-byte cp.async loads and transposed 4-byte stores instead; the arithmetic is the same on both routes.
// No copy uses cluster multicast, and every tensor map covers memory of this GPU only.
//
// One persistent CTA per SM, 20 warps in 5 warpgroups, warp-specialised (registers rebalanced with setmaxnreg):
//   warps 0-7   accumulate + epilogue: 128 running sums per thread, started from the bias; the residual is added one
//               32-column batch at a time (fetched into the warp's tile behind a Dhi drain); per drain group += Dhi
//               (tcgen05.ld); per tile += Dlo (folded in before the tile's last drain: Dlo is complete one run of hi
//               MMAs before Dhi is), oscale, chunk statistics and the store
//   warps 8-15  activation producers, two per warp scheduler: affine -> Snake / leaky -> hi / lo split of the current chunk's raw window into
//               shared memory in the K-major no-swizzle UMMA layout [16-byte K chunk][time row][4 f32 or 8 f16
//               channels]: a tap shift of kk*d time steps is a +16*kk*d byte offset of the descriptor start address,
//               so one staged window serves all taps (on the unaligned route they also issue the cp.async of the next
//               chunk's raw window)
//   warp 16     weight producer: one cp.async.bulk per tap group (up to 6 taps; hi | lo of [128 co x 16 ci] per tap,
//               pre-packed in the UMMA layout, L2-resident) into a ring of shared-memory slots
//   warp 17     MMA issuer (one elected lane): per tap group one wait, the group's MMAs back to back, one release
//   warp 18     raw-window loader of the aligned route (one lane): two tiled TMA loads per chunk, one chunk ahead
//   warp 19     idle (completes the fifth warpgroup)
// Launches with few tiles take a second form of the same kernel (template parameter SPLIT): a cluster of CTAs per
// 128- or 64-column tile, each contracting a part of the input channels, reduced over distributed shared memory. Whole pairs of
// output-channel blocks take CTA pairs (conv_pair.cu).
// All hand-offs are mbarriers. Every wait is bounded: on a timeout the kernel records a status word, drains its
// copies in flight and returns (TMEM is freed on every path).
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "conv_tc.cuh"

namespace lkc {
using namespace tc;

namespace {

// Shared-memory carve-up of one CTA (byte offsets from the 1024-byte aligned base). The epilogue tiles come first:
// the 128-byte swizzle of the aligned route needs each warp's 4 KB box on a 1024-byte boundary.
struct SmemLayout {
  uint32_t act, raw, w, par, bar, total;
};
// split: columns of a split tile, or 0.
__host__ __device__ inline SmemLayout smemLayout(int split, int ci, int rows, int ext, int nb, int wStages, int wG,
                                                 int actRowBytes, int wStageBytes) {
  SmemLayout s;
  s.act = split ? 0 : EPI_WARPS * STAGE_FLOATS * 4;  // tiles: [0, act)
  s.raw = (s.act + uint32_t(nb) * actRowBytes * rows + 127u) & ~127u;
  s.w = s.raw + uint32_t(NRAW) * KC * ((split ? split : NT) + ext) * 4;  // a multiple of 128
  s.par = s.w + uint32_t(wStages) * wG * wStageBytes;
  if (split && s.par < uint32_t(partBytes(split) + recvBytes(split))) s.par = partBytes(split) + recvBytes(split);
  s.bar = s.par + uint32_t(4) * ci * 4;
  s.total = s.bar + 512;
  return s;
}

__device__ int gTcStatus = 0;       // 0 = ok; low 16 bits (role << 8 | code) of the first bounded wait that gave up; flag bits above
__device__ long long gTcProf[16];   // wait / phase cycle sums of one representative warp per role (profiling build)

// Second half of a split tile, one epilogue warp. The CTAs of the cluster own a run of its output channels each. Every CTA
// copies the rows of its partial tile to their owners (send); the owner adds the partials in rank order out of its own shared
// memory (finish). One bulk copy per pair of CTAs: loads or stores from one SM to another move about 11 bytes per clock
// (5-7 k clocks for the 56 KB of a CTA).
// conv: a unit is one output channel of the tile, four columns per lane (a warp has two at a time where the tile has 64); the
// rank's 128 / split channels go round robin over the epilogue warps, UB at a time so that their loads overlap. What does not
// depend on the contraction (bias, residual) is loaded by prefetch(), for the first UB units before the accumulation.
// ConvTranspose: a unit is one output channel x 32 input-rate columns, whose 32 * TS output samples are one run.
template <int TS, int COLS>
struct SplitTail {
  static_assert(TS == 0 || COLS == NTS, "ConvTranspose: 128 columns");
  static constexpr int PART_PITCH = partPitch(COLS);
  static constexpr int LPC = COLS / 4;                // lanes per channel
  static constexpr int STEP = EPI_WARPS * 32 / LPC;  // channels that the epilogue warps have at a time
  static constexpr int UB = 4;
  float4 res[UB];
  float bias[UB];
  int row0, units, tt, cb;
  int slot;  // rows that a CTA keeps per sender, enough for the largest share

  // Rows [first, last) of the tile that CTA r owns. ConvTranspose: from its first channel's to its last one's, with the zero
  // rows between two groups of 32.
  static __device__ __forceinline__ void share(int split, int r, int& first, int& last) {
    if constexpr (TS == 0) {
      first = MT * r / split, last = MT * (r + 1) / split;
    } else {
      constexpr int CQ = 32 / TS, CH = 4 * CQ;
      const int c0 = CH * r / split, c1 = CH * (r + 1) / split - 1;
      first = (c0 / CQ) * 32 + (c0 % CQ) * TS, last = (c1 / CQ) * 32 + (c1 % CQ) * TS + TS;
    }
  }

  __device__ __forceinline__ SplitTail(const TcArgs& a, int tile, int rank) {
    tt = tile / a.numCoBlk, cb = tile - tt * a.numCoBlk;
    if constexpr (TS == 0) {
      row0 = MT * rank / a.split, units = MT * (rank + 1) / a.split - row0;
      slot = (MT + a.split - 1) / a.split;
    } else {
      constexpr int CH = 4 * (32 / TS);
      row0 = CH * rank / a.split, units = (NTS / 32) * (CH * (rank + 1) / a.split - row0);  // row0: first channel
      constexpr int CQ = 32 / TS;
      const int n = (CH + a.split - 1) / a.split;  // channels: n * TS rows and the gaps between at most this many groups
      slot = n * TS + (n + CQ - 2) / CQ * (32 - CQ * TS);
    }
  }

  // u0: the first channel (of the rank's) of this lane
  __device__ __forceinline__ void prefetch(const TcArgs& a, int u0, int lane) {
    if constexpr (TS == 0) {
      const bool vecRes = a.residual && ((reinterpret_cast<uintptr_t>(a.residual) | uintptr_t(a.resPitch * 4)) & 15) == 0;
      const int64_t col = int64_t(tt) * COLS + lane % LPC * 4;
#pragma unroll
      for (int e = 0; e < UB; ++e) {
        const int u = u0 + e * STEP, co = cb * MT + row0 + u;
        res[e] = make_float4(0.f, 0.f, 0.f, 0.f), bias[e] = 0.f;
        if (u < units && co < a.co) {
          if (a.bias) bias[e] = a.bias[co];
          if (a.residual && col < a.lo) {
            const float* rp = a.residual + int64_t(co) * a.resPitch + col;
            if (vecRes && col + 4 <= a.lo) {
              res[e] = *reinterpret_cast<const float4*>(rp);
            } else {
              res[e].x = rp[0];
              if (col + 1 < a.lo) res[e].y = rp[1];
              if (col + 2 < a.lo) res[e].z = rp[2];
              if (col + 3 < a.lo) res[e].w = rp[3];
            }
          }
        }
      }
    }
  }

  // What CTA `to` owns of this CTA's partial tile. `recv` = where every CTA of the cluster receives, counted by `bar`.
  __device__ __forceinline__ void send(const TcArgs& a, const float* tile, const float* recv, uint64_t* bar, int rank, int to) const {
    int first, last;
    share(a.split, to, first, last);
    bulkCopyPeer(peerAddr(smemAddr(recv + rank * slot * PART_PITCH), to), tile + first * PART_PITCH,
                 uint32_t((last - first) * PART_PITCH * 4), peerAddr(smemAddr(bar), to));
  }
  // Bytes that CTA `rank` receives.
  static __device__ __forceinline__ uint32_t expected(const TcArgs& a, int rank) {
    int first, last;
    share(a.split, rank, first, last);
    return uint32_t(a.split * (last - first) * PART_PITCH * 4);
  }

  static __device__ __forceinline__ int firstUnit(int warp, int lane) { return warp * (32 / LPC) + lane / LPC; }

  // N channels of this lane, u0, u0 + STEP, .., side by side through the reductions, whose latency is what the phase lasts. As many
  // as there are, in twos: an absent channel takes as long as one. us per launch one after the other / UB always / as it is:
  // [128, 1441] K = 3, eight CTAs with two channels a warp 11.1 / 11.3 / 10.7; [48, 1210] K = 11, three CTAs, 48 of 128 channels
  // 11.8 / 12.1 / 11.0; [256, 3200] K = 3, two CTAs with eight a warp 19.6 / 18.6 / 18.5.
  template <int N>
  __device__ __forceinline__ void finishChannels(const TcArgs& a, const float* parts, int u0, int lane) {
    const bool vecOut = ((reinterpret_cast<uintptr_t>(a.out) | uintptr_t(a.outPitch * 4)) & 15) == 0;
    const int sub = lane % LPC;
    const int64_t tChunk = int64_t(tt) * COLS, col = tChunk + sub * 4;
    // valid columns of the tile, and from this lane's first on
    const int nValid = a.lo - tChunk < COLS ? int(a.lo - tChunk) : COLS, mine = nValid - sub * 4;
    float acc[N][4];
    bool ok[N];  // this lane has columns of channel e
#pragma unroll
    for (int e = 0; e < N; ++e) {
      ok[e] = u0 + e * STEP < units && cb * MT + row0 + u0 + e * STEP < a.co && mine > 0;
      acc[e][0] = acc[e][1] = acc[e][2] = acc[e][3] = 0.f;
    }
    const float* at = parts + u0 * PART_PITCH + sub * 4;
#pragma unroll 2
    for (int r = 0; r < a.split; ++r, at += slot * PART_PITCH) {
#pragma unroll
      for (int e = 0; e < N; ++e)
        if (ok[e]) {
          const float4 v = *reinterpret_cast<const float4*>(at + e * STEP * PART_PITCH);
          acc[e][0] += v.x, acc[e][1] += v.y, acc[e][2] += v.z, acc[e][3] += v.w;
        }
    }
    __syncwarp();
    float mean[N], m2[N];
#pragma unroll
    for (int e = 0; e < N; ++e) {
      const float rs[4] = {res[e].x, res[e].y, res[e].z, res[e].w};
      mean[e] = 0.f, m2[e] = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[e][j] += bias[e];
        if (a.residual) acc[e][j] = (acc[e][j] + rs[j]) * a.outScale;
        if (j < mine) mean[e] += acc[e][j];
      }
      float* op = a.out + int64_t(cb * MT + row0 + u0 + e * STEP) * a.outPitch + col;
      if (ok[e]) {
        if (vecOut && mine >= 4) {
          *reinterpret_cast<float4*>(op) = make_float4(acc[e][0], acc[e][1], acc[e][2], acc[e][3]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (j < mine) op[j] = acc[e][j];
        }
      }
    }
    if (!a.stats) return;
#pragma unroll
    for (int o = LPC / 2; o > 0; o >>= 1)
#pragma unroll
      for (int e = 0; e < N; ++e) mean[e] += __shfl_xor_sync(0xffffffffu, mean[e], o);
#pragma unroll
    for (int e = 0; e < N; ++e) {
      mean[e] /= float(nValid);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < mine) m2[e] = fmaf(acc[e][j] - mean[e], acc[e][j] - mean[e], m2[e]);
    }
#pragma unroll
    for (int o = LPC / 2; o > 0; o >>= 1)
#pragma unroll
      for (int e = 0; e < N; ++e) m2[e] += __shfl_xor_sync(0xffffffffu, m2[e], o);
#pragma unroll
    for (int e = 0; e < N; ++e)
      if (sub == 0 && ok[e]) {
        float* st = a.stats + (int64_t(cb * MT + row0 + u0 + e * STEP) * a.nchunks + tt) * 2;
        st[0] = mean[e], st[1] = m2[e];
      }
  }

  __device__ __forceinline__ void finish(const TcArgs& a, const float* parts, int warp, int lane) {
    if constexpr (TS == 0) {
      const int have = a.co - cb * MT - row0 < units ? a.co - cb * MT - row0 : units;  // channels that exist
#pragma unroll 1
      for (int base = firstUnit(warp, 0); base < have; base += UB * STEP) {  // warp-uniform
        const int u0 = base + lane / LPC;
        if (base != firstUnit(warp, 0)) prefetch(a, u0, lane);
        if (base + UB / 2 * STEP >= have) finishChannels<UB / 2>(a, parts, u0, lane);
        else finishChannels<UB>(a, parts, u0, lane);
      }
    } else {
      constexpr int CQ = 32 / TS, CH = 4 * CQ, SEGS = NTS / 32;
      const int64_t uEnd = a.lo * TS;
      const int firstRow = (row0 / CQ) * 32 + (row0 % CQ) * TS;
#pragma unroll 1
      for (int u = warp; u < units; u += EPI_WARPS) {
        const int ch = row0 + u / SEGS, seg = u % SEGS, co = cb * CH + ch;
        const int64_t o0 = (int64_t(tt) * NTS + seg * 32) * TS + lane;
        if (co >= a.co || o0 - lane >= uEnd) continue;
        float* const orow = a.out + int64_t(co) * a.outPitch;
        const float* const rrow = a.residual ? a.residual + int64_t(co) * a.resPitch : nullptr;
        const float b = a.bias ? a.bias[co] : 0.f;
        float acc[TS], rs[TS];
        const float* off[TS];
#pragma unroll
        for (int f = 0; f < TS; ++f) {
          const int idx = f * 32 + lane;
          off[f] = parts + ((ch / CQ) * 32 + (ch % CQ) * TS - firstRow + idx % TS) * PART_PITCH + seg * 32 + idx / TS;
          acc[f] = b;
          rs[f] = rrow && o0 + f * 32 < uEnd ? rrow[a.padLeft + o0 + f * 32] : 0.f;
        }
#pragma unroll 2
        for (int r = 0; r < a.split; ++r)
#pragma unroll
          for (int f = 0; f < TS; ++f) acc[f] += off[f][r * slot * PART_PITCH];
#pragma unroll
        for (int f = 0; f < TS; ++f) {
          const int64_t o = o0 + f * 32;
          if (o < uEnd) orow[a.padLeft + o] = acc[f] + rs[f];
          // left reflect pad: out[co, 0] = unpadded[co, 1] + residual[co, 0]
          if (a.padLeft && o == 1 && o < uEnd) orow[0] = acc[f] + (rrow ? rrow[0] : 0.f);
        }
      }
    }
  }
};

// PARTIAL: Co is not a multiple of 128 (the last output-channel block has rows that do not exist).
// TS: 0 = conv1d; 6 / 10 = polyphase ConvTranspose1d of that stride (see the comment above convtTcPackKernel).
// TMAO: residual and output boxes travel by TMA (rows 16-byte aligned; conv1d with Co % 128 == 0 only).
// SPLIT (columns of the tile, or 0): a cluster of a.split CTAs shares one tile of 128 or 64 columns. Each CTA contracts its own
// run of input-channel chunks. When the MMAs of all of them are done (a cluster barrier under the last drain) it sends the rows
// of its partial tile to the CTAs that own them, over the operand buffers there, which nothing reads any more; when it has all
// of its own it finishes them: the partials are added in rank order, then bias, residual, scale, statistics and coalesced
// stores. For launches with fewer tiles than SMs, where one tile's serial chain of chunks is the launch's time (see splitFor).
// NARROW: tiles of a.tileCols < NT columns. A form of its own: the width as a run-time value cost 256-column tiles 5 % (K = 7).
template <int ACT, bool PARTIAL, int TS, bool F16, bool TMAO, int SPLIT, bool NARROW>
__global__ void __launch_bounds__(NTHREADS, 1)
    convTcKernel(const TcArgs a, const __grid_constant__ CUtensorMap mapX, const __grid_constant__ CUtensorMap mapExt,
                 const __grid_constant__ CUtensorMap mapRes, const __grid_constant__ CUtensorMap mapOut) {
  constexpr int W_STAGE_BYTES = Fmt<F16>::W_STAGE_BYTES, W_STAGE_FLOATS = Fmt<F16>::W_STAGE_FLOATS;
  constexpr int NTK = SPLIT ? SPLIT : NT;  // time columns of this kernel's tiles
  constexpr int PART_PITCH = partPitch(NTK);
  constexpr int EC = NTK / 2;            // columns of one epilogue warp
  // Dhi buffers: a 128-column tile leaves room for two, so that the hi MMAs of a drain group need not wait for the drain
  // of the one before (the lo MMAs that cover it are shorter here)
  constexpr int HB = SPLIT ? 2 : 1;
  const uint32_t kIdesc = NARROW ? idescOf(F16, 0) | (uint32_t(a.tileCols >> 3) << 17) : idescOf(F16, NTK);
  const int NB = a.nb;
  extern __shared__ __align__(1024) unsigned char smemRaw[];
  const int rows = a.rows, ext = a.ext;
  const SmemLayout lay = smemLayout(SPLIT, a.ci, rows, ext, NB, a.wStages, a.wG, Fmt<F16>::ACT_BYTES_PER_ROW, W_STAGE_BYTES);
  const int actBufFloats = Fmt<F16>::ACT_BYTES_PER_ROW / 4 * rows;  // hi + lo
  const int rawBufFloats = KC * (NTK + ext);
  float* const sStage = reinterpret_cast<float*>(smemRaw);           // EPI_WARPS tiles
  float* const sAct = reinterpret_cast<float*>(smemRaw + lay.act);   // NB buffers of [2 (hi, lo)][16-byte K chunks][rows]
  float* const sRaw = reinterpret_cast<float*>(smemRaw + lay.raw);   // NRAW buffers of [KC][NTK], [KC][ext] raw input
  float* const sW = reinterpret_cast<float*>(smemRaw + lay.w);       // wStages slots of wG taps of [2 (hi, lo)][16-byte K chunks][MT]
  float* const sPar = reinterpret_cast<float*>(smemRaw + lay.par);   // [4][ci]: folded prologue constants
  uint64_t* const bFull = reinterpret_cast<uint64_t*>(smemRaw + lay.bar);
  uint64_t* const bEmpty = bFull + MAX_NB;
  uint64_t* const wFull = bEmpty + MAX_NB;
  uint64_t* const wEmpty = wFull + MAX_W_STAGES;
  uint64_t* const hiFull = wEmpty + MAX_W_STAGES;
  uint64_t* const hiEmpty = hiFull + 2;
  uint64_t* const loFull = hiEmpty + 2;
  uint64_t* const loEmpty = loFull + 1;
  uint64_t* const rawFull = loEmpty + 1;
  uint64_t* const rawEmpty = rawFull + NRAW;
  uint64_t* const resBar = rawEmpty + NRAW;  // one per epilogue warp
  uint64_t* const recvBar = resBar + EPI_WARPS;  // split form: the rows from the CTAs of the cluster
  uint64_t* const tileBar = recvBar + 1;     // and this CTA's partial tile, complete
  uint32_t* const tmemSlot = reinterpret_cast<uint32_t*>(tileBar + 1);
  volatile int* const abortFlag = reinterpret_cast<int*>(tmemSlot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (TMAO && (smemAddr(smemRaw) & 1023u)) {
    // the 128-byte swizzle of the boxes assumes a 1024-byte aligned base; report instead of computing garbage
    if (threadIdx.x == 0) atomicOr(a.status, (6 << 8) | 1);
    return;
  }
  static_assert(!(SPLIT && NARROW), "a split tile is one statistics chunk");
  const int W = NARROW ? a.tileCols : NTK;
  const int numTiles = a.numTTiles * a.numCoBlk;
  // tiles of this CTA: tile0, tile0 + tileStep, ...; its chunks of a tile: cBegin .. cBegin + nChunks16
  const int rank = SPLIT ? int(clusterRank()) : 0;
  const int tile0 = SPLIT ? int(blockIdx.x) / a.split : int(blockIdx.x), tileStep = SPLIT ? numTiles : int(gridDim.x);
  const int nChunksAll = a.ci / KC;
  const int cBegin = SPLIT ? nChunksAll * rank / a.split : 0;
  const int nChunks16 = SPLIT ? nChunksAll * (rank + 1) / a.split - cBegin : nChunksAll;
  const int nGroups = (nChunks16 + a.drainN - 1) / a.drainN;  // Dhi drains per tile
  // tap groups of a chunk: the first tgExtra groups have tgBase + 1 taps, the others tgBase
  const int nTapGroups = (a.k + a.wG - 1) / a.wG, tgBase = a.k / nTapGroups, tgExtra = a.k % nTapGroups;

  if (threadIdx.x == 0) {
    for (int i = 0; i < NB; ++i) mbarInit(&bFull[i], PRO_WARPS), mbarInit(&bEmpty[i], 1);
    for (int i = 0; i < MAX_W_STAGES; ++i) mbarInit(&wFull[i], 1), mbarInit(&wEmpty[i], 1);
    for (int i = 0; i < HB; ++i) mbarInit(&hiFull[i], 1), mbarInit(&hiEmpty[i], EPI_WARPS);
    mbarInit(loFull, 1), mbarInit(loEmpty, EPI_WARPS);
    for (int i = 0; i < NRAW; ++i) mbarInit(&rawFull[i], 1), mbarInit(&rawEmpty[i], PRO_WARPS);
    for (int i = 0; i < EPI_WARPS; ++i) mbarInit(&resBar[i], 1);
    mbarInit(recvBar, 1), mbarInit(tileBar, EPI_WARPS);
    *abortFlag = 0;
    fenceBarrierInit();
  }
  if (warp == MMA_WARP) {  // the MMA warp owns the TMEM allocation
    tmemAlloc(tmemSlot, 512);
    tmemRelinquish();
  }
  tcFenceBefore();
  __syncthreads();
  tcFenceAfter();
  const uint32_t tmemBase = *tmemSlot;
  const uint32_t tmemHi = tmemBase, tmemLo = tmemBase + NT;

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
  auto profAddIf = [&](bool mine, int slot, long long v) {  // one lane of a role adds the counts that it holds
    if (kProf && a.prof && mine)
      atomicAdd(reinterpret_cast<unsigned long long*>(a.prof + slot), (unsigned long long)v);
  };
  auto profAdd = [&](int slot, long long v) { profAddIf(lane == 0, slot, v); };
  // First timeout wins the low 16 bits; the flag bits above them are kept. One lane of a role reports; in the MMA issuer the
  // only lane that runs, whichever it is.
  auto giveUp = [&](int role, int code) {
    if (lane == 0 || warp == MMA_WARP) {
      int old = *a.status;
      while ((old & kStatusWaitMask) == 0) {
        const int seen = atomicCAS(a.status, old, old | (role << 8) | code);
        if (seen == old) break;
        old = seen;
      }
      *abortFlag = 1;
    }
  };

  // Split form with statsIn: each CTA folds the chunk statistics of the channels it contracts into their AdaIN affine (sPar, see
  // the producers). A launch of its own costs 3.5 us plus a gap in front of every conv; here it is, for rows of up to 32 pairs
  // (4096 columns), one round of loads under the first weight and input copies, eight lanes per channel on the sixteen warps that
  // have nothing to do yet. In double and relative to the row's first mean, so that one pass over the pairs gives mean and
  // variance as adainAffineKernel's two do: a first mean far from the row's costs at most a factor of the number of pairs of 2^-53.
  // Two passes on eight warps took 1.6-1.9 us; this and the finish phase's channels side by side together 339 -> 320 us at T = 24.
  const bool fold = SPLIT != 0 && ACT != 0 && TS == 0 && a.statsIn != nullptr;
  if (fold && warp < EPI_WARPS + PRO_WARPS) {
    dependenciesWait();
    constexpr int R = 4;  // pairs per lane in flight
    const int cEnd = (cBegin + nChunks16) * KC, sub = lane & 7, nch = int((a.l + NTS - 1) / NTS);
    const double nT = double(NTS), nLast = double(a.l - int64_t(nch - 1) * NTS), invL = 1.0 / double(a.l);
#pragma unroll 1
    for (int c0 = cBegin * KC + warp * 4; c0 < cEnd; c0 += (EPI_WARPS + PRO_WARPS) * 4) {  // warp-uniform; KC is a multiple of 4
      const int c = c0 + (lane >> 3);
      // 8-byte aligned, as adain_affine wants
      const float2* const st = reinterpret_cast<const float2*>(a.statsIn) + int64_t(c) * nch;
      const float gamma = a.gb[c], beta = a.gb[a.ci + c], al = ACT == 1 ? a.alpha[c] : 1.f;
      const double first = double(st[0].x);
      double s1 = 0.0, s2 = 0.0;  // sum of (x - first), sum of (x - first)^2
#pragma unroll 1
      for (int t0 = sub; t0 < nch; t0 += 8 * R) {
        float2 v[R];
#pragma unroll
        for (int e = 0; e < R; ++e) v[e] = t0 + 8 * e < nch ? st[t0 + 8 * e] : make_float2(0.f, 0.f);
#pragma unroll
        for (int e = 0; e < R; ++e) {
          const int t = t0 + 8 * e;
          const double cols = t + 1 < nch ? nT : t < nch ? nLast : 0.0, d = double(v[e].x) - first;
          s1 += cols * d, s2 += double(v[e].y) + cols * d * d;
        }
      }
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) s1 += __shfl_xor_sync(0xffffffffu, s1, o), s2 += __shfl_xor_sync(0xffffffffu, s2, o);
      if (sub == 0) {
        const double dm = s1 * invL, v = s2 * invL - dm * dm;
        const float var = v < 0.0 ? 0.f : float(v);  // (a NaN stays one)
        sPar[c] = -float(first + dm);
        sPar[a.ci + c] = (1.f + gamma) * (1.0f / sqrtf(var + a.eps)) * al;
        sPar[2 * a.ci + c] = beta * al;
        sPar[3 * a.ci + c] = 1.f / al;
      }
      __syncwarp();
    }
  }

  if (warp < EPI_WARPS) {
    // ------------------------------------------------------------------ accumulate + epilogue
    if (fold) asm volatile("bar.arrive 1, %0;" ::"n"((EPI_WARPS + PRO_WARPS) * 32) : "memory");  // the producers wait for this part
    regInc<EPI_REGS>();
    dependenciesWait();
    const int q = warp & 3, g = warp >> 2;  // TMEM lane quarter, half of the tile
    // 32-column batches of this warp (of 256 columns: 4) and its first column
    const int nb0 = NARROW ? ((W >> 5) + 1) >> 1 : EC / 32, nbat = NARROW && g ? (W >> 5) - nb0 : nb0, gcol = g * nb0 * 32;
    float* const tile = sStage + warp * STAGE_FLOATS;                                  // unaligned route: [32][33]
    unsigned char* const box = smemRaw + warp * BOX_BYTES;                             // aligned route: swizzled 32 x 32
    unsigned char* const boxRow = box + lane * 128;                                    // this lane's row of the box
    const int swz = lane & 7;  // 128-byte swizzle: 16-byte chunk c of row r sits at chunk c ^ (r & 7)
    uint64_t* const myRes = &resBar[warp];
    static_assert(!TMAO || (TS == 0 && !PARTIAL), "boxes need whole 32-channel row groups of a conv1d");
    constexpr bool tmaOut = TMAO;
    const uint32_t laneBase = uint32_t(q * 32) << 16;
    constexpr uint32_t kSleepEpi = SPLIT ? SLEEP_EPI_SPLIT_NS : SLEEP_EPI_NS;
    uint32_t groupIt = 0, tileIt = 0, resIt = 0;
    bool dead = false, resInFlight = false, arrived = false;
    SplitTail<TS, SPLIT ? SPLIT : NTS> tail(a, tile0, rank);
    float* const recv = sStage + partBytes(NTK) / 4;
    if (SPLIT && threadIdx.x == 0) mbarArriveExpectTx(recvBar, tail.expected(a, rank));
    if constexpr (SPLIT != 0) tail.prefetch(a, tail.firstUnit(warp, lane), lane);
    long long wHi = 0, wLo = 0, cPre = 0, cFin = 0;
    const long long tStart = kProf ? clock64() : 0;
    for (int t = tile0; t < numTiles && !dead; t += tileStep, ++tileIt) {
      const int tt = t / a.numCoBlk, cb = t - tt * a.numCoBlk;
      const long long tPre = kProf ? clock64() : 0;
      const int64_t tChunk = int64_t(tt) * W + gcol;  // first output column of this warp
      const int64_t nValid64 = a.lo - tChunk;
      const int nValid = nValid64 <= 0 ? 0 : (nValid64 < nbat * 32 ? int(nValid64) : nbat * 32);
      // conv: the warp's rows are 32 consecutive output channels. ConvTranspose: rows are (channel, phase) pairs,
      // CQ channels x TS phases per warp (lane = cl * TS + r), the last 32 - CQ * TS rows are zero padding.
      constexpr int CQ = TS ? 32 / TS : 32, ROWS = TS ? CQ * TS : 32;
      // Row pitch of the warp's transpose tile. ConvTranspose: 35 floats, so that both the row-wise accesses (lane =
      // row: 3 * lane mod 32 is a permutation) and the interleaved ones (phase r, column q -> bank 3 r + q: at most
      // two lanes per bank) stay cheap; its 30 rows still fit the tile (30 x 35 <= 32 x 33).
      constexpr int TP = TS ? 35 : STAGE_PITCH;
      static_assert(ROWS * TP <= STAGE_FLOATS, "transpose tile");
      const int coBase = TS ? (cb * 4 + q) * CQ : cb * MT + q * 32;
      const int co = TS ? coBase + lane / (TS ? TS : 1) : coBase + lane;
      const bool rowOk = TS ? (lane < ROWS && co < a.co) : (!PARTIAL || co < a.co);
      const float bias = (!SPLIT && a.bias && rowOk) ? a.bias[co] : 0.f;
      // channels of this warp that exist (may be <= 0 in the last block)
      const int coValid = (TS || PARTIAL) ? (a.co - coBase < CQ ? a.co - coBase : CQ) : 32;
      // Running sums start from the bias. The residual is added one 32-column batch at a time: while the warp waits
      // for drain group c, residual batch c travels into the warp's tile (a TMA box, or cp.async with lanes along
      // time); after the group has been drained the batch is read back with lanes along channels and added.
      // The global latency hides behind a whole group of MMAs and no registers are held while waiting.
      float S[128];
#pragma unroll
      for (int j = 0; j < EC; ++j) S[j] = bias;
      const bool hasRes = !SPLIT && a.residual != nullptr;
      // ConvTranspose with the left reflect pad: out[co, 0] = unpadded[co, 1] + res[co, 0] (the reference copies
      // the column, then adds the residual). The lane that owns (column 0, phase 1) keeps that element's residual
      // out of its running sum and adds it last, so the reflect column gets the plain conv sum.
      const bool reflectLane = TS != 0 && a.padLeft != 0 && tChunk == 0 && lane < ROWS && (lane % (TS ? TS : 1)) == 1;
      float resHeld = 0.f;
      auto fetchResidual = [&](int b) {  // batch b of the warp's 128 columns -> tile (zero where out of range)
        if (tmaOut) {
          if (lane == 0) {
            bulkWaitRead();  // the stores of the previous tile have read the box
            mbarArriveExpectTx(myRes, BOX_BYTES);
            tmaLoad2d(box, &mapRes, int(tChunk) + b * BOX, coBase, myRes);
          }
          resInFlight = true;
          return;
        }
        if constexpr (TS == 0) {
          const bool ok = b * 32 + lane < nValid;
          const float* rp = a.residual + int64_t(coBase) * a.resPitch + tChunk + b * 32 + lane;
          float* tp = tile + lane;
          const int rowsOk = ok ? (PARTIAL ? (coValid < 0 ? 0 : coValid) : 32) : 0;  // rows this lane copies
          int i = 0;
#pragma unroll 8
          for (; i < rowsOk; ++i, tp += STAGE_PITCH, rp += a.resPitch) cpAsync4(tp, rp);
          for (; i < 32; ++i, tp += STAGE_PITCH) *tp = 0.f;
        } else {
          // channel cl: the 32 * TS output samples u = (tChunk + 32 b) * TS + idx are contiguous in memory; copy
          // i = cl * TS + f moves idx = 32 f + lane, which is column idx / TS of phase idx % TS
          // The tile offsets of the TS copies of a channel depend on the lane only: computed once per batch, then a
          // rolled loop over the channels with pointer increments (this runs four times per tile on every epilogue
          // warp; the index arithmetic of the (channel, copy) pair per element cost more than the copies).
          const int64_t uEnd = a.lo * TS, u0 = (tChunk + b * 32) * TS;
          int off[TS ? TS : 1];
#pragma unroll
          for (int f = 0; f < TS; ++f) off[f] = ((f * 32 + lane) % TS) * TP + (f * 32 + lane) / TS;
          const int64_t left = uEnd - u0 - lane;  // copy f of this lane is inside the row iff f * 32 < left
          const float* rp = a.residual + int64_t(coBase) * a.resPitch + a.padLeft + u0 + lane;
          float* tp = tile;
#pragma unroll 1
          for (int cl = 0; cl < CQ; ++cl, rp += a.resPitch, tp += TS * TP) {
            const bool chOk = cl < coValid;
#pragma unroll
            for (int f = 0; f < TS; ++f) {
              if (chOk && f * 32 < left) cpAsync4(tp + off[f], rp + f * 32);
              else tp[off[f]] = 0.f;
            }
          }
        }
        cpAsyncCommit();
      };
      auto addResidual = [&](int b) {
        if (tmaOut) {
          if (!mbarWait(myRes, resIt & 1, abortFlag, 32)) {
            giveUp(1, 3);
            dead = true;
            return;
          }
          ++resIt, resInFlight = false;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const float4 v = *reinterpret_cast<const float4*>(boxRow + ((c ^ swz) << 4));
            S[b * 32 + 4 * c] += v.x, S[b * 32 + 4 * c + 1] += v.y, S[b * 32 + 4 * c + 2] += v.z,
                S[b * 32 + 4 * c + 3] += v.w;
          }
          __syncwarp();
          return;
        }
        cpAsyncWait<0>();
        __syncwarp();
        if (TS == 0 || lane < ROWS) {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float r = tile[lane * TP + j];
            if (TS != 0 && b == 0 && j == 0 && reflectLane) resHeld = r;
            else S[b * 32 + j] += r;
          }
        }
        __syncwarp();
      };
      if (kProf) cPre += clock64() - tPre;
      // wait for the group's hi chain, add it to the running sums, hand Dhi back
      auto drainGroup = [&]() -> bool {
        const uint32_t hb = HB == 2 ? groupIt & 1 : 0;
        if (!waitT(&hiFull[hb], (HB == 2 ? groupIt >> 1 : groupIt) & 1, wHi, kSleepEpi)) {
          giveUp(1, 1);
          return false;
        }
        tcFenceAfter();
        // Everything this CTA's MMAs read is read: peers may write over the operand buffers.
        if (SPLIT && groupIt + 1 == uint32_t(nGroups)) clusterArrive(), arrived = true;
#pragma unroll
        for (int b = 0; b < EC / 16; ++b) {
          if (NARROW && b >= 2 * nbat) break;
          uint32_t v[16];
          tmemLoad16Async(tmemHi + hb * NTK + laneBase + gcol + b * 16, v);
          tmemWaitLoads();
#pragma unroll
          for (int j = 0; j < 16; j += 2) {  // packed f32x2 adds: half the instructions of the accumulate loop
            const float2 sum = __fadd2_rn(make_float2(S[b * 16 + j], S[b * 16 + j + 1]),
                                          make_float2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])));
            S[b * 16 + j] = sum.x, S[b * 16 + j + 1] = sum.y;
          }
        }
        tcFenceBefore();
        __syncwarp();
        if (lane == 0) mbarArrive(&hiEmpty[hb]);
        ++groupIt;
        return true;
      };
      // Four residual batches per tile. With four or more drains the first four each carry one (fetched before the
      // wait for the group, added after the drain); with fewer drains the surplus batches get steps of their own
      // where this warp would otherwise only wait for a group: right after the first drain (the second group's MMAs
      // hide their fetch latency; before the first drain the warp is still busy with the previous tile's final
      // phase), or before the only drain of a tile, instead of between the last drain and the final phase.
      // One copy of the fetch and of the drain in the code (this kernel is far larger than the instruction cache,
      // and straight-line code that runs once per tile is fetched at a fraction of the issue rate); only the add
      // needs static register indices.
      const int nPre = hasRes && nGroups < nbat ? nbat - nGroups : 0;
      const int nSteps = nPre + nGroups, preAt = nGroups == 1 ? 0 : 1;  // first step without a drain
      int rb = 0;  // next residual batch
#pragma unroll 1
      for (int c = 0; c < nSteps && !dead; ++c) {
        const bool doRes = hasRes && rb < nbat;
        if (doRes) fetchResidual(rb);
        if (c == nSteps - 1) {
          // Last step of the tile (always a drain): Dlo is complete before the last hi MMAs are, so it is folded in
          // first and handed back, and the next tile's lo MMAs need not wait for the last drain and the final phase.
          if (!waitT(loFull, tileIt & 1, wLo, kSleepEpi)) {
            giveUp(1, 2);
            dead = true;
            break;
          }
          tcFenceAfter();
#pragma unroll
          for (int b = 0; b < EC / 32; ++b) {  // two 16-column loads in flight per wait
            if (NARROW && b >= nbat) break;
            uint32_t va[16], vb[16];
            tmemLoad16Async(tmemLo + laneBase + gcol + b * 32, va);
            tmemLoad16Async(tmemLo + laneBase + gcol + b * 32 + 16, vb);
            tmemWaitLoads();
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const float x = __uint_as_float(va[j]), y = __uint_as_float(vb[j]);
              S[b * 32 + j] = F16 ? fmaf(x, 1.f / kLoScale, S[b * 32 + j]) : S[b * 32 + j] + x;
              S[b * 32 + 16 + j] = F16 ? fmaf(y, 1.f / kLoScale, S[b * 32 + 16 + j]) : S[b * 32 + 16 + j] + y;
            }
          }
          tcFenceBefore();
          __syncwarp();
          if (lane == 0) mbarArrive(loEmpty);
        }
        if (c < preAt || c >= preAt + nPre) dead = !drainGroup();
        if (doRes && !dead) {
          switch (rb) {
            case 0: addResidual(0); break;
            case 1: addResidual(1); break;
            case 2: addResidual(2); break;
            default: addResidual(3); break;
          }
          ++rb;
        }
      }
      if (dead) break;
      const long long tFin = kProf ? clock64() : 0;
      if constexpr (SPLIT != 0) {
        float* const row = sStage + (q * 32 + lane) * PART_PITCH + gcol;
#pragma unroll
        for (int j = 0; j < EC; j += 4) *reinterpret_cast<float4*>(row + j) = make_float4(S[j], S[j + 1], S[j + 2], S[j + 3]);
        fenceProxyAsync();  // generic-proxy stores -> visible to the bulk copies
        __syncwarp();
        if (lane == 0) mbarArrive(tileBar);
        clusterWait();
        if (warp < a.split) {
          if (!mbarWait(tileBar, 0, abortFlag, 0)) {
            giveUp(1, 5);
            dead = true;
          } else if (lane == 0) {
            tail.send(a, sStage, recv, recvBar, rank, warp);
          }
        }
        if (kProf) cFin += clock64() - tFin;
        continue;
      }
      if (a.residual && a.outScale != 1.f) {
#pragma unroll
        for (int j = 0; j < 128; ++j) S[j] *= a.outScale;
      }

      if constexpr (TS == 0) {
        // Per 32-column batch: chunk statistics of this lane's channel from the registers, and the store. Aligned
        // route: the registers go to the warp's box in the 128-byte swizzle (8 conflict-free 16-byte stores), one
        // lane sends the box with a bulk tensor store (clipped at the end of the row) and the statistics of the
        // batch run while the TMA unit reads it. Unaligned route: the registers go to the [32][33] tile and rolled
        // loops store it transposed, lanes along time (rolled loops stay in the instruction cache; the unrolled form
        // of this phase, 1100 instructions run once per tile, ran at about 20 clocks per instruction).
        float pMean[4], pM2[4];
        const int rowsValid = PARTIAL ? (coValid < 0 ? 0 : coValid) : 32;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int nb = nValid - b * 32 <= 0 ? 0 : (nValid - b * 32 < 32 ? nValid - b * 32 : 32);  // valid columns
          if (tmaOut) {
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
                tmaStore2d(&mapOut, int(tChunk) + b * BOX, coBase, box);
                bulkCommit();
              }
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) tile[lane * STAGE_PITCH + j] = S[b * 32 + j];
            __syncwarp();
          }
          // statistics of the valid columns of this lane's channel (two passes over the registers, four chains)
          float m, q0 = 0.f, q1 = 0.f, q2 = 0.f, q3 = 0.f;
          {
            float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
            if (nb == 32) {
#pragma unroll
              for (int j = 0; j < 32; j += 4)
                s0 += S[b * 32 + j], s1 += S[b * 32 + j + 1], s2 += S[b * 32 + j + 2], s3 += S[b * 32 + j + 3];
              m = ((s0 + s1) + (s2 + s3)) * (1.f / 32.f);
#pragma unroll
              for (int j = 0; j < 32; j += 4) {
                const float d0 = S[b * 32 + j] - m, d1 = S[b * 32 + j + 1] - m, d2 = S[b * 32 + j + 2] - m,
                            d3 = S[b * 32 + j + 3] - m;
                q0 = fmaf(d0, d0, q0), q1 = fmaf(d1, d1, q1), q2 = fmaf(d2, d2, q2), q3 = fmaf(d3, d3, q3);
              }
            } else {  // ragged end of a row: rolled loops over the copy in shared memory (rare: keeps the code small)
              auto at = [&](int j) -> float {
                return tmaOut ? *reinterpret_cast<const float*>(boxRow + (((j >> 2) ^ swz) << 4) + ((j & 3) << 2))
                              : tile[lane * STAGE_PITCH + j];
              };
#pragma unroll 1
              for (int j = 0; j < nb; ++j) s0 += at(j);
              m = nb > 0 ? s0 / float(nb) : 0.f;
#pragma unroll 1
              for (int j = 0; j < nb; ++j) {
                const float d = at(j) - m;
                q0 = fmaf(d, d, q0);
              }
            }
          }
          pMean[b] = m, pM2[b] = (q0 + q1) + (q2 + q3);
          if (!tmaOut) {
            // store with lanes along time
            if (lane < nb) {
              float* op = a.out + int64_t(coBase) * a.outPitch + tChunk + b * 32 + lane;
              const float* col = tile + lane;
              int i = 0;
#pragma unroll 1
              for (; i + 8 <= rowsValid; i += 8) {
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = col[(i + e) * STAGE_PITCH];
#pragma unroll
                for (int e = 0; e < 8; ++e) op[int64_t(i + e) * a.outPitch] = v[e];
              }
              for (; i < rowsValid; ++i) op[int64_t(i) * a.outPitch] = col[i * STAGE_PITCH];
            }
            __syncwarp();
          }
        }
        if (NARROW && a.stats && (!PARTIAL || co < a.co)) {  // a pair per 32 columns
          float2* const st = reinterpret_cast<float2*>(a.stats) + int64_t(co) * a.nchunks + tChunk / 32;
#pragma unroll
          for (int b = 0; b < 4; ++b)
            if (b * 32 < nValid) st[b] = make_float2(pMean[b], pM2[b]);
        } else if (a.stats && nValid > 0 && (!PARTIAL || co < a.co)) {
          // exact combine of the four 32-column partials: mean = sum n_b m_b / n, M2 = sum M2_b + sum n_b (m_b - mean)^2
          float sum = 0.f;
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const int nb = nValid - b * 32 <= 0 ? 0 : (nValid - b * 32 < 32 ? nValid - b * 32 : 32);
            sum = fmaf(float(nb), pMean[b], sum);
          }
          const float mean = sum / float(nValid);
          float m2 = 0.f;
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const int nb = nValid - b * 32 <= 0 ? 0 : (nValid - b * 32 < 32 ? nValid - b * 32 : 32);
            const float d = pMean[b] - mean;
            m2 += pM2[b] + float(nb) * d * d;
          }
          float* st = a.stats + (int64_t(co) * a.nchunks + tChunk / 128) * 2;
          if ((reinterpret_cast<uintptr_t>(a.stats) & 7) == 0) *reinterpret_cast<float2*>(st) = make_float2(mean, m2);
          else st[0] = mean, st[1] = m2;
        }
      } else {
        // ConvTranspose: interleave the TS phases of each channel back into contiguous output samples
        const int64_t uEnd = a.lo * TS;
        float reflectVal = 0.f;
        if (reflectLane) {
          reflectVal = S[0];   // plain conv sum of (column 0, phase 1) = unpadded[co, 1]
          S[0] += resHeld;     // the element's own residual, added last
        }
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          if (NARROW && b >= nbat) break;
          const int64_t u0 = (tChunk + b * 32) * TS;
          if (lane < ROWS) {
#pragma unroll
            for (int j = 0; j < 32; ++j) tile[lane * TP + j] = S[b * 32 + j];
          }
          __syncwarp();
          int off[TS ? TS : 1];  // as in the residual fetch: lane-only tile offsets, then pointer increments
#pragma unroll
          for (int f = 0; f < TS; ++f) off[f] = ((f * 32 + lane) % TS) * TP + (f * 32 + lane) / TS;
          const int64_t left = uEnd - u0 - lane;
          float* op = a.out + int64_t(coBase) * a.outPitch + a.padLeft + u0 + lane;
          const float* tp = tile;
#pragma unroll 1
          for (int cl = 0; cl < CQ; ++cl, op += a.outPitch, tp += TS * TP) {
            if (cl >= coValid) break;
#pragma unroll
            for (int f = 0; f < TS; ++f)
              if (f * 32 < left) op[f * 32] = tp[off[f]];
          }
          __syncwarp();
        }
        if (reflectLane && co < a.co && uEnd > 1) {
          const int64_t row = int64_t(co) * a.outPitch;
          a.out[row] = reflectVal + (a.residual ? a.residual[int64_t(co) * a.resPitch] : 0.f);
        }
      }
      if (kProf) cFin += clock64() - tFin;
    }
    if constexpr (SPLIT != 0) {
      if (dead && !arrived) clusterArrive(), clusterWait();  // the arrival that the peers wait for
      const bool got = __all_sync(0xffffffffu, !dead && mbarWait(recvBar, 0, abortFlag, 0));
      clusterArrive();  // what the peers sent here has arrived; they need not wait for what is left
      if (got) tail.finish(a, recv, warp, lane);
      else if (!dead) giveUp(1, 4);
    }
    // Copies of this warp still in flight must end before the CTA may exit: a residual box after an abort, and the
    // output boxes on every path.
    if (resInFlight) mbarWaitQuiet(myRes, resIt & 1);
    if (tmaOut && lane == 0) bulkWaitAll();
    if (kProf && warp == 0)
      profAdd(5, wHi), profAdd(6, wLo), profAdd(7, cPre), profAdd(8, cFin), profAdd(9, clock64() - tStart);
  } else if (warp < EPI_WARPS + PRO_WARPS) {
    // ------------------------------------------------------------------ activation producers
    regDec<PRO_REGS>();
    dependenciesWait();
    const int pw = warp - EPI_WARPS;
    const int cg = pw & 3, hf = pw >> 2;  // channel group of 4 inside the 16-channel chunk; half of the tile's columns
    // A warp stages the rows of its half, SLOTS per lane, with addresses that are immediates. The rows beyond the tile's
    // columns (at most 53) take one more slot for up to 32 of them: the first 32 go to the warps of half `raw buffer`, so
    // that the halves take turns, the rest to the other half.
    const int mainRows = NARROW ? a.mainRows : NTK, halfRows = mainRows / 2, slots = mainRows / 64;
    const bool tmaIn = a.tmaIn != 0;
    // per-channel parameters, once: sPar = [-mean | a | b | inv] with a = scale, b = beta (x alpha for Snake), inv = 1/alpha
    for (int c = cBegin * KC + pw * 32 + lane; !fold && c < (cBegin + nChunks16) * KC; c += PRO_WARPS * 32) {
      const float al = ACT == 1 ? a.alpha[c] : 1.f;
      sPar[c] = a.affine ? -a.affine[c] : 0.f;
      sPar[a.ci + c] = (a.affine ? a.affine[a.ci + c] : 1.f) * al;
      sPar[2 * a.ci + c] = (a.affine ? a.affine[2 * a.ci + c] : 0.f) * al;
      sPar[3 * a.ci + c] = 1.f / al;
    }
    if (fold) asm volatile("bar.sync 1, %0;" ::"n"((EPI_WARPS + PRO_WARPS) * 32) : "memory");
    else asm volatile("bar.sync 1, %0;" ::"n"(PRO_WARPS * 32) : "memory");  // producer warps only

    // First row beyond the tile's columns that this lane stages from raw buffer rb.
    auto extRow = [&](uint32_t rb) { return NTK + (uint32_t(hf) == rb ? 0 : 32) + lane; };

    // Unaligned route: cp.async of this thread's part of the raw window of chunk c of the tile whose window starts at
    // input position posT (= tile * W - padding) into staging buffer rb. This runs once per chunk on every producer
    // thread. A thread copies what it will itself read back.
    auto issueCopies = [&](int64_t posT, int c, int rb) {
      const float* xc = a.x + int64_t((cBegin + c) * KC + cg * 4) * a.xPitch + posT;
      float* const base = sRaw + rb * rawBufFloats;
      auto copy = [&](int r, float* dst, int pitch) {
        const int64_t pos = posT + r;
        if (pos >= 0 && pos < a.l) {
          const float* src = xc + r;
#pragma unroll
          for (int j = 0; j < 4; ++j) cpAsync4(dst + j * pitch, src + j * a.xPitch);
        }
      };
      const int r0 = hf * halfRows + lane;
#pragma unroll 1
      for (int sl = 0; sl < slots; ++sl) copy(r0 + sl * 32, base + cg * 4 * NTK + r0 + sl * 32, NTK);
      const int r = extRow(rb);
      if (r < rows) copy(r, base + KC * NTK + cg * 4 * ext + r - NTK, ext);
    };

    int t = tile0, c = 0;
    uint32_t buf = 0, bufPar = 1, rawBuf = 0, rawPar = 0;  // activation buffer + parity of its last release; raw buffer + parity of its fill
    long long wB = 0, wCp = 0, cTr = 0;
    const long long tStart = kProf ? clock64() : 0;
    int64_t pos0 = int64_t(t / a.numCoBlk) * W - a.padding;  // input position of row 0 of the current tile's window
    if (!tmaIn) {
      if (t < numTiles) issueCopies(pos0, c, 0);
      cpAsyncCommit();
    }
    while (t < numTiles) {
      int tn = t, cn = c + 1;
      int64_t posN = pos0;
      if (cn == nChunks16) {
        cn = 0, tn = t + tileStep;
        posN = int64_t(tn / a.numCoBlk) * W - a.padding;
      }
      if (tmaIn) {
        if (!waitT(&rawFull[rawBuf], rawPar, wCp, SLEEP_PRO_NS)) {
          giveUp(2, 2);
          break;
        }
      } else {
        if (tn < numTiles) issueCopies(posN, cn, rawBuf ^ 1);
        cpAsyncCommit();
        const long long tCp = kProf ? clock64() : 0;
        cpAsyncWait<1>();  // this chunk's copies (the older group) have landed; the next chunk's stay in flight
        if (kProf) wCp += clock64() - tCp;
      }
      if (!waitT(&bEmpty[buf], bufPar, wB, SLEEP_PRO_NS)) {
        giveUp(2, 1);
        break;
      }
      const long long tTr = kProf ? clock64() : 0;
      // tf32 split: [cg][rows][4 f32]; f16 split: [cg / 2][rows][8 f16], this thread's 4 channels = half of a chunk
      float* const hi = F16 ? sAct + buf * actBufFloats + (cg >> 1) * rows * 4 + (cg & 1) * 2
                            : sAct + buf * actBufFloats + cg * rows * 4;
      float* const lo = hi + actBufFloats / 2;
      const float* const raw = sRaw + rawBuf * rawBufFloats;
      // this thread's four channels: constants in registers for the whole chunk
      const float* par = sPar + (cBegin + c) * KC + cg * 4;
      const float4 nm = *reinterpret_cast<const float4*>(par), pa = *reinterpret_cast<const float4*>(par + a.ci),
                   pb = *reinterpret_cast<const float4*>(par + 2 * a.ci), pi = *reinterpret_cast<const float4*>(par + 3 * a.ci);
      float big = 0.f;  // largest |value| this thread staged in the chunk (f16 range check, once per chunk)
      // rows [okLo, okHi) are inside the valid range, the others are zero padding (after the activation)
      const int64_t x0 = pos0 - a.delta;
      const int okLo = x0 >= a.validLo ? 0 : int(a.validLo - x0 < rows ? a.validLo - x0 : rows);
      const int okHi = a.validHi - x0 >= rows ? rows : int(a.validHi - x0);
      // One row of four channels; sp: this thread's first channel of the row, the others `pitch` floats on. Branch-free, so
      // that the slots' dependency chains interleave.
      auto stage = [&](auto edge, int r, const float* sp, int pitch) {
        float2 v01 = activate2<ACT>(make_float2(sp[0], sp[pitch]), make_float2(nm.x, nm.y), make_float2(pa.x, pa.y),
                                    make_float2(pb.x, pb.y), make_float2(pi.x, pi.y), a.slope);
        float2 v23 = activate2<ACT>(make_float2(sp[2 * pitch], sp[3 * pitch]), make_float2(nm.z, nm.w), make_float2(pa.z, pa.w),
                                    make_float2(pb.z, pb.w), make_float2(pi.z, pi.w), a.slope);
        if constexpr (decltype(edge)::value) {
          const bool ok = r >= okLo && r < okHi;
          v01.x = ok ? v01.x : 0.f, v01.y = ok ? v01.y : 0.f, v23.x = ok ? v23.x : 0.f, v23.y = ok ? v23.y : 0.f;
        }
        if constexpr (!F16) {
          float4 h, l;
          h.x = tf32Round(v01.x), h.y = tf32Round(v01.y), h.z = tf32Round(v23.x), h.w = tf32Round(v23.y);
          const float2 l01 = __fadd2_rn(v01, make_float2(-h.x, -h.y)), l23 = __fadd2_rn(v23, make_float2(-h.z, -h.w));
          l = make_float4(l01.x, l01.y, l23.x, l23.y);
          *reinterpret_cast<float4*>(hi + r * 4) = h;
          *reinterpret_cast<float4*>(lo + r * 4) = l;
        } else {
          // hi = f16(v), lo = f16((v - hi) * 2^11); 4 channels = 8 bytes of the row's 16-byte K chunk (channel groups
          // 2 j and 2 j + 1 share chunk j). A value beyond the f16 range becomes infinite here and is reported below.
          big = max3(max3(big, fabsf(v01.x), fabsf(v01.y)), fabsf(v23.x), fabsf(v23.y));
          const __half2 h01 = __float22half2_rn(v01), h23 = __float22half2_rn(v23);
          const float2 sc = make_float2(kLoScale, kLoScale);
          const float2 f01 = __half22float2(h01), f23 = __half22float2(h23);
          const __half2 l01 = __float22half2_rn(__fmul2_rn(__fadd2_rn(v01, make_float2(-f01.x, -f01.y)), sc));
          const __half2 l23 = __float22half2_rn(__fmul2_rn(__fadd2_rn(v23, make_float2(-f23.x, -f23.y)), sc));
          uint2 hw, lw;
          hw.x = *reinterpret_cast<const uint32_t*>(&h01), hw.y = *reinterpret_cast<const uint32_t*>(&h23);
          lw.x = *reinterpret_cast<const uint32_t*>(&l01), lw.y = *reinterpret_cast<const uint32_t*>(&l23);
          *reinterpret_cast<uint2*>(hi + r * 4) = hw;
          *reinterpret_cast<uint2*>(lo + r * 4) = lw;
        }
      };
      const int r0 = hf * halfRows + lane, rx = extRow(rawBuf);
      const float* const sp0 = raw + cg * 4 * NTK + r0;
      const float* const spx = raw + KC * NTK + cg * 4 * ext + rx - NTK;
      if (okLo == 0 && okHi == rows) {  // all but the tiles at the ends of the valid range
        auto all = [&](auto n) {
#pragma unroll
          for (int sl = 0; sl < decltype(n)::value; ++sl) stage(std::false_type{}, r0 + sl * 32, sp0 + sl * 32, NTK);
        };
        if (!NARROW) all(std::integral_constant<int, NTK / 64>{});
        else if (slots == 4) all(std::integral_constant<int, 4>{});
        else all(std::integral_constant<int, 3>{});
        if (rx < rows) stage(std::false_type{}, rx, spx, ext);
      } else {
#pragma unroll 2
        for (int sl = 0; sl < slots; ++sl) stage(std::true_type{}, r0 + sl * 32, sp0 + sl * 32, NTK);
        if (rx < rows) stage(std::true_type{}, rx, spx, ext);
      }
      if (F16 && big > 65504.f) atomicOr(a.status, kStatusF16Range);
      fenceProxyAsync();  // generic-proxy stores -> visible to the tensor core (async proxy)
      __syncwarp();
      if (lane == 0) {
        mbarArrive(&bFull[buf]);
        if (tmaIn) mbarArrive(&rawEmpty[rawBuf]);  // the raw buffer may be refilled
      }
      if (kProf) cTr += clock64() - tTr;
      t = tn, c = cn, pos0 = posN;
      if (++rawBuf == NRAW) rawBuf = 0, rawPar ^= 1;
      if (++buf == uint32_t(NB)) buf = 0, bufPar ^= 1;
    }
    cpAsyncWait<0>();
    if (kProf && pw == 0) profAdd(10, wB), profAdd(11, wCp), profAdd(12, cTr), profAdd(13, clock64() - tStart);
  } else {
    regDec<CTL_REGS>();
    if (warp == W_WARP) {
      // ---------------------------------------------------------------- weight producer
      dependenciesWait();  // the pack may have been queued just before; the input window is waited for longer anyway
      uint32_t wIt = 0, ws = 0, wPh = 1;  // stages issued, ring slot, parity of the slot's previous release
      bool dead = false;
      long long wW = 0;
      const long long tStart = kProf ? clock64() : 0;
      const int64_t blocksPerCo = int64_t(nChunksAll) * a.k;  // one block (hi + lo of one tap) per chunk and tap
      const int slotFloats = a.wG * W_STAGE_FLOATS;
      for (int t = tile0; t < numTiles && !dead; t += tileStep) {
        const int tt = t / a.numCoBlk, cb = t - tt * a.numCoBlk;
        const float* src = a.wp + (int64_t(cb) * blocksPerCo + int64_t(cBegin) * a.k) * W_STAGE_FLOATS;
        for (int c = 0; c < nChunks16 && !dead; ++c) {
          for (int gi = 0; gi < nTapGroups; ++gi, ++wIt) {
            const int n = tgBase + (gi < tgExtra ? 1 : 0);
            if (!waitT(&wEmpty[ws], wPh, wW, SLEEP_W_NS)) {
              giveUp(3, 1);
              dead = true;
              break;
            }
            if (lane == 0) {
              mbarArriveExpectTx(&wFull[ws], n * W_STAGE_BYTES);
              bulkCopyG2S(sW + ws * slotFloats, src, n * W_STAGE_BYTES, &wFull[ws]);
            }
            __syncwarp();
            src += n * W_STAGE_FLOATS;
            if (++ws == uint32_t(a.wStages)) ws = 0, wPh ^= 1;  // wrap counters: a division here cost more than the copy
          }
        }
      }
      if (kProf) profAdd(14, wW), profAdd(15, clock64() - tStart);
      // Every copy this warp issued must have landed before the CTA may exit. On the normal path the MMA warp has
      // consumed them all; after an abort, wait (bounded) for the stages still in flight.
      if (*abortFlag) {
        const uint32_t issued = wIt;
        for (uint32_t i = issued > uint32_t(a.wStages) ? issued - a.wStages : 0; i < issued; ++i)
          mbarWaitQuiet(&wFull[i % a.wStages], (i / a.wStages) & 1);
      }
    } else if (warp == RAW_WARP) {
      // ---------------------------------------------------------------- raw-window loader (aligned route)
      // Per (tile, chunk): the 16 channels' windows from the 16-byte boundary at or below their first column, as two boxes
      // (a box holds at most 256 elements per dimension): the tile's columns and what lies beyond them. Columns outside
      // [0, L) arrive as zeros and are never used: the producers write the zero padding themselves, after the activation.
      if (a.tmaIn && lane == 0) {
        dependenciesWait();
        uint32_t rb = 0, ph = 1, issued = 0;
        long long wR = 0;
        bool dead = false;
        const uint32_t bytes = uint32_t(rawBufFloats) * 4;
        for (int t = tile0; t < numTiles && !dead; t += tileStep) {
          const int x0 = (t / a.numCoBlk) * W - a.padding - a.delta;
          for (int c = 0; c < nChunks16; ++c, ++issued) {
            if (!waitT(&rawEmpty[rb], ph, wR, SLEEP_W_NS)) {
              giveUp(5, 1);
              dead = true;
              break;
            }
            float* dst = sRaw + rb * rawBufFloats;
            mbarArriveExpectTx(&rawFull[rb], bytes);
            tmaLoad2d(dst, &mapX, x0, (cBegin + c) * KC, &rawFull[rb]);
            if (ext) tmaLoad2d(dst + KC * NTK, &mapExt, x0 + NTK, (cBegin + c) * KC, &rawFull[rb]);
            if (++rb == NRAW) rb = 0, ph ^= 1;
          }
        }
        if (*abortFlag) {
          for (uint32_t i = issued > NRAW ? issued - NRAW : 0; i < issued; ++i)
            mbarWaitQuiet(&rawFull[i % NRAW], (i / NRAW) & 1);
        }
      }
    } else if (warp == MMA_WARP) {
      // ---------------------------------------------------------------- MMA issuer
      // One thread issues every MMA: hi*hi into Dhi, lo*hi and hi*lo into Dlo. It walks the (tile, chunk, tap group)
      // sequence, one tap group per round: a single wait for the group's weight slot, its MMAs back to back, a single
      // release. Measured on this part: a lone thread streams MMAs at the pipe's rate (128 clocks for M128 N256 K16)
      // as long as nothing but MMAs is issued; the thread is held while an MMA waits for the pipe, and what it
      // executes between two MMAs is covered by no more than the one MMA in flight. So the bookkeeping for the next
      // round (ring counters, a first poll of the next slot's barrier) sits where it is free, and only the release
      // and, rarely, a real wait separate two rounds.
      // Order inside a round: the lo MMAs first, then the hi MMAs, so that the wait for the Dhi drain at the start of a
      // drain group is covered by the round's own lo MMAs. At the start of a tile too: the epilogue folds Dlo before the
      // tile's last drain, so Dlo is handed back first. (Issuing hi first in the last round of a drain group, which
      // lengthens the cover of the drain to this round's and the next round's lo MMAs, shortened the waits but not the
      // tile: the extra code in this loop cost what the waits gave back.)
      const uint64_t dA0 = makeDesc(smemAddr(sW), MT * 16, 128);
      const uint64_t dB0 = makeDesc(smemAddr(sAct), rows * 16, 128) + uint32_t(a.delta);
      constexpr uint32_t kStageU = W_STAGE_BYTES >> 4, kLoAU = (W_STAGE_BYTES / 2) >> 4, kKsAU = (2 * MT * 16) >> 4;
      // activation buffer: hi half then lo half; one MMA spans two 16-byte K chunks (K8 of f32 or K16 of f16);
      // one staged time row = 16 bytes = one descriptor address unit
      const uint32_t bufU = uint32_t(actBufFloats * 4) >> 4, loBU = bufU >> 1, ksBU = 2 * uint32_t(rows);
      const uint32_t slotU = uint32_t(a.wG) * kStageU;
      const int dil = a.dilation, wStages = a.wStages, drainN = a.drainN;
      int slot = 0, buf = 0, g = 0;
      uint32_t slotPh = 0, bufPh = 0, groupPar = 0, tilePar = 0, hb = 0;
      bool dead = false, ready = false;  // ready: the next round's weight slot is already known to be full
      long long wBf = 0, wHe = 0, wWf = 0, wLe = 0;
      const long long tStart = kProf ? clock64() : 0;
      const bool leader = electOne();
      for (int tile = tile0; leader && tile < numTiles && !dead; tile += tileStep) {
        for (int c = 0; c < nChunks16 && !dead; ++c) {
          if (!waitT(&bFull[buf], bufPh, wBf, SLEEP_MMA_NS)) {
            giveUp(4, 2);
            dead = true;
            break;
          }
          const uint64_t dBc = dB0 + uint32_t(buf) * bufU;
          int kk = 0;
          for (int gi = 0; gi < nTapGroups; ++gi) {
            const int gN = tgBase + (gi < tgExtra ? 1 : 0);
            if (!ready && !waitT(&wFull[slot], slotPh, wWf, SLEEP_MMA_NS)) {
              giveUp(4, 3);
              dead = true;
              break;
            }
            tcFenceAfter();
            const uint64_t dA = dA0 + uint32_t(slot) * slotU, dB = dBc + uint32_t(kk * dil);
            const uint32_t accHi = (kk | g) == 0 ? 0u : 1u, accLo = (kk | c) == 0 ? 0u : 1u;
            const bool needHi = (kk | g) == 0, needLo = (kk | c) == 0;  // Dhi drained / Dlo of the last tile folded
            const uint32_t aLo = uint32_t(dA), aHi = uint32_t(dA >> 32), bLo = uint32_t(dB), bHi = uint32_t(dB >> 32);
            // Rolled issue loops: the issuer's code between two MMAs has to be fetched and issued while at most one
            // MMA is in flight, so the loops are kept to a handful of instructions and exist once per order.
            const uint32_t tmemD = tmemHi + hb * NTK;
            auto issueHi = [&](uint32_t acc) {
              if constexpr (F16) {
                uint32_t aj = aLo, bj = bLo;
#pragma unroll 1
                for (int j = 0; j < gN; ++j, aj += kStageU, bj += uint32_t(dil), acc = 1u)
                  mmaF16W(tmemD, aj, aHi, bj, bHi, kIdesc, acc);
              } else {
                uint64_t dAh = dA, dBh = dB;
#pragma unroll 1
                for (int j = 0; j < gN; ++j, dAh += kStageU, dBh += uint32_t(dil), acc = 1u) {
                  mmaTf32(tmemD, dAh, dBh, kIdesc, acc);
                  mmaTf32(tmemD, dAh + kKsAU, dBh + ksBU, kIdesc, 1u);
                }
              }
            };
            auto issueLo = [&](uint32_t acc) {
              if constexpr (F16) {
                uint32_t aj = aLo, bj = bLo;
#pragma unroll 1
                for (int j = 0; j < gN; ++j, aj += kStageU, bj += uint32_t(dil), acc = 1u) {
                  mmaF16W(tmemLo, aj + kLoAU, aHi, bj, bHi, kIdesc, acc);
                  mmaF16W(tmemLo, aj, aHi, bj + loBU, bHi, kIdesc, 1u);
                }
              } else {
                uint64_t dAh = dA, dBh = dB;
#pragma unroll 1
                for (int j = 0; j < gN; ++j, dAh += kStageU, dBh += uint32_t(dil), acc = 1u) {
                  const uint64_t dAl = dAh + kLoAU, dBl = dBh + loBU;
                  mmaTf32(tmemLo, dAl, dBh, kIdesc, acc);
                  mmaTf32(tmemLo, dAh, dBl, kIdesc, 1u);
                  mmaTf32(tmemLo, dAl + kKsAU, dBh + ksBU, kIdesc, 1u);
                  mmaTf32(tmemLo, dAh + kKsAU, dBl + ksBU, kIdesc, 1u);
                }
              }
            };
            int nslot = slot + 1;
            uint32_t nph = slotPh;
            if (nslot == wStages) nslot = 0, nph ^= 1;
            const bool lastRound = c == nChunks16 - 1 && gi == nTapGroups - 1;  // of the tile
            if (needLo) {
              if (!waitT(loEmpty, tilePar ^ 1, wLe, SLEEP_MMA_NS)) {
                giveUp(4, 4);
                dead = true;
                break;
              }
              tcFenceAfter();
            }
            issueLo(accLo);
            // the tile's lo chain is complete: the epilogue folds Dlo under the hi MMAs of this last round
            if (lastRound) mmaCommit(loFull);
            if (needHi) {
              if (!waitT(&hiEmpty[hb], groupPar ^ 1, wHe, SLEEP_MMA_NS)) {
                giveUp(4, 1);
                dead = true;
                break;
              }
              tcFenceAfter();
            }
            issueHi(accHi);
            // first poll of the next slot's barrier, with the whole round queued behind it
            ready = mbarTestWait(&wFull[nslot], nph);
            mmaCommit(&wEmpty[slot]);  // weight slot free once the MMAs have read it
            kk += gN;
            slot = nslot, slotPh = nph;
          }
          if (dead) break;
          const bool lastChunk = c == nChunks16 - 1;
          // the hi chain of a drain group (drainN chunks, or what is left of the tile) is complete
          if (g == drainN - 1 || lastChunk) mmaCommit(&hiFull[hb]);
          mmaCommit(&bEmpty[buf]);  // activation buffer free once the MMAs have read it
          if (++buf == NB) buf = 0, bufPh ^= 1;
          if (++g == drainN || lastChunk) {
            g = 0;
            if (HB == 1 || hb == 1) groupPar ^= 1;
            if (HB == 2) hb ^= 1;
          }
        }
        tilePar ^= 1;
      }
      // This CTA's tensor work is queued: what follows it may set itself up under the tail. One lane's signal counts for the
      // CTA, so the 31 that do not issue have to wait here (us without this wait: [512, 4000] K = 11 88.1 -> 89.9, resblocks
      // [128, 19201] K = 3 / 11 128 / 166 -> 133 / 172).
      __syncwarp();
      dependentsLaunch();
      if (kProf)
        profAddIf(leader, 0, wBf), profAddIf(leader, 1, wHe), profAddIf(leader, 2, wWf), profAddIf(leader, 3, wLe),
            profAddIf(leader, 4, clock64() - tStart);
    }
  }

  tcFenceBefore();
  if constexpr (SPLIT != 0) {
    // No CTA leaves before what it sent has arrived: a second barrier, at which the epilogue warps have arrived in their branch, in
    // front of the finish phase (behind it 0.3 to 1 % more per forward).
    if (warp >= EPI_WARPS) clusterArrive(), clusterWait(), clusterArrive();
    clusterWait();
  }
  __syncthreads();
  if (warp == MMA_WARP) {
    tcFenceAfter();
    tmemDealloc(tmemBase, 512);
  }
}

// One packed element: tf32 split -> f32 hi or lo; f16 split -> f16 hi or lo (lo scaled by 2^11).
__device__ __forceinline__ float splitTf32(float v, int part) {
  const float h = tf32Round(v);
  return part == 0 ? h : v - h;
}
// A weight beyond the f16 range is clamped and reported through the status word (kStatusF16Weights): the caller then
// packs this weight in the tf32 format, which has the range of f32.
__device__ __forceinline__ __half splitF16(float v, int part, int* status) {
  if (part == 0 && fabsf(v) > 65504.f) atomicOr(status, kStatusF16Weights);
  const __half h = __float2half_rn(fminf(fmaxf(v, -65504.f), 65504.f));
  return part == 0 ? h : __float2half_rn((v - __half2float(h)) * kLoScale);
}

// Conv weight pack: stage (cb, c16, kk) = [hi | lo], each [16-byte K chunk][128 rows][chunk elements]
// (4 f32 or 8 f16 per chunk). Rows past Co are zero.
template <bool F16>
__global__ void packWeightsKernel(const float* __restrict__ w, void* __restrict__ wpOut, int co, int ci, int k,
                                  int* status) {
  constexpr int CE = F16 ? 8 : 4, NCH = KC / CE;  // elements per chunk, chunks per 16 channels
  const int nC16 = ci / KC;
  const int64_t n = int64_t((co + MT - 1) / MT) * nC16 * k * 2 * NCH * MT * CE;
  for (int64_t idx = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; idx < n; idx += int64_t(gridDim.x) * blockDim.x) {
    int64_t r = idx;
    const int e = int(r % CE);
    r /= CE;
    const int col = int(r % MT);
    r /= MT;
    const int kc = int(r % NCH);
    r /= NCH;
    const int part = int(r % 2);
    r /= 2;
    const int kk = int(r % k);
    r /= k;
    const int c16 = int(r % nC16);
    const int cb = int(r / nC16);
    const int row = cb * MT + col;
    const float v = row < co ? w[(int64_t(row) * ci + (c16 * KC + kc * CE + e)) * k + kk] : 0.f;
    if constexpr (F16) static_cast<__half*>(wpOut)[idx] = splitF16(v, part, status);
    else static_cast<float*>(wpOut)[idx] = splitTf32(v, part);
  }
}

// Polyphase ConvTranspose1d (K = 2 s, 2 p = s) on the same kernel: out[co, j s + r] = sum_c sum_tt Wr[r][co][c][tt] *
// leaky(x)[c, j + q_r - 1 + tt], q_r = (r + p) div s, is a 3-tap conv over the window (j - 1, j, j + 1) whose output rows
// are (channel, phase) pairs: window tap wt carries Wr[..][tt = wt - q_r] when that is 0 or 1 and zero otherwise (one
// of the three taps of every row is zero). Rows are grouped so that each epilogue warp (32 accumulator rows) owns
// CQ = 32 / s whole channels with all their phases (row = cl * s + r, the last 32 - CQ s rows are zero), which lets it
// write each channel's samples j s + r as one contiguous run. One 128-row block therefore holds 4 CQ channels.
template <bool F16>
__global__ void convtTcPackKernel(const float* __restrict__ w, void* __restrict__ wpOut, int ci, int co, int k, int s,
                                  int p, int* status) {
  constexpr int CE = F16 ? 8 : 4, NCH = KC / CE;
  const int nC16 = ci / KC, cq = 32 / s, cpb = 4 * cq;
  const int64_t n = int64_t((co + cpb - 1) / cpb) * nC16 * 3 * 2 * NCH * MT * CE;
  for (int64_t idx = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; idx < n; idx += int64_t(gridDim.x) * blockDim.x) {
    int64_t r = idx;
    const int e = int(r % CE);
    r /= CE;
    const int row = int(r % MT);
    r /= MT;
    const int kc = int(r % NCH);
    r /= NCH;
    const int part = int(r % 2);
    r /= 2;
    const int wt = int(r % 3);
    r /= 3;
    const int c16 = int(r % nC16);
    const int cb = int(r / nC16);
    const int q = row / 32, i = row % 32, cl = i / s, ph = i % s;
    const int o = (cb * 4 + q) * cq + cl, c = c16 * KC + kc * CE + e;
    const int tt = wt - (ph + p) / s;
    float v = 0.f;
    if (i < cq * s && o < co && (tt == 0 || tt == 1)) v = w[(int64_t(c) * co + o) * k + (ph + p) % s + (1 - tt) * s];
    if constexpr (F16) static_cast<__half*>(wpOut)[idx] = splitF16(v, part, status);
    else static_cast<float*>(wpOut)[idx] = splitTf32(v, part);
  }
}

}  // namespace

// Row floats of the second raw-input box (its 16-byte granularity): what a window of `rows` columns has beyond `cols`.
static int rawExt(int rows, int cols) { return rows <= cols ? 0 : (rows - cols + 3) & ~3; }

// Dynamic shared memory of one CTA and the weight ring it leaves room for: the largest taps-per-slot (<= TAP_GROUP)
// that still gives PREF_W_STAGES slots, else the deepest ring. Returns 0 when even single-tap slots do not fit.
static size_t convTcSmemBytes(int split, int64_t ci, int rows, int k, bool f16, int* wStages, int* wG) {
  const int tap = f16 ? Fmt<true>::W_STAGE_BYTES : Fmt<false>::W_STAGE_BYTES;
  const int actRow = f16 ? Fmt<true>::ACT_BYTES_PER_ROW : Fmt<false>::ACT_BYTES_PER_ROW;
  const int nb = f16 ? Fmt<true>::NB : Fmt<false>::NB;
  const int ext = rawExt(rows, split ? split : NT);
  SmemLayout base = smemLayout(split, int(ci), rows, ext, nb, 0, 0, actRow, tap);
  base.total -= base.par - base.w;  // without the split form's memory behind the MMAs, which the ring may lie in
  if (base.total > uint32_t(kMaxSmem)) return 0;
  const size_t avail = size_t(kMaxSmem) - base.total;
  // Large groups matter more than a deep ring (measured: two slots of four taps beat four slots of three, and at
  // K = 11 two slots of six beat three of four).
  int bestG = 0, bestWs = 0;
  for (int g = TAP_GROUP; g >= 1; --g) {
    const int groups = (k + g - 1) / g, gmax = (k + groups - 1) / groups;  // near-equal groups, the largest has gmax taps
    int ws = int(avail / (size_t(gmax) * tap));
    if (ws > MAX_W_STAGES) ws = MAX_W_STAGES;
    if (ws >= PREF_W_STAGES) {
      bestG = gmax, bestWs = ws;
      break;
    }
    if (ws >= MIN_W_STAGES && ws > bestWs) bestG = gmax, bestWs = ws;
  }
  if (bestG == 0) return 0;
  if (wStages) *wStages = bestWs;
  if (wG) *wG = bestG;
  const size_t total = smemLayout(split, int(ci), rows, ext, nb, bestWs, bestG, actRow, tap).total;
  return total <= size_t(kMaxSmem) ? total : 0;
}

// The hi chain between two drains holds at most MAX_CHAIN MMAs: whole chunks while they fit, and a chunk that alone
// has more (K > 24 with f16 halves, K > 12 with tf32 halves) goes to the CUDA-core kernel, so the chain (and the
// truncation drift it accumulates, about 1.5e-8 of the result per MMA: 3.7e-7 at 24) stays bounded.
static bool chainOk(int64_t k, bool f16) { return k * (f16 ? 1 : 2) <= MAX_CHAIN; }

bool convTcEligible(const ConvFusedParams& p, bool f16) {
  if (!(p.state != nullptr && p.x2 == nullptr && p.ci % KC == 0 && p.co >= 1 && p.ci >= KC && p.k >= 1 &&
        chainOk(p.k, f16) && (p.k - 1) * p.dilation <= MAX_HALO && p.lo >= 1 && p.padding <= (1 << 20) && p.ci <= 4096 &&
        p.l < (int64_t(1) << 30)))
    return false;
  return convTcSmemBytes(0, p.ci, NT + int((p.k - 1) * p.dilation), int(p.k), false, nullptr, nullptr) != 0;  // the larger format
}

int64_t convTcPackFloats(int64_t co, int64_t ci, int64_t k, bool f16) {
  return ((co + MT - 1) / MT) * (ci / KC) * k * (f16 ? Fmt<true>::W_STAGE_FLOATS : Fmt<false>::W_STAGE_FLOATS);
}

// Per-device constants, looked up once (the first call on a device must not be inside a stream capture).
struct DeviceInfo {
  int* status = nullptr;
  long long* prof = nullptr;
  int smCount = 0;
  int32_t clusters[MAX_SPLIT + 1] = {};  // [n]: clusters of n CTAs of the split form that the device holds at a time
};
// A cluster lives inside one GPC, of whose SMs a remainder is left over: 148 SMs hold 74 clusters of two, but 45 of three,
// 33 of four, 26 of five, 22 of six, 15 of seven or eight (one B200; which SMs are fused off differs).
static void countClusters(DeviceInfo& d) {
  const auto kernel = convTcKernel<1, false, 0, true, false, NTS, false>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem) != cudaSuccess) {
    cudaGetLastError();
    return;  // no split launches
  }
  for (int n = 2; n <= MAX_SPLIT; ++n) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(n), attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(unsigned(n) * unsigned(d.smCount)), cfg.blockDim = dim3(NTHREADS), cfg.dynamicSmemBytes = SPLIT_SMEM;
    cfg.attrs = attr, cfg.numAttrs = 1;
    int count = 0;
    if (cudaOccupancyMaxActiveClusters(&count, kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      count = 0;
    }
    d.clusters[n] = count;
  }
}
static int deviceInfo(const DeviceInfo** out) {
  static DeviceInfo info[64];
  int dev = 0;
  cudaGetDevice(&dev);
  LKC_REQUIRE(dev >= 0 && dev < 64, "conv (tensor-core): device index out of range");
  DeviceInfo& d = info[dev];
  if (!d.status) {
    int* ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), gTcStatus);
    if (e != cudaSuccess) return failCuda("conv (tensor-core): cudaGetSymbolAddress", e);
    e = cudaDeviceGetAttribute(&d.smCount, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return failCuda("conv (tensor-core): cudaDeviceGetAttribute", e);
    long long* pp = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&pp), gTcProf);
    if (e != cudaSuccess) return failCuda("conv (tensor-core): cudaGetSymbolAddress", e);
    d.prof = pp;
    countClusters(d);
    d.status = ptr;
  }
  *out = &d;
  return 0;
}

int convTcPack(const float* w, float* wp, int64_t co, int64_t ci, int64_t k, bool f16, cudaStream_t s) {
  LKC_REQUIRE(ci % KC == 0 && co > 0 && ci > 0 && k >= 1 && k <= 64,
              "conv1d_tc_pack_f32_cuda: needs Ci % 16 == 0, 1 <= K <= 64");
  const DeviceInfo* d = nullptr;
  if (int rc = deviceInfo(&d)) return rc;
  const int64_t n = convTcPackFloats(co, ci, k, f16) * (f16 ? 2 : 1);  // packed elements
  const int blocks = static_cast<int>(ceilDiv(n, 256) > 4096 ? 4096 : ceilDiv(n, 256));
  if (f16) packWeightsKernel<true><<<blocks, 256, 0, s>>>(w, wp, int(co), int(ci), int(k), d->status);
  else packWeightsKernel<false><<<blocks, 256, 0, s>>>(w, wp, int(co), int(ci), int(k), d->status);
  return launched("conv1d_tc_pack_f32_cuda");
}

// ---- tensor maps (cuTensorMapEncodeTiled, looked up through the runtime: the library does not link libcuda)

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encodeTiled() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    cudaGetLastError();
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}
static bool gTmaEnabled = true;  // lkc_set_conv_io: false forces the 4-byte route (A/B testing)

// Map of an f32 [rowsC, cols] tensor with row pitch `pitch` floats; box = boxCols x boxRows. False when the tensor's
// rows are not 16-byte aligned (or the driver entry point is missing): the caller then takes the 4-byte route.
static bool makeMap(CUtensorMap* map, const float* base, int64_t rowsC, int64_t cols, int64_t pitch, int boxCols,
                    int boxRows, bool swizzle128) {
  if (!gTmaEnabled || !base || (reinterpret_cast<uintptr_t>(base) & 15) || (pitch & 3) || pitch < cols || cols < 1 ||
      rowsC < 1 || cols >= (int64_t(1) << 31))
    return false;
  EncodeTiledFn fn = encodeTiled();
  if (!fn) return false;
  const cuuint64_t dims[2] = {cuuint64_t(cols), cuuint64_t(rowsC)};
  const cuuint64_t strides[1] = {cuuint64_t(pitch) * 4};
  const cuuint32_t box[2] = {cuuint32_t(boxCols), cuuint32_t(boxRows)};
  const cuuint32_t elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int convTcSetIo(int mode) {
  LKC_REQUIRE(mode == 0 || mode == 1, "set_conv_io: mode must be 0 (TMA where rows are aligned) or 1 (4-byte route only)");
  gTmaEnabled = mode == 0;
  return 0;
}

template <int ACT, bool PARTIAL, int TS, bool F16, bool TMAO, int SPLIT, bool NARROW>
static int launchTc5(const TcArgs& a, const TcMaps& m, int grid, size_t smem, cudaStream_t s) {
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  const auto kernel = convTcKernel<ACT, PARTIAL, TS, F16, TMAO, SPLIT, NARROW>;
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    if (e != cudaSuccess) return failCuda("conv (tensor-core): cudaFuncSetAttribute", e);
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cfg.gridDim = dim3(unsigned(grid)), cfg.blockDim = dim3(NTHREADS), cfg.dynamicSmemBytes = smem, cfg.stream = s, cfg.attrs = attr;
  if (a.early) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (SPLIT) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = unsigned(a.split), attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, a, m.x, m.ext, m.res, m.out);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return failCuda("conv (tensor-core)", e);
  }
  return launched("conv (tensor-core)");
}

template <int ACT, bool PARTIAL, int TS, bool F16, bool TMAO, int SPLIT>
static int launchTc4(const TcArgs& a, const TcMaps& m, int grid, size_t smem, cudaStream_t s) {
  if constexpr (F16 && SPLIT == 0) {
    if (a.tileCols < NT) return launchTc5<ACT, PARTIAL, TS, F16, TMAO, SPLIT, true>(a, m, grid, smem, s);
  }
  return launchTc5<ACT, PARTIAL, TS, F16, TMAO, SPLIT, false>(a, m, grid, smem, s);
}

template <int ACT, bool PARTIAL, int TS, bool F16>
static int launchTc3(const TcArgs& a, const TcMaps& m, int grid, size_t smem, cudaStream_t s) {
  if constexpr (F16 || (ACT == 0 && TS == 0)) {  // the second half of a split tile handles every Co and alignment
    if constexpr (TS == 0) {
      if (a.split && a.tileCols == NTS2) return launchTc4<ACT, false, TS, F16, false, NTS2>(a, m, grid, smem, s);
    }
    if (a.split) return launchTc4<ACT, false, TS, F16, false, NTS>(a, m, grid, smem, s);
  }
  if constexpr (TS == 0 && !PARTIAL) {
    if (a.tmaOut) return launchTc4<ACT, PARTIAL, TS, F16, true, 0>(a, m, grid, smem, s);
  }
  return launchTc4<ACT, PARTIAL, TS, F16, false, 0>(a, m, grid, smem, s);
}

template <int ACT, bool PARTIAL, int TS = 0>
static int launchTc2(const TcArgs& a, const TcMaps& m, bool f16, int grid, size_t smem, cudaStream_t s) {
  return f16 ? launchTc3<ACT, PARTIAL, TS, true>(a, m, grid, smem, s) : launchTc3<ACT, PARTIAL, TS, false>(a, m, grid, smem, s);
}

template <int ACT>
static int launchTc(const TcArgs& a, const TcMaps& m, bool f16, int grid, size_t smem, cudaStream_t s) {
  return a.co % MT == 0 ? launchTc2<ACT, false>(a, m, f16, grid, smem, s) : launchTc2<ACT, true>(a, m, f16, grid, smem, s);
}

static bool gProfileOn = false;

// Profiling counters of the tensor-core kernel (cycles, summed over CTAs and launches since the last reset; one
// representative warp per role): [0..4] MMA warp: wait activations, wait Dhi drained, wait weights, wait Dlo folded,
// total; [5..9] epilogue warp 0: wait Dhi, wait Dlo, residual preload, final phase, total; [10..13] producer warp 0:
// wait buffer free, wait raw window, transform, total; [14..15] weight producer: wait stage free, total.
int convTcProfile(int enable, long long* out16) {
  LKC_REQUIRE(kProf, "conv1d_tc_profile: the library was built without -DLKC_TC_PROF=1");
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return failCuda("conv1d_tc_profile: cudaDeviceSynchronize", e);
  gProfileOn = enable != 0;
  if (out16) {
    e = cudaMemcpyFromSymbol(out16, gTcProf, sizeof(long long) * 16);
    if (e != cudaSuccess) return failCuda("conv1d_tc_profile", e);
  }
  static const long long zeros[16] = {};
  e = cudaMemcpyToSymbol(gTcProf, zeros, sizeof zeros);
  if (e != cudaSuccess) return failCuda("conv1d_tc_profile", e);
  return 0;
}

// CTAs per tile: 0 = the persistent form. The split form is taken where at least two CTAs per 128-column tile fit on the
// launch's share of the SMs and all its clusters, by themselves, are resident at a time (clusters[n], see countClusters):
// there the time is one tile's chain of 16-channel chunks plus about 7 us of fixed cost (launch, first loads, exchange), and
// the chain shrinks with every CTA. With one CTA per tile it gains little over 256-column tiles (an M128 N128 MMA takes about
// 0.8 of the time of an N256 one here) and doubles the weight traffic; with a second wave it loses: [128, 6144] K = 11,
// 48 clusters of three where 45 fit, 36 us against 30 us unsplit and 21 us with two CTAs per tile.
// Measured (us, persistent -> split): [256, 240] K = 11: 52 -> 15; [256, 1210] K = 7: 49 -> 17; [128, 1441] K = 3: 29 -> 12;
// [1104 -> 1024, 61] K = 3: 130 -> 19; [256, 3200] K = 11, two CTAs per tile: 52 -> 30.
// Of the convs with tf32 halves the pointwise ones without an activation split (the decoder's shortcuts).
static bool splits(bool f16, int64_t k, Act act) { return f16 || (k == 1 && act == Act::None); }
static int splitFor(bool can, int ci, int64_t lo, int64_t coBlocks, int sms, const int32_t* clusters) {
  if (!can) return 0;
  const int n = ci / KC;
  const int64_t tiles = ceilDiv(lo, NTS) * coBlocks;
  for (int sp = int(std::min<int64_t>(std::min(MAX_SPLIT, n), sms / tiles)); sp >= 2; --sp) {
    const int serial = (n + sp - 1) / sp, ctas = (n + serial - 1) / serial;  // no more CTAs than shorten the longest run
    if (tiles <= clusters[ctas]) return ctas;
  }
  return 0;
}

int convTcSplitRule(int64_t ci, int64_t co, int64_t lo, int sms, const int32_t* clusters) {
  return splitFor(true, int(ci), lo, ceilDiv(co, MT), sms, clusters);
}

int convTcDevice(int* sms, const int32_t** clusters) {
  const DeviceInfo* d = nullptr;
  if (int rc = deviceInfo(&d)) return rc;
  *sms = d->smCount, *clusters = d->clusters;
  return 0;
}

// Columns per tile of the persistent form, for a launch that may spread over smPercent of the device's SMs.
// Alone, the launch's time is the rounds of tiles that its busiest SM runs times a tile's time, which is about that of its
// columns plus 48 more: a narrower tile pays where it takes fewer SM-columns in whole rounds.
// Beside other launches the columns all together count, of which wide tiles cost fewer, unless there are few: then the
// narrowest tiles that find room in one round of the launch's share shorten its chain.
// Widths other than NT (a form of the kernel with f16 halves) leave chunk statistics per 32 columns, which the caller has to
// take (fineOk).
static int tileColsFor(bool fineOk, int64_t lo, int64_t coBlocks, int sms, int smPercent) {
  int best = NT;
  if (!fineOk) return best;
  int64_t cost = ceilDiv(ceilDiv(lo, NT) * coBlocks, sms) * (NT + 48);
  for (int w = NT - 32; w >= 160; w -= 32) {
    const int64_t tiles = ceilDiv(lo, w) * coBlocks, c = ceilDiv(tiles, sms) * (w + 48);
    if (smPercent < 100 ? tiles <= int64_t(sms) * smPercent / 100 : c < cost) best = w, cost = c;
  }
  return best;
}

int convTcTileRule(int64_t co, int64_t lo, int sms, int smPercent) { return tileColsFor(true, lo, ceilDiv(co, MT), sms, smPercent); }

// Columns of a split tile of a conv. Of a row of up to 64, half of a 128-column tile's MMA time, partial tile, exchange and
// output are padding: the decoder at F = 61 244 -> 215 us. Tiles of 64 for longer rows lose more to their number (fewer CTAs per
// tile, each reading more weights) than their shorter exchange gives: T = 24 320 -> 352, F = 100 244 -> 254.
int convTcSplitCols(int64_t lo) { return lo <= NTS2 ? NTS2 : NTS; }

// The form of a launch. Everybody who has to know it asks here: the launch itself, and the whole-model calls, which give split
// convs chunk statistics and read the statistics of narrow tiles.
struct TcForm {
  int split, tileCols;
  bool pair;  // tiles of CTA pairs (conv_pair.cu), 160 columns wide or 128
};
static TcForm formFor(const DeviceInfo& d, bool canSplit, bool fineOk, bool conv, int64_t ci, int64_t lo, int64_t coBlocks,
                      int smPercent) {
  TcForm f;
  f.pair = false;
  f.split = splitFor(canSplit, int(ci), lo, coBlocks, d.smCount * smPercent / 100, d.clusters);
  f.tileCols = f.split ? (conv ? convTcSplitCols(lo) : NTS) : tileColsFor(fineOk, lo, coBlocks, d.smCount, smPercent);
  return f;
}
// Columns per (mean, M2) pair that a launch of this form leaves.
static int statColsOf(int split, int tileCols) { return split || tileCols == NT || tileCols == NTS ? 128 : 32; }

static bool rowsAligned(const float* p, int64_t pitch) { return ((reinterpret_cast<uintptr_t>(p) | uintptr_t(pitch * 4)) & 15) == 0; }
static int pairRows(int w, int64_t k, int64_t dilation, int64_t padding) {  // staged window columns of a CTA
  return w / 2 + int((k - 1) * dilation) + int(-padding & 3);
}
// Columns per tile of the pair form (conv_pair.cu), for a conv with f16 halves that is not split and whose rows the TMA unit can
// address, or 0 where tiles of oneCols columns of one CTA are the faster ones: 160, or 128 where the statistics have to be of 128.
// Pairs stage half of the window columns and have finer tiles, but theirs come in whole rounds too, and their set-up takes longer.
// Alone, the clocks of both forms decide: a launch's, a tile's, and per chunk the longest of staging, MMAs and, for pairs, refilling
// the weight slots (a slot of seven taps takes longer than the MMAs of the other one). The constants are fitted to launches timed in
// both forms, Ci 16 to 1104, Co 256 to 1024, K 1 to 16, L 1600 to 60000. From 128 channels on (1848 launches): the geometric mean of
// the times is 0.814 of that without pairs (0.812 if the better form were known; 0.826 with pairs wherever they can run), at worst
// 1.024 (1.44), up to K = 11 1.008. us, one CTA -> pairs: [256, 20800] K = 3 / 7 / 11 54 -> 40, 68 -> 57, 93 -> 72;
// [256, 8000] 29 -> 17, 35 -> 23, 48 -> 29; not taken: a resblock of [256, 12000], 126 tiles of 192 columns or 75 of pairs where 74 run
// at a time, K = 7 / 11 221 -> 267, 285 -> 356; [512, 4800] K = 7 36 -> 37. A launch behind its adain_affine starts under it either way, which
// makes two rounds of pairs 5000 clocks cheaper (resblock [256, 14000] K = 3 197 -> 186). With few channels memory and set-up are the time,
// which the clocks do not know ([16, 9600] K = 1 9.3 -> 12.4, [64, 60000] 79 -> 89): pairs have to be 5 % faster by them then, in
// at most three rounds (1148 launches: 0.957, at worst 1.041, three of [64, 30000]; 1.018 and 1.47 wherever they can run).
// Beside other launches the SM time of all tiles together counts, which is that of 256-column tiles of one CTA; there pairs are taken for
// launches of one round. us per generator forward as a graph, without pairs / those of one round of the launch's share / of the device:
// T = 260 827 / 796 / 796, T = 320 866 / 809 / 809, T = 400 913 / 887 / 887, T = 480 1043 / 1021 / 992, T = 640 1328 / 1333 / 1320,
// T = 800 1497 / 1497 / 1472; with pairs of two rounds T = 2080 3680 / 3740.
static int pairColsFor(bool fineOk, int64_t ci, int64_t co, int64_t lo, int64_t k, int64_t dilation, int64_t padding, Act act, int oneCols,
                       bool behindAffine, int smPercent, int sms, const int32_t* clusters) {
  if (co % (2 * MT) || clusters[2] < 1) return 0;
  const int w = fineOk ? 160 : 128, rows = pairRows(w, k, dilation, padding);
  int nb, nRaw, ws, wG;
  if (pairSmem(int(ci), rows, (rows + 3) & ~3, int(k), &nb, &nRaw, &ws, &wG) == 0) return 0;
  const int64_t rounds = ceilDiv(ceilDiv(lo, w) * (co / (2 * MT)), clusters[2]), n = ci / KC;
  if (smPercent < 100) return rounds == 1 ? w : 0;
  const int64_t groups = ceilDiv(k, wG), mma = 3 * k * w / 2 + 172 * groups;
  const int64_t stage = 840 + (act == Act::Snake ? 14 * rows / 5 : 0), refill = (mma + 1270 * groups + 112 * k) / ws;
  const int64_t pair = (behindAffine ? 7000 : 12000) + rounds * (5450 + n * std::max(std::max(stage, mma), refill));
  const int64_t oneStage = 1460 + (act == Act::Snake ? 81 : 20) * (oneCols + (k - 1) * dilation) / 20;
  const int64_t oneMma = 3 * k * oneCols / 2 + 455 * ceilDiv(k, TAP_GROUP);
  const int64_t one = 11700 + ceilDiv(ceilDiv(lo, oneCols) * ceilDiv(co, MT), sms) * (1550 + 22 * oneCols + n * std::max(oneStage, oneMma));
  return (n < 8 ? rounds <= 3 && pair * 21 < one * 20 : pair * 101 < one * 100) ? w : 0;
}
int convTcPairRule(int64_t ci, int64_t co, int64_t lo, int64_t k, int64_t dilation, int64_t padding, Act act, bool fineOk,
                   bool behindAffine, int smPercent, int sms, const int32_t* clusters) {
  const int64_t blocks = ceilDiv(co, MT);
  if ((k - 1) * dilation > MAX_HALO || splitFor(true, int(ci), lo, blocks, sms * smPercent / 100, clusters)) return 0;
  return pairColsFor(fineOk, ci, co, lo, k, dilation, padding, act, tileColsFor(fineOk, lo, blocks, sms, smPercent), behindAffine, smPercent,
                     sms, clusters);
}
static int formOf(const ConvFusedParams& p, bool f16, TcForm* f) {
  const DeviceInfo* d = nullptr;
  if (int rc = deviceInfo(&d)) return rc;
  const bool fineOk = f16 && (p.fineStats || !p.stats);
  *f = formFor(*d, splits(f16, p.k, p.act), fineOk, true, p.ci, p.lo, ceilDiv(p.co, MT), p.smPercent);
  if (f->split || !f16 || !gTmaEnabled || !encodeTiled() || !rowsAligned(p.x, p.xPitch ? p.xPitch : p.l) ||
      !rowsAligned(p.out, p.outPitch ? p.outPitch : p.lo) || (p.residual && !rowsAligned(p.residual, p.resPitch ? p.resPitch : p.lo)))
    return 0;
  if (const int w = pairColsFor(fineOk, p.ci, p.co, p.lo, p.k, p.dilation, p.padding - p.xOrigin, p.act, f->tileCols, p.behindAffine,
                                p.smPercent, d->smCount, d->clusters))
    f->pair = true, f->tileCols = w;
  return 0;
}

enum class Start { BehindAffine, Urgent, Patient };  // see ConvFusedParams
static Start startOf(const ConvFusedParams& p) { return p.behindAffine ? Start::BehindAffine : p.urgent ? Start::Urgent : Start::Patient; }

// Geometry and tensor maps of the pair form. False: a map could not be made, and the launch takes the form of one CTA that leaves
// the same statistics.
static bool finishPair(TcArgs& a, TcMaps& m, const DeviceInfo& d, Start start, int smPercent, int* grid, size_t* smem) {
  a.delta = -a.padding & 3;
  a.rows = pairRows(a.tileCols, a.k, a.dilation, a.padding), a.ext = (a.rows + 3) & ~3;  // ext: columns of a raw buffer
  int nb = 0;
  *smem = pairSmem(a.ci, a.rows, a.ext, a.k, &nb, &a.nRaw, &a.wStages, &a.wG);
  constexpr int tapRows = Fmt<true>::W_STAGE_BYTES / 1024;  // the pack as rows of 1 KB
  const int64_t wRows = int64_t(a.co / MT) * (a.ci / KC) * a.k * tapRows;
  if (*smem == 0 || wRows >= (int64_t(1) << 30) || !makeMap(&m.x, a.x, a.ci, a.l, a.xPitch, a.ext, KC, false) ||
      !makeMap(&m.out, a.out, a.co, a.lo, a.outPitch, BOX, BOX, true) ||
      (a.residual && !makeMap(&m.res, a.residual, a.co, a.lo, a.resPitch, BOX, BOX, true)) ||
      !makeMap(&m.w, a.wp, wRows, 256, 256, 256, a.wG * tapRows, false) ||
      (a.k % a.wG && !makeMap(&m.w1, a.wp, wRows, 256, 256, 256, (a.wG - 1) * tapRows, false)))
    return false;
  a.tmaIn = a.tmaOut = 1, a.nb = nb;
  a.numCoBlk = a.co / (2 * MT);
  const int tiles = a.numTTiles * a.numCoBlk;
  *grid = 2 * std::min(tiles, d.clusters[2]);
  a.early = start == Start::BehindAffine || (smPercent == 100 && tiles <= d.clusters[2]);
  return true;
}

// Launch geometry and tensor maps shared by the conv and ConvTranspose entry points.
static int finishArgs(TcArgs& a, TcMaps& m, bool f16, TcForm form, bool boxesOk, Start start, int smPercent, int* grid, size_t* smem) {
  const DeviceInfo* d = nullptr;
  if (int rc = deviceInfo(&d)) return rc;
  a.split = form.split, a.tileCols = form.tileCols, a.pair = form.pair;
  LKC_REQUIRE(!a.statsIn || a.split, "conv (tensor-core): only the split form takes chunk statistics");
  const int nt = a.split ? a.tileCols : NT;  // staged columns of the first box
  if (a.stats && statColsOf(a.split, a.tileCols) == 32) a.nchunks = ceilDiv(a.lo, 32);
  a.numTTiles = int(ceilDiv(a.lo, a.tileCols));
  // TMA routes: tensors whose rows are 16-byte aligned. A map that is not used still has to be a valid kernel
  // argument: it stays zero-filled and is never dereferenced.
  std::memset(&m, 0, sizeof m);
  a.nb = f16 ? Fmt<true>::NB : Fmt<false>::NB;
  a.status = d->status;
  a.prof = (kProf && gProfileOn) ? d->prof : nullptr;
  // Dhi is drained into the f32 running sums after as many whole chunks as fit in the longest chain of MMAs.
  const int perChunk = a.k * (f16 ? 1 : 2);
  const int n = (!f16 && a.k == 1 ? MAX_CHAIN_POINT32 : MAX_CHAIN) / perChunk;
  a.drainN = n < 1 ? 1 : n;
  if (a.pair) {
    const int coBlk = a.numCoBlk;
    if (finishPair(a, m, *d, start, smPercent, grid, smem)) return 0;
    std::memset(&m, 0, sizeof m);
    a.pair = 0, a.numCoBlk = coBlk, a.nb = Fmt<true>::NB;
    if (a.tileCols == NTS) a.tileCols = NT, a.numTTiles = int(ceilDiv(a.lo, NT));
  }
  a.tmaIn = makeMap(&m.x, a.x, a.ci, a.l, a.xPitch, nt, KC, false) ? 1 : 0;
  auto layOut = [&] {
    a.delta = a.tmaIn ? -a.padding & 3 : 0;  // tiles start on multiples of 4 columns
    const int need = a.tileCols + (a.k - 1) * a.dilation + a.delta;
    a.mainRows = std::min(nt, (need + 63) & ~63);
    a.rows = std::max(need, a.mainRows);
    a.ext = rawExt(a.rows, nt);
    *smem = convTcSmemBytes(a.split ? nt : 0, a.ci, a.rows, a.k, f16, &a.wStages, &a.wG);
  };
  layOut();
  if (*smem == 0 && a.tmaIn) a.tmaIn = 0, layOut();  // no room for the rows in front of the window: the 4-byte route has none
  if (a.tmaIn && a.ext)
    LKC_REQUIRE(makeMap(&m.ext, a.x, a.ci, a.l, a.xPitch, a.ext, KC, false), "conv (tensor-core): tensor map of the input");
  LKC_REQUIRE(*smem != 0, "conv (tensor-core): window too large");
  if (a.split && *smem < SPLIT_SMEM) *smem = SPLIT_SMEM;
  const int tiles = a.numTTiles * a.numCoBlk;
  *grid = a.split ? tiles * a.split : (tiles < d->smCount ? tiles : d->smCount);
  // A launch of one round starts as the SMs come free and sets itself up under the end of the one before it: 3 us of a split
  // launch's 14. CTAs that wait hold SMs that a ready launch of another stream could use, so beside other launches this is for the
  // split ones (in a branch that nobody waits for soon, those of few tiles: T = 64 425 -> 436 with the second noise branch early),
  // and for any behind its adain_affine, which lets it start only when the conv before has ended. us per generator forward as a
  // graph, split ones of few tiles / all split ones / behind adain_affine too: T = 121 544 / - / 531 and with all split ones 509,
  // T = 140 580 -> 560, T = 160 638 -> 627, T = 200 682 / 661 / 647; without split ones T = 320 809 -> 761, T = 480 990 -> 966,
  // T = 640 1317 -> 1271, T = 800 1470 -> 1450. Decoder F = 320 / 384 308 -> 300, 313 -> 304.
  // A share of 100 % counts as alone, which the decoder's launches above 384 frames say as well, though its shortcuts run beside
  // its main convs (see there).
  a.early = start == Start::BehindAffine ? 1
            : smPercent == 100           ? tiles <= d->smCount
                                         : a.split && (start == Start::Urgent || tiles * 8 <= d->smCount);
  a.tmaOut = 0;
  if (boxesOk && a.co % MT == 0 && makeMap(&m.out, a.out, a.co, a.lo, a.outPitch, BOX, BOX, true) &&
      (!a.residual || makeMap(&m.res, a.residual, a.co, a.lo, a.resPitch, BOX, BOX, true)))
    a.tmaOut = 1;
  return 0;
}

bool convTcSplits(const ConvFusedParams& p, bool f16) {
  TcForm f;
  return formOf(p, f16, &f) == 0 && f.split != 0;
}

int convTcStatCols(const ConvFusedParams& p, bool f16) {
  TcForm f;
  return formOf(p, f16, &f) == 0 ? statColsOf(f.split, f.tileCols) : 128;
}

static int convTcLaunch(const ConvFusedParams& p, const float* wp, bool f16, cudaStream_t s);

// Columns of the first launch of a conv that goes in two, or 0. Alone, a conv whose tiles fill some rounds of the device and a part
// of one more lasts as if that were full. Where so few columns are over that they can be split over the CTAs of clusters they are a
// launch of their own, if that saves more MMA clocks (half a column's width each, three to a tap and chunk) than the split form's
// fixed cost and a second launch's, at most 24,000 (12 us). The rounds are those of 256-column tiles in both forms of whole tiles, so
// that rows of every alignment give the same bits; two rounds of pairs have as many columns where pairs fill the device (where clusters
// of two leave SMs over, pairColsFor sees the rounds that they take). Statistics per 32 columns leave no choice: a split tile has one
// pair.
// Measured (us, one launch -> two): [512, 9500] K = 7: 96 -> 79; [512, 19200] K = 7: 163 -> 156, K = 11: 233 -> 219;
// [256, 19201] K = 11: 99 -> 67; [128, 38000] K = 11: 53 -> 41, [128, 40000] 57 -> 46. Unchanged by the rule: [512, 19200] K = 3 (105).
int64_t convTcRoundsRule(int64_t ci, int64_t co, int64_t lo, int64_t k, int sms, const int32_t* clusters) {
  const int64_t blocks = ceilDiv(co, MT), n = ci / KC;
  const int64_t cols = ceilDiv(lo, NT) * blocks / sms * sms / blocks * NT;
  if (cols < 1 || cols >= lo || cols > (1 << 24)) return 0;
  const int split = splitFor(true, int(ci), lo - cols, blocks, sms, clusters);
  if (!split) return 0;
  const int64_t saved = 3 * k * (n * (blocks % 2 ? NT : NTS) / 2 - ceilDiv(n, split) * NTS / 2);  // pairs: by their tiles
  return saved > 24000 ? cols : 0;
}
static int64_t fullRounds(const ConvFusedParams& p, bool f16, const TcForm& form) {
  const DeviceInfo* d = nullptr;
  if (deviceInfo(&d) || p.smPercent < 100 || !p.stats || p.fineStats || form.split || !splits(f16, p.k, p.act)) return 0;
  return convTcRoundsRule(p.ci, p.co, p.lo, p.k, d->smCount, d->clusters);
}

int convTc(const ConvFusedParams& p, const float* wp, bool f16, cudaStream_t s) {
  TcForm form;
  if (int rc = formOf(p, f16, &form)) return rc;
  const int64_t cols = fullRounds(p, f16, form);
  if (cols == 0) return convTcLaunch(p, wp, f16, s);
  ConvFusedParams first = p;
  first.xPitch = p.xPitch ? p.xPitch : p.l, first.resPitch = p.resPitch ? p.resPitch : p.lo;
  first.outPitch = p.outPitch ? p.outPitch : p.lo, first.statsStride = p.statsStride ? p.statsStride : statChunks(p.lo);
  ConvFusedParams rest = first;
  first.lo = cols;
  rest.lo = p.lo - cols, rest.xOrigin = p.xOrigin + cols, rest.out = p.out + cols;
  if (p.residual) rest.residual = p.residual + cols;
  if (p.stats) rest.stats = p.stats + 2 * (cols / NTS);
  if (int rc = convTcLaunch(first, wp, f16, s)) return rc;
  return convTcLaunch(rest, wp, f16, s);
}

static int convTcLaunch(const ConvFusedParams& p, const float* wp, bool f16, cudaStream_t s) {
  TcArgs a;
  TcMaps m;
  a.x = p.x, a.wp = wp, a.bias = p.bias, a.affine = p.affine, a.alpha = p.alpha, a.residual = p.residual;
  a.out = p.out, a.stats = p.stats;
  a.ci = int(p.ci), a.co = int(p.co), a.k = int(p.k), a.dilation = int(p.dilation), a.padding = int(p.padding);
  a.l = p.l, a.lo = p.lo, a.nchunks = p.statsStride ? p.statsStride : statChunks(p.lo), a.padLeft = 0;
  a.padding = int(p.padding - p.xOrigin);  // window row 0 of output column t is x column t - padding + xOrigin
  a.validLo = p.validLo, a.validHi = p.validHi < 0 ? p.l : p.validHi;
  a.xPitch = p.xPitch ? p.xPitch : p.l, a.resPitch = p.resPitch ? p.resPitch : p.lo;
  a.outPitch = p.outPitch ? p.outPitch : p.lo;
  a.slope = p.slope, a.outScale = p.outScale;
  a.statsIn = p.statsIn, a.gb = p.gb, a.eps = p.eps;
  const int64_t tTiles = ceilDiv(p.lo, NTS);
  const int64_t coBlk = ceilDiv(p.co, MT);  // output channels past Co are zero rows of the pack and never stored
  LKC_REQUIRE(tTiles * coBlk < (1 << 30), "conv (tensor-core): too many tiles");
  a.numCoBlk = int(coBlk);
  int grid = 0;
  size_t smem = 0;
  TcForm form;
  if (int rc = formOf(p, f16, &form)) return rc;
  if (int rc = finishArgs(a, m, f16, form, true, startOf(p), p.smPercent, &grid, &smem)) return rc;
  if (a.pair) return convPair(a, m, p.act, grid, smem, s);
  switch (p.act) {
    case Act::None: return launchTc<0>(a, m, f16, grid, smem, s);
    case Act::Snake: return launchTc<1>(a, m, f16, grid, smem, s);
    case Act::Leaky: return launchTc<2>(a, m, f16, grid, smem, s);
  }
  return fail("conv (tensor-core): bad activation");
}

// ---- polyphase ConvTranspose1d on the tensor-core kernel

bool convtTcEligible(int64_t ci, int64_t co, int64_t k, int64_t stride, int64_t padding) {
  return (stride == 6 || stride == 10) && k == 2 * stride && 2 * padding == stride && ci % KC == 0 && ci >= KC &&
         ci <= 4096 && co >= 1 && convTcSmemBytes(0, ci, NT + 2, 3, false, nullptr, nullptr) != 0;
}

int64_t convtTcPackFloats(int64_t ci, int64_t co, int64_t stride, bool f16) {
  const int64_t cpb = 4 * (32 / stride);
  return ceilDiv(co, cpb) * (ci / KC) * 3 * (f16 ? Fmt<true>::W_STAGE_FLOATS : Fmt<false>::W_STAGE_FLOATS);
}

int convtTcPack(const float* w, float* wp, int64_t ci, int64_t co, int64_t k, int64_t stride, int64_t padding,
                bool f16, cudaStream_t s) {
  LKC_REQUIRE(convtTcEligible(ci, co, k, stride, padding),
              "convt_tc_pack_f32_cuda: needs stride 6 or 10, K = 2 stride, 2 padding = stride, Ci % 16 == 0");
  const DeviceInfo* d = nullptr;
  if (int rc = deviceInfo(&d)) return rc;
  const int64_t n = convtTcPackFloats(ci, co, stride, f16) * (f16 ? 2 : 1);
  const int blocks = static_cast<int>(ceilDiv(n, 256) > 4096 ? 4096 : ceilDiv(n, 256));
  if (f16)
    convtTcPackKernel<true><<<blocks, 256, 0, s>>>(w, wp, int(ci), int(co), int(k), int(stride), int(padding), d->status);
  else
    convtTcPackKernel<false><<<blocks, 256, 0, s>>>(w, wp, int(ci), int(co), int(k), int(stride), int(padding), d->status);
  return launched("convt_tc_pack_f32_cuda");
}

int convtTc(const ConvtParams& p, const float* wp, bool f16, cudaStream_t s) {
  TcArgs a;
  TcMaps m;
  a.x = p.x, a.wp = wp, a.bias = p.bias, a.affine = nullptr, a.alpha = nullptr, a.residual = p.res;
  a.out = p.out, a.stats = nullptr;
  // x holds haloLeft + l + haloRight columns; output (input-rate) column j reads x columns j + haloLeft + {-1, 0, 1}
  const int64_t lx = p.haloLeft + p.l + p.haloRight;
  a.ci = int(p.ci), a.co = int(p.co), a.k = 3, a.dilation = 1, a.padding = int(1 - p.haloLeft);
  const int64_t lo = p.l * p.stride + p.padLeft;
  a.l = lx, a.lo = p.l, a.nchunks = 0, a.padLeft = int(p.padLeft);
  a.validLo = 0, a.validHi = lx;
  a.xPitch = p.xPitch ? p.xPitch : lx, a.resPitch = p.resPitch ? p.resPitch : lo, a.outPitch = p.outPitch ? p.outPitch : lo;
  a.slope = p.slope, a.outScale = 1.f;
  a.statsIn = nullptr, a.gb = nullptr, a.eps = 0.f;
  const int64_t tTiles = ceilDiv(p.l, NTS), coBlk = ceilDiv(p.co, 4 * (32 / p.stride));
  LKC_REQUIRE(tTiles * coBlk < (1 << 30) && p.l < (int64_t(1) << 30), "conv_transpose1d_poly (tensor-core): too many tiles");
  a.numCoBlk = int(coBlk);
  int grid = 0;
  size_t smem = 0;
  const DeviceInfo* d = nullptr;
  if (int rc = deviceInfo(&d)) return rc;
  const TcForm form = formFor(*d, f16, f16, false, p.ci, p.l, coBlk, p.smPercent);
  if (int rc = finishArgs(a, m, f16, form, false, Start::Urgent, p.smPercent, &grid, &smem)) return rc;
  if (p.stride == 6) return launchTc2<2, false, 6>(a, m, f16, grid, smem, s);
  return launchTc2<2, false, 10>(a, m, f16, grid, smem, s);
}

// Reads (and optionally clears) the status word after all work queued on the device has finished: the kernels run on
// the caller's streams, which the default stream does not wait for, so the whole device is synchronised first.
int convTcStatus(int* out, bool reset) {
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return failCuda("conv1d_tc_status: cudaDeviceSynchronize", e);
  int v = 0;
  e = cudaMemcpyFromSymbol(&v, gTcStatus, sizeof v);
  if (e != cudaSuccess) return failCuda("conv1d_tc_status", e);
  if (reset && v != 0) {
    const int z = 0;
    e = cudaMemcpyToSymbol(gTcStatus, &z, sizeof z);
    if (e != cudaSuccess) return failCuda("conv1d_tc_status", e);
  }
  *out = v;
  return 0;
}

// Stream-ordered read of the status word: queues a 4-byte copy into `hostOut` (pinned host memory) behind the work
// already on `s`; nothing is synchronised and nothing is cleared. The caller looks at *hostOut after it has
// synchronised with `s` (an event, a stream synchronise).
int convTcStatusAsync(int* hostOut, cudaStream_t s) {
  const DeviceInfo* d = nullptr;
  if (int rc = deviceInfo(&d)) return rc;
  const cudaError_t e = cudaMemcpyAsync(hostOut, d->status, sizeof(int), cudaMemcpyDeviceToHost, s);
  return e == cudaSuccess ? 0 : failCuda("conv1d_tc_status_async: cudaMemcpyAsync", e);
}

}  // namespace lkc
