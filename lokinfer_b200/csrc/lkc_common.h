// Internal helpers shared by the lkc kernel sources: error reporting and argument decoding.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <exception>
#include <new>

#include "lkc.h"

namespace lkc {

// Records a failure message for lkc_last_error() and returns 1.
int fail(const char* msg);
int failCuda(const char* what, cudaError_t e);

inline const float* F(const LkcArgs* a, int i) { return static_cast<const float*>(a->ptrs[i]); }
inline float* O(const LkcArgs* a, int i) { return static_cast<float*>(a->ptrs[i]); }
inline cudaStream_t S(void* stream) { return static_cast<cudaStream_t>(stream); }

int64_t& launchCount();  // kernels that this thread has queued (api.cu)

// Checks and counts the launch that was just issued (no synchronisation).
inline int launched(const char* what) {
  cudaError_t e = cudaPeekAtLastError();
  if (e != cudaSuccess) {
    cudaGetLastError();
    return failCuda(what, e);
  }
  ++launchCount();
  return 0;
}

// Runs the body of a C entry point that allocates host memory: an exception becomes an error code.
template <class Fn>
int noThrow(Fn body) {
  try {
    return body();
  } catch (const std::bad_alloc&) {
    return fail("out of host memory");
  } catch (const std::exception&) {
    return fail("unexpected exception");
  }
}

#ifdef __CUDACC__
// Programmatic dependent launch. wait: until every kernel this launch depends on has finished and its writes are visible.
// launch: the kernel that follows may start (it waits in the same way before it touches what this one writes or reads).
__device__ __forceinline__ void dependenciesWait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dependentsLaunch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

#define LKC_REQUIRE(cond, msg) \
  do {                         \
    if (!(cond)) return ::lkc::fail(msg); \
  } while (0)

constexpr int64_t kStatChunk = 128;
inline int64_t statChunks(int64_t l) { return (l + kStatChunk - 1) / kStatChunk; }
inline int64_t ceilDiv(int64_t a, int64_t b) { return (a + b - 1) / b; }

enum class Act : int { None = 0, Snake = 1, Leaky = 2 };

// Operands of the fused conv family (one struct for the CUDA-core and the tensor-core kernels).
struct ConvFusedParams {
  const float* x = nullptr;
  const float* x2 = nullptr;  // mean3 prologue: input = ((x + x2) + x3) * inScale
  const float* x3 = nullptr;
  const float* w = nullptr;  // [co, ci, k]
  const float* bias = nullptr;
  const float* affine = nullptr;  // [3, ci] rows mean, scale, beta; null = identity
  const float* alpha = nullptr;
  const float* residual = nullptr;
  float* out = nullptr;
  float* stats = nullptr;  // may be null
  int64_t ci = 0, l = 0, co = 0, k = 0, dilation = 1, padding = 0, lo = 0;
  // Row pitches in floats of the [C, L] tensors x (x2, x3 share it), residual and out; 0 = contiguous rows.
  int64_t xPitch = 0, resPitch = 0, outPitch = 0;
  // Window extension (time-sharded tensors): output column t reads x columns xOrigin + t * stride - padding + kk *
  // dilation; x columns outside [validLo, validHi) count as zero padding (applied after the activation). A regular
  // call has xOrigin = 0 and the valid range [0, l) (validHi < 0 = not set). statsStride = row stride of `stats` in
  // chunks (0 = ceil(lo / 128)): the chunk statistics can be written into a slice of a longer row.
  int64_t xOrigin = 0, validLo = 0, validHi = -1, statsStride = 0;
  Act act = Act::None;
  float slope = 0.f, outScale = 1.f, inScale = 1.f;
  const void* state = nullptr;
  int smPercent = 100;  // part of the device's SMs this launch may spread over (others run beside it); 100 is planned as alone
  // Instead of `affine`, where convFoldsAffine: chunk statistics [ci, ceil(l / 128), 2] of x and the (gamma | beta) of its
  // AdaIN; the conv computes the affine itself.
  const float *statsIn = nullptr, *gb = nullptr;
  float eps = 0.f;
  // When it may start before what it waits for has ended (convTc's rule): the launch in front of it is its adain_affine, which says so
  // only when the conv before has ended; false: a branch that nobody waits for soon.
  bool behindAffine = false, urgent = true;
  bool fineStats = false;  // stats may come as one pair per 32 columns (convStatCols says which)
};

// One fused conv, routed to the tensor-core kernel when the shape qualifies, else to the CUDA-core kernel (api.cu).
int convFused(const ConvFusedParams& p, cudaStream_t s);
// Whether that route takes p.statsIn / p.gb instead of p.affine (the tensor-core kernel's split form).
bool convFoldsAffine(const ConvFusedParams& p);
// Columns per (mean, M2) pair of p.stats on that route: 128, or 32 where p.fineStats lets the tensor-core kernel choose.
int convStatCols(const ConvFusedParams& p);
// CUDA-core implicit-GEMM conv for any shape (conv_simt.cu). stride > 1 only for the plain conv1d.
int convSimt(const ConvFusedParams& p, int64_t stride, cudaStream_t s);

// Tensor-core (tcgen05, split operands) fused conv (conv_tc.cu). `state` of ConvFusedParams is an LkcConvState.
struct ConvState {
  const float* wp;  // packed weights (convTcPack / convtTcPack)
  int64_t co, ci, k;
  int64_t stride;  // 0 = conv1d pack; otherwise the ConvTranspose1d stride the pack was made for
  bool f16;        // operand format of the pack: f16 hi/lo split (true) or tf32 hi/lo split (false)
};
// Operands of the polyphase ConvTranspose1d (convt.cu decodes them, conv_tc.cu can run them).
struct ConvtParams {
  const float *x, *bias, *res;
  float* out;
  int64_t ci, l, co, stride, padLeft;
  float slope;
  int64_t xPitch = 0, resPitch = 0, outPitch = 0;  // row pitches in floats; 0 = contiguous rows
  // Window extension: x holds haloLeft / haloRight real columns before / after the l columns that produce output
  // (time-sharded tensors; the zero padding of the transposed conv then applies only where a halo is absent).
  int64_t haloLeft = 0, haloRight = 0;
  int smPercent = 100;  // as in ConvFusedParams
};
bool convtTcEligible(int64_t ci, int64_t co, int64_t k, int64_t stride, int64_t padding);
int64_t convtTcPackFloats(int64_t ci, int64_t co, int64_t stride, bool f16);
int convtTcPack(const float* w, float* wp, int64_t ci, int64_t co, int64_t k, int64_t stride, int64_t padding, bool f16,
                cudaStream_t s);
int convtTc(const ConvtParams& p, const float* wp, bool f16, cudaStream_t s);
bool convPathForcedSimt();
bool convPackF16();  // operand format new packs are made in (lkc_set_conv_path)
bool convTcEligible(const ConvFusedParams& p, bool f16);
bool convTcSplits(const ConvFusedParams& p, bool f16);  // of an eligible conv
int convTcStatCols(const ConvFusedParams& p, bool f16);  // of an eligible conv
int convTcTileRule(int64_t co, int64_t lo, int sms, int smPercent);
int convTcDevice(int* sms, const int32_t** clusters);  // what the rules are asked with on the current device
int convTcSplitRule(int64_t ci, int64_t co, int64_t lo, int sms, const int32_t* clusters);
int convTcSplitCols(int64_t lo);
int convTcPairRule(int64_t ci, int64_t co, int64_t lo, int64_t k, int64_t dilation, int64_t padding, Act act, bool fineOk,
                   bool behindAffine, int smPercent, int sms, const int32_t* clusters);
int64_t convTcRoundsRule(int64_t ci, int64_t co, int64_t lo, int64_t k, int sms, const int32_t* clusters);
int64_t convTcPackFloats(int64_t co, int64_t ci, int64_t k, bool f16);
int convTcPack(const float* w, float* wp, int64_t co, int64_t ci, int64_t k, bool f16, cudaStream_t s);
int convTc(const ConvFusedParams& p, const float* wp, bool f16, cudaStream_t s);
int convTcStatus(int* out, bool reset);
int convTcStatusAsync(int* hostOut, cudaStream_t s);
int convTcSetIo(int mode);
int convTcProfile(int enable, long long* out16);

// Launchers behind the C-ABI entry points of the same names (elementwise.cu, istft.cu, conv_tc.cu); arguments checked by
// the caller. Row pitches in floats.
int channelStats(const float* x, float* stats, int64_t c, int64_t l, int64_t pitch, int64_t statsStride, cudaStream_t s);
int adainAffine(const float* stats, const float* gb, float* affine, int64_t c, int64_t l, float eps, cudaStream_t s, int statCols = 128,
                bool early = false);  // it may start, and let what follows it start, before what it waits for has ended
int gemmBias(const float* x, const float* wt, const float* b, float* out, int64_t m, int64_t k, int64_t n, cudaStream_t s);
int addRows(const float* a, const float* b, float* out, int64_t n, cudaStream_t s);
int add3Scale(const float* a, const float* b, const float* c, float* out, int64_t n, float scale, cudaStream_t s);
int spaceToDepth(const float* x, float* y, int64_t ci, int64_t l, int64_t rows, int64_t ly, int64_t xPitch, int64_t yPitch,
                 int64_t stride, int64_t pad, cudaStream_t s);
// Decoder (decoder.cu): the rows around the convs' results in both kinds of block input; AdaIN, leaky ReLU and the depthwise
// pool of the upsampling block in one pass; nearest-neighbour upsampling by 2.
int decoderInputs(const float* asr, int64_t asrPitch, const float* f0, const float* n, const float* f0w, const float* f0b,
                  const float* nw, const float* nb, float* enc, int64_t encRows, float* cat, int64_t catRow, int64_t catRows,
                  int64_t l, int64_t pitch, cudaStream_t s);
int adainLeakyPool(const float* x, const float* affine, const float* w, const float* bias, float* out, int64_t c, int64_t l,
                   int64_t xPitch, int64_t outPitch, float slope, cudaStream_t s);
int upsampleRows2(const float* x, float* out, int64_t c, int64_t l, int64_t xPitch, int64_t outPitch, cudaStream_t s);
int istftLogits(const float* x, float* out, int64_t l, int64_t pitch, int nfft, int hop, cudaStream_t s);

}  // namespace lkc
