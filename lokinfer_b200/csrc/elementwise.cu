// Basic (unfused) layer and the HBM-bound statistics kernels of the Kokoro generator path:
// snake / leaky_relu / add / add3_scale / scale / pad_reflect1d / adain1d, channel_stats, adain_affine and the
// style-bank GEMV. Each is a streaming kernel: one pass over its operands, coalesced along time, grids sized
// from the element count.
#include "lkc_common.h"

namespace lkc {
namespace {

constexpr int kThreads = 256;

inline int gridFor(int64_t n, int perThread = 1) {
  int64_t b = ceilDiv(n, int64_t(kThreads) * perThread);
  return static_cast<int>(b < 1 ? 1 : (b > 148 * 32 ? 148 * 32 : b));
}

__device__ __forceinline__ float warpSum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warpSumD(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__global__ void snakeKernel(const float* __restrict__ x, const float* __restrict__ alpha, float* __restrict__ out,
                            int64_t c, int64_t l) {
  const int64_t n = c * l;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const float a = alpha[i / l], v = x[i];
    const float s = sinf(a * v);
    out[i] = v + (1.f / a) * (s * s);
  }
}

__global__ void leakyKernel(const float* __restrict__ x, float* __restrict__ out, int64_t n, float slope) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const float v = x[i];
    out[i] = v > 0.f ? v : v * slope;
  }
}

__global__ void addKernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ out,
                          int64_t n) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    out[i] = a[i] + b[i];
}

__global__ void add3ScaleKernel(const float* __restrict__ a, const float* __restrict__ b, const float* __restrict__ c,
                                float* __restrict__ out, int64_t n, float s) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    out[i] = __fmul_rn(__fadd_rn(__fadd_rn(a[i], b[i]), c[i]), s);
}

__global__ void scaleKernel(const float* __restrict__ x, float* __restrict__ out, int64_t n, float s) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    out[i] = x[i] * s;
}

__global__ void padReflectKernel(const float* __restrict__ x, float* __restrict__ out, int64_t c, int64_t l,
                                 int64_t left, int64_t right) {
  const int64_t lo = left + l + right, n = c * lo;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t ch = i / lo, j = i - ch * lo;
    int64_t src = j - left;
    if (src < 0) src = -src;
    if (src >= l) src = 2 * (l - 1) - src;
    out[i] = x[ch * l + src];
  }
}

// One block per channel: two-pass mean / biased variance, then (x - mean) * a + b.
__global__ void adain1dKernel(const float* __restrict__ x, const float* __restrict__ gb, float* __restrict__ out,
                              int64_t c, int64_t l, float eps) {
  __shared__ double red[kThreads / 32];
  __shared__ float bc[2];
  const int64_t ch = blockIdx.x;
  const float* xr = x + ch * l;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double s = 0.0;
  for (int64_t i = threadIdx.x; i < l; i += blockDim.x) s += xr[i];
  s = warpSumD(s);
  if (lane == 0) red[wid] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) t += red[w];
    bc[0] = static_cast<float>(t / static_cast<double>(l));
  }
  __syncthreads();
  const float mean = bc[0];
  double q = 0.0;
  for (int64_t i = threadIdx.x; i < l; i += blockDim.x) {
    const float d = xr[i] - mean;
    q += d * d;
  }
  q = warpSumD(q);
  __syncthreads();
  if (lane == 0) red[wid] = q;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) t += red[w];
    const float var = static_cast<float>(t / static_cast<double>(l));
    bc[1] = (1.f + gb[ch]) * (1.0f / sqrtf(var + eps));
  }
  __syncthreads();
  const float a = bc[1], b = gb[c + ch];
  float* o = out + ch * l;
  for (int64_t i = threadIdx.x; i < l; i += blockDim.x) o[i] = (xr[i] - mean) * a + b;
}

// One warp per (channel, 128-sample chunk): mean, then M2 = sum (v - mean)^2 from registers. Lanes side by side on every
// row layout. Four consecutive samples per lane instead (one 16-byte load where the rows allow it): aligned rows the same within
// 3 %, others 7 to 14 % slower ([128, 124801] 14.6 -> 16.1 us, [512, 4161] 3.6 -> 4.1), also when turned through shared memory.
__global__ void channelStatsKernel(const float* __restrict__ x, float* __restrict__ stats, int64_t l,
                                   int64_t nchunks, int64_t pitch, int64_t statsStride) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t chunk = blockIdx.x * int64_t(blockDim.x >> 5) + wid, ch = blockIdx.y;
  if (chunk >= nchunks) return;
  const int64_t t0 = chunk * kStatChunk;
  const int n = static_cast<int>(l - t0 < kStatChunk ? l - t0 : kStatChunk);
  const float* xr = x + ch * pitch + t0;
  float v[4];
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int i = lane + 32 * j;
    v[j] = i < n ? xr[i] : 0.f;
    s += v[j];
  }
  s = warpSum(s);
  const float mean = s / static_cast<float>(n);
  float q = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float d = (lane + 32 * j) < n ? v[j] - mean : 0.f;
    q = fmaf(d, d, q);
  }
  q = warpSum(q);
  if (lane == 0) {
    float* st = stats + (ch * statsStride + chunk) * 2;
    st[0] = mean;
    st[1] = q;
  }
}

// One 128-thread block per channel: exact combine of the (count, mean, M2) partials in double, in one pass relative to the row's
// first mean (to 0 where that is not finite, so that infinities and NaN come out as from sums). A first mean far from the row's costs
// at most a factor of the number of pairs of 2^-53, as it is in the variance itself. What bounds it is latency, between two convs:
// one round of loads (up to 8 pairs per thread in flight; longer rows loop), one of shuffles, one barrier. Two passes with
// a division each and five barriers cost 0.5 us more per step: us per generator forward as a graph T = 121 514 -> 506, T = 200
// 642 -> 631, T = 320 761 -> 751, T = 480 967 -> 954.
// Its inputs are not __restrict__: an early launch reads what the one in front of it may still be writing, and loads of read-only
// data could be moved in front of the wait.
constexpr int kAffineThreads = 128;
__global__ void __launch_bounds__(kAffineThreads) adainAffineKernel(const float* stats, const float* gb, float* affine, int64_t c,
                                                                    int64_t l, int64_t nchunks, int statCols, double invL, float eps,
                                                                    int early) {
  dependenciesWait();
  if (early) dependentsLaunch();  // not before: a conv that waits holds SMs, and what it waits for is then this kernel alone
  __shared__ double red[2 * kAffineThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t ch = blockIdx.x;
  const float2* sc = reinterpret_cast<const float2*>(stats) + ch * nchunks;  // (mean, M2) pairs, 8-byte aligned
  const double nT = static_cast<double>(statCols), nLast = static_cast<double>(l - (nchunks - 1) * statCols);
  constexpr int R = 8;
  float2 v[R];
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const int64_t t = threadIdx.x + int64_t(j) * kAffineThreads;
    v[j] = t < nchunks ? sc[t] : make_float2(0.f, 0.f);
  }
  const float x0 = sc[0].x, gamma = gb[ch], beta = gb[c + ch];
  const double pivot = fabsf(x0) <= 3.402823466e38f ? static_cast<double>(x0) : 0.0;
  double s1 = 0.0, s2 = 0.0;  // sum of (x - pivot), sum of (x - pivot)^2
  auto add = [&](float2 p, int64_t t) {
    const double n = t + 1 < nchunks ? nT : nLast, d = static_cast<double>(p.x) - pivot;
    s1 += n * d, s2 += static_cast<double>(p.y) + n * d * d;
  };
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const int64_t t = threadIdx.x + int64_t(j) * kAffineThreads;
    if (t < nchunks) add(v[j], t);
  }
  for (int64_t t = threadIdx.x + int64_t(R) * kAffineThreads; t < nchunks; t += kAffineThreads) add(sc[t], t);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s1 += __shfl_xor_sync(0xffffffffu, s1, o), s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  if (lane == 0) red[wid] = s1, red[kAffineThreads / 32 + wid] = s2;
  __syncthreads();
  if (threadIdx.x == 0) {
    s1 = s2 = 0.0;
    for (int w = 0; w < kAffineThreads / 32; ++w) s1 += red[w], s2 += red[kAffineThreads / 32 + w];
    const double dm = s1 * invL, q = s2 * invL - dm * dm;
    const float var = q < 0.0 ? 0.f : static_cast<float>(q);  // (a NaN stays one)
    affine[ch] = static_cast<float>(pivot + dm);
    affine[c + ch] = (1.f + gamma) * (1.0f / sqrtf(var + eps));
    affine[2 * c + ch] = beta;
  }
}

// out[m, n] = sum_k x[m, k] wt[k, n] + b[n]; one thread per output column, coalesced over n.
__global__ void gemmBiasKernel(const float* __restrict__ x, const float* __restrict__ wt, const float* __restrict__ b,
                               float* __restrict__ out, int64_t m, int64_t k, int64_t n) {
  extern __shared__ float xs[];
  const int64_t row = blockIdx.y;
  for (int64_t i = threadIdx.x; i < k; i += blockDim.x) xs[i] = x[row * k + i];
  __syncthreads();
  const int64_t col = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (col >= n) return;
  float acc = 0.f;
  for (int64_t i = 0; i < k; ++i) acc = fmaf(xs[i], wt[i * n + col], acc);
  out[row * n + col] = acc + b[col];
}

// The same for few outputs (the style bank: M = 1, K = 128), where the latency of the loads is the time: GEMV_K threads share a
// column's sum, so that 16 rows of wt are in flight per thread and four times the blocks run.
constexpr int GEMV_N = 64, GEMV_K = 4;
__global__ void gemvBiasKernel(const float* __restrict__ x, const float* __restrict__ wt, const float* __restrict__ b,
                               float* __restrict__ out, int64_t m, int64_t k, int64_t n) {
  extern __shared__ float xs[];  // x's row, then the partial sums
  const int64_t row = blockIdx.y;
  const int tc = threadIdx.x % GEMV_N, tk = threadIdx.x / GEMV_N;
  for (int64_t i = threadIdx.x; i < k; i += blockDim.x) xs[i] = x[row * k + i];
  __syncthreads();
  const int64_t col = blockIdx.x * int64_t(GEMV_N) + tc, k0 = k * tk / GEMV_K, k1 = k * (tk + 1) / GEMV_K;
  float acc = 0.f;
  if (col < n) {
#pragma unroll 16
    for (int64_t i = k0; i < k1; ++i) acc = fmaf(xs[i], wt[i * n + col], acc);
  }
  __syncthreads();
  xs[threadIdx.x] = acc;
  __syncthreads();
  if (tk == 0 && col < n)
    out[row * n + col] = ((xs[tc] + xs[GEMV_N + tc]) + (xs[2 * GEMV_N + tc] + xs[3 * GEMV_N + tc])) + b[col];
}

}  // namespace

// ---- launchers shared by the C-ABI entry points below and the whole-model calls (model.cu)

int channelStats(const float* x, float* stats, int64_t c, int64_t l, int64_t pitch, int64_t statsStride, cudaStream_t s) {
  const int64_t nchunks = statChunks(l);
  dim3 grid(static_cast<unsigned>(ceilDiv(nchunks, kThreads / 32)), static_cast<unsigned>(c));
  channelStatsKernel<<<grid, kThreads, 0, s>>>(x, stats, l, nchunks, pitch, statsStride);
  return launched("channel_stats_f32_cuda");
}

// Early between two convs, beside other launches too: the launch itself (1.5 us of a 3.5 us step between two convs) is over when
// the first conv ends. Its blocks do not fit beside a conv CTA, which leaves 4096 registers of an SM where a block takes 7168:
// they wait on SMs that hold no conv, and where there are none start as the first conv's CTAs leave. One that waits keeps a
// ready conv CTA of another branch off its SM. The conv behind it starts early where it says so itself. us per forward as
// a graph, early only where nothing runs beside it -> everywhere: T = 16 303 -> 306, T = 24 319 -> 319, T = 80 498 -> 488, T = 121
// 563 -> 552, T = 170 685 -> 688, T = 320 879 -> 867, T = 640 1344 -> 1335, T = 800 1510 -> 1502, T = 2080 the same.
int adainAffine(const float* stats, const float* gb, float* affine, int64_t c, int64_t l, float eps, cudaStream_t s,
                int statCols, bool early) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3(unsigned(c)), cfg.blockDim = dim3(kAffineThreads), cfg.stream = s, cfg.attrs = attr;
  if (early) {
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 1;
  }
  const cudaError_t e = cudaLaunchKernelEx(&cfg, adainAffineKernel, stats, gb, affine, c, l, ceilDiv(l, statCols), statCols,
                                           1.0 / double(l), eps, early ? 1 : 0);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return failCuda("adain_affine_f32_cuda", e);
  }
  return launched("adain_affine_f32_cuda");
}

// us with one thread per column / with four: [1, 128] x [128, 19104] 5.4 / 3.6, [1, 512] x [512, 19104] 15.5 / 8.1. One is better
// for sums of fewer than 64 terms (K = 33, N = 100: 2.6 / 3.1) and where the outputs fill the device already, from about 400
// blocks of 256 on: [300, 512] x [512, 512] (600) 19 / 26, [64, 128] x [128, 19104] 37 / 51, [32, 512] x [512, 4096] (512) 19 / 22;
// below, [16, 128] x [128, 4096] (256) 5.7 / 5.2, [4, 512] x [512, 19104] (298) 16.7 / 15.6, [4, 128] x [128, 19104] 5.9 / 6.1. Sums
// of thousands of terms over a wide matrix can go the other way ([32, 4096] x [4096, 4096] 192 / 171).
int gemmBias(const float* x, const float* wt, const float* b, float* out, int64_t m, int64_t k, int64_t n, cudaStream_t s) {
  static_assert(GEMV_K == 4, "the sum of the parts");
  constexpr int kGemvThreads = GEMV_N * GEMV_K;
  const auto grid = [&](int64_t cols) { return dim3(static_cast<unsigned>(ceilDiv(n, cols)), static_cast<unsigned>(m)); };
  if (k < 64 || m * n > 400 * 256)
    gemmBiasKernel<<<grid(kThreads), kThreads, static_cast<size_t>(k) * 4, s>>>(x, wt, b, out, m, k, n);
  else
    gemvBiasKernel<<<grid(GEMV_N), kGemvThreads, static_cast<size_t>(k > kGemvThreads ? k : kGemvThreads) * 4, s>>>(x, wt, b, out, m, k, n);
  return launched("gemm_bias_f32_cuda");
}

int addRows(const float* a, const float* b, float* out, int64_t n, cudaStream_t s) {
  addKernel<<<gridFor(n), kThreads, 0, s>>>(a, b, out, n);
  return launched("add_f32_cuda");
}

int add3Scale(const float* a, const float* b, const float* c, float* out, int64_t n, float scale, cudaStream_t s) {
  add3ScaleKernel<<<gridFor(n), kThreads, 0, s>>>(a, b, c, out, n, scale);
  return launched("add3_scale_f32_cuda");
}

namespace {

int64_t numel(const int64_t* dims, int rank) {
  int64_t n = 1;
  for (int i = 0; i < rank; ++i) n *= dims[i];
  return n;
}

// Rank of the operands of an elementwise op with `nOperands` operands and one out, all of the same rank.
int rankOf(const LkcArgs* a, int nOperands) { return static_cast<int>(a->numInts) / (nOperands + 1); }

}  // namespace
}  // namespace lkc

using namespace lkc;

extern "C" LKC_API int lkc_snake_f32_cuda(const LkcArgs* a, void* stream) {
  LKC_REQUIRE(a && a->numPtrs == 3 && a->numInts >= 5, "snake_f32_cuda: expected x, alpha | out");
  const int64_t c = a->ints[0], l = a->ints[1];
  LKC_REQUIRE(a->ints[2] == c, "snake_f32_cuda: alpha must be f32[C]");
  if (c * l == 0) return 0;
  snakeKernel<<<gridFor(c * l), kThreads, 0, S(stream)>>>(F(a, 0), F(a, 1), O(a, 2), c, l);
  return launched("snake_f32_cuda");
}

extern "C" LKC_API int lkc_leaky_relu_f32_cuda(const LkcArgs* a, void* stream) {
  LKC_REQUIRE(a && a->numPtrs == 2 && a->floats, "leaky_relu_f32_cuda: expected x | out and slope");
  const int64_t n = numel(a->ints, rankOf(a, 1));
  if (n == 0) return 0;
  leakyKernel<<<gridFor(n), kThreads, 0, S(stream)>>>(F(a, 0), O(a, 1), n, static_cast<float>(a->floats[0]));
  return launched("leaky_relu_f32_cuda");
}

extern "C" LKC_API int lkc_add_f32_cuda(const LkcArgs* a, void* stream) {
  LKC_REQUIRE(a && a->numPtrs == 3, "add_f32_cuda: expected a, b | out");
  const int64_t n = numel(a->ints, rankOf(a, 2));
  if (n == 0) return 0;
  return addRows(F(a, 0), F(a, 1), O(a, 2), n, S(stream));
}

extern "C" LKC_API int lkc_add3_scale_f32_cuda(const LkcArgs* a, void* stream) {
  LKC_REQUIRE(a && a->numPtrs == 4 && a->floats, "add3_scale_f32_cuda: expected a, b, c | out and scale");
  const int64_t n = numel(a->ints, rankOf(a, 3));
  if (n == 0) return 0;
  return add3Scale(F(a, 0), F(a, 1), F(a, 2), O(a, 3), n, static_cast<float>(a->floats[0]), S(stream));
}

extern "C" LKC_API int lkc_scale_f32_cuda(const LkcArgs* a, void* stream) {
  LKC_REQUIRE(a && a->numPtrs == 2 && a->floats, "scale_f32_cuda: expected x | out and scale");
  const int64_t n = numel(a->ints, rankOf(a, 1));
  if (n == 0) return 0;
  scaleKernel<<<gridFor(n), kThreads, 0, S(stream)>>>(F(a, 0), O(a, 1), n, static_cast<float>(a->floats[0]));
  return launched("scale_f32_cuda");
}

extern "C" LKC_API int lkc_pad_reflect1d_f32_cuda(const LkcArgs* a, void* stream) {
  LKC_REQUIRE(a && a->numPtrs == 2 && a->numInts == 6, "pad_reflect1d_f32_cuda: expected x | out, left, right");
  const int64_t c = a->ints[0], l = a->ints[1], left = a->ints[4], right = a->ints[5];
  LKC_REQUIRE(left >= 0 && right >= 0 && left < l && right < l, "pad_reflect1d_f32_cuda: reflect padding must be < L");
  LKC_REQUIRE(a->ints[3] == l + left + right, "pad_reflect1d_f32_cuda: out must be f32[C, left + L + right]");
  const int64_t n = c * (l + left + right);
  if (n == 0) return 0;
  padReflectKernel<<<gridFor(n), kThreads, 0, S(stream)>>>(F(a, 0), O(a, 1), c, l, left, right);
  return launched("pad_reflect1d_f32_cuda");
}

// Polyphase view of a strided conv's input: y[ci * s + r, t] = x[ci, s t + r - pad] (zero outside [0, L)); rows from
// Ci * s on are zero (channel padding up to the row count of y). A conv with stride s, K = taps * s and padding pad
// over x equals a stride-1 conv with `taps` taps over y with the weights w'[co, ci * s + r, j] = w[co, ci, s j + r],
// which is a shape the tensor-core conv takes. No counterpart in the reference (its strided conv is direct,
// kernels/cpu/kokoro_conv.cpp:32-69).
__global__ void spaceToDepthKernel(const float* __restrict__ x, float* __restrict__ y, int64_t ci, int64_t l,
                                   int64_t rows, int64_t ly, int64_t xPitch, int64_t yPitch, int s, int64_t pad) {
  // A block row is one input channel, blockDim columns of its s rows at a time: they are s * blockDim consecutive input samples,
  // read once along time and written through shared memory. The block rows behind the channels write zero rows. Bound by
  // memory (22 -> 144 rows, T = 2080: 23 MB).
  extern __shared__ float sx[];
  for (int64_t c = blockIdx.y; c < ci + rows - ci * s; c += gridDim.y) {
    for (int64_t t0 = blockIdx.x * int64_t(blockDim.x); t0 < ly; t0 += int64_t(gridDim.x) * blockDim.x) {
      const int64_t t = t0 + threadIdx.x;
      if (c >= ci) {
        if (t < ly) y[(ci * s + (c - ci)) * yPitch + t] = 0.f;
        continue;
      }
      const int64_t pos0 = int64_t(s) * t0 - pad;
      for (int i = threadIdx.x; i < s * int(blockDim.x); i += blockDim.x) {
        const int64_t pos = pos0 + i;
        sx[i] = pos >= 0 && pos < l ? x[c * xPitch + pos] : 0.f;
      }
      __syncthreads();
      if (t < ly)
        for (int r = 0; r < s; ++r) y[(c * s + r) * yPitch + t] = sx[threadIdx.x * s + r];
      __syncthreads();
    }
  }
}

// The same for large strides and small calls: 1 << lc columns at a time, the threads spread over columns and phases, and a gap of
// one float per 32 in shared memory, since lanes `s` floats apart would meet in one bank where s is a multiple of 32.
__global__ void spaceToDepthWideKernel(const float* __restrict__ x, float* __restrict__ y, int64_t ci, int64_t l, int64_t rows,
                                       int64_t ly, int64_t xPitch, int64_t yPitch, int s, int64_t pad, int lc) {
  extern __shared__ float sx[];
  const int n = s << lc, last = (1 << lc) - 1;
  for (int64_t c = blockIdx.y; c < ci + rows - ci * s; c += gridDim.y) {
    for (int64_t t0 = int64_t(blockIdx.x) << lc; t0 < ly; t0 += int64_t(gridDim.x) << lc) {
      if (c >= ci) {
        const int64_t t = t0 + threadIdx.x;
        if (int(threadIdx.x) <= last && t < ly) y[(ci * s + (c - ci)) * yPitch + t] = 0.f;
        continue;
      }
      const int64_t pos0 = int64_t(s) * t0 - pad;
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int64_t pos = pos0 + i;
        sx[i + (i >> 5)] = pos >= 0 && pos < l ? x[c * xPitch + pos] : 0.f;
      }
      __syncthreads();
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int r = i >> lc, t = i & last, at = t * s + r;
        if (t0 + t < ly) y[(c * s + r) * yPitch + t0 + t] = sx[at + (at >> 5)];
      }
      __syncthreads();
    }
  }
}

// Stride 1: a copy with padding and zero rows, four loads in flight per thread ([22, 124801] 5.4 us, through shared memory 14.6).
__global__ void spaceToDepthCopyKernel(const float* __restrict__ x, float* __restrict__ y, int64_t ci, int64_t l, int64_t rows,
                                       int64_t ly, int64_t xPitch, int64_t yPitch, int64_t pad) {
  for (int64_t c = blockIdx.y; c < rows; c += gridDim.y) {
    const float* const xr = x + c * xPitch - pad;
    for (int64_t t = blockIdx.x * int64_t(4 * kThreads) + threadIdx.x; t < ly; t += int64_t(gridDim.x) * 4 * kThreads) {
      float v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int64_t at = t + j * kThreads;
        v[j] = c < ci && at >= pad && at - pad < l ? xr[at] : 0.f;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (t + j * kThreads < ly) y[c * yPitch + t + j * kThreads] = v[j];
    }
  }
}

namespace lkc {
// us for [channels, length], stride: one thread per column and all its phases / the wide form (columns at a time). Few blocks are
// better spread: [3, 4000], 8 3.6 / 1.9 (16), 15 5.0 / 1.9 (16), 33 8.6 / 2.5 (16); [3, 400000], 17 6.2 / 5.0 (64). So are strides
// that put a warp's lanes into few banks: [500, 200000], 16 356 / 310 (64), 32 555 / 284, and the largest: [100, 40000], 63 17.6 /
// 10.2. Otherwise the first reads and writes in longer runs: [500, 200000], 17 241 / 323, 20 250 / 299; [22, 124801], 6 6.8 / 11.9.
int spaceToDepth(const float* x, float* y, int64_t ci, int64_t l, int64_t rows, int64_t ly, int64_t xPitch, int64_t yPitch,
                 int64_t stride, int64_t pad, cudaStream_t s) {
  const auto grid = [&](int64_t cols, int64_t most, int64_t blockRows) {
    const int64_t bx = ceilDiv(ly, cols);
    return dim3(unsigned(bx < most ? bx : most), unsigned(blockRows < 65535 ? blockRows : 65535));
  };
  const int64_t blockRows = ci + rows - ci * stride;
  const bool few = ceilDiv(ly, kThreads) * ci < 296;  // two blocks per SM of a B200
  if (stride == 1) {
    spaceToDepthCopyKernel<<<grid(4 * kThreads, 4096, rows), kThreads, 0, s>>>(x, y, ci, l, rows, ly, xPitch, yPitch, pad);
  } else if (stride < 8 || (stride <= 33 && !few && (stride < 16 || stride % 8 != 0))) {
    const int threads = stride <= 32 ? kThreads : kThreads / 2;  // at most 32 KB of shared memory
    spaceToDepthKernel<<<grid(threads, 512, blockRows), threads, size_t(stride) * threads * 4, s>>>(x, y, ci, l, rows, ly, xPitch,
                                                                                                   yPitch, int(stride), pad);
  } else {
    int lc = 6;
    while (lc > 4 && ceilDiv(ly, int64_t(1) << lc) * ci < 512) --lc;
    const size_t n = size_t(stride) << lc;  // at most 4096 floats
    spaceToDepthWideKernel<<<grid(int64_t(1) << lc, 4096, blockRows), kThreads, (n + n / 32) * 4, s>>>(x, y, ci, l, rows, ly, xPitch,
                                                                                                      yPitch, int(stride), pad, lc);
  }
  return launched("space_to_depth_f32_cuda");
}
}  // namespace lkc

// ints: x(Ci, L) y(rows, Ly) pad stride [x_pitch y_pitch]
extern "C" LKC_API int lkc_space_to_depth_f32_cuda(const LkcArgs* a, void* stream) {
  LKC_REQUIRE(a && a->numPtrs == 2 && (a->numInts == 6 || a->numInts == 8), "space_to_depth_f32_cuda: expected x | y, pad, stride");
  const int64_t ci = a->ints[0], l = a->ints[1], rows = a->ints[2], ly = a->ints[3], pad = a->ints[4], s = a->ints[5];
  const int64_t xPitch = a->numInts == 8 ? a->ints[6] : l, yPitch = a->numInts == 8 ? a->ints[7] : ly;
  LKC_REQUIRE(s >= 1 && s <= 64 && pad >= 0 && ci >= 1 && l >= 1, "space_to_depth_f32_cuda: invalid stride / padding");
  LKC_REQUIRE(rows >= ci * s && ly >= 1 && yPitch >= ly && xPitch >= l,
              "space_to_depth_f32_cuda: y must be f32[rows >= Ci * stride, Ly]");
  return spaceToDepth(F(a, 0), O(a, 1), ci, l, rows, ly, xPitch, yPitch, s, pad, S(stream));
}

extern "C" LKC_API int lkc_adain1d_f32_cuda(const LkcArgs* a, void* stream) {
  LKC_REQUIRE(a && a->numPtrs == 3 && a->numInts == 5 && a->floats, "adain1d_f32_cuda: expected x, gb | out and eps");
  const int64_t c = a->ints[0], l = a->ints[1];
  LKC_REQUIRE(a->ints[2] == 2 * c, "adain1d_f32_cuda: gb must be f32[2C]");
  LKC_REQUIRE(l >= 1, "adain1d_f32_cuda: empty sequence");
  if (c == 0) return 0;
  adain1dKernel<<<static_cast<int>(c), kThreads, 0, S(stream)>>>(F(a, 0), F(a, 1), O(a, 2), c, l,
                                                                 static_cast<float>(a->floats[0]));
  return launched("adain1d_f32_cuda");
}

extern "C" LKC_API int lkc_channel_stats_f32_cuda(const LkcArgs* a, void* stream) {
  LKC_REQUIRE(a && a->numPtrs == 2 && a->numInts >= 5 && a->numInts <= 7, "channel_stats_f32_cuda: expected x | stats");
  const int64_t c = a->ints[0], l = a->ints[1], nchunks = statChunks(l);
  const int64_t pitch = a->numInts >= 6 ? a->ints[5] : l;  // optional trailing ints: row pitch of x, row stride of stats in chunks
  const int64_t statsStride = a->numInts == 7 ? a->ints[6] : nchunks;
  LKC_REQUIRE(pitch >= l && statsStride >= nchunks, "channel_stats_f32_cuda: a row pitch is smaller than the row");
  LKC_REQUIRE(l >= 1, "channel_stats_f32_cuda: empty sequence");
  LKC_REQUIRE(a->ints[2] == c && a->ints[3] == nchunks && a->ints[4] == 2,
              "channel_stats_f32_cuda: stats must be f32[C, ceil(L/128), 2]");
  LKC_REQUIRE(c <= 65535, "channel_stats_f32_cuda: too many channels");
  if (c == 0) return 0;
  return channelStats(F(a, 0), O(a, 1), c, l, pitch, statsStride, S(stream));
}

extern "C" LKC_API int lkc_adain_affine_f32_cuda(const LkcArgs* a, void* stream) {
  LKC_REQUIRE(a && a->numPtrs == 3 && a->numInts == 7 && a->floats,
              "adain_affine_f32_cuda: expected stats, gb | affine, length and eps");
  const int64_t c = a->ints[0], nchunks = a->ints[1], l = a->ints[6];
  LKC_REQUIRE(l >= 1 && nchunks == statChunks(l), "adain_affine_f32_cuda: stats chunks don't match length");
  LKC_REQUIRE(a->ints[3] == 2 * c, "adain_affine_f32_cuda: gb must be f32[2C]");
  LKC_REQUIRE(a->ints[4] == 3 && a->ints[5] == c, "adain_affine_f32_cuda: affine must be f32[3, C]");
  if (c == 0) return 0;
  LKC_REQUIRE(c <= 0x7fffffff, "adain_affine_f32_cuda: too many channels");
  LKC_REQUIRE((reinterpret_cast<uintptr_t>(a->ptrs[0]) & 7) == 0, "adain_affine_f32_cuda: stats must be 8-byte aligned");
  return adainAffine(F(a, 0), F(a, 1), O(a, 2), c, l, static_cast<float>(a->floats[0]), S(stream));
}

extern "C" LKC_API int lkc_gemm_bias_f32_cuda(const LkcArgs* a, void* stream) {
  LKC_REQUIRE(a && a->numPtrs == 4 && a->numInts == 7, "gemm_bias_f32_cuda: expected x, wt, b | out");
  const int64_t m = a->ints[0], k = a->ints[1], n = a->ints[3];
  LKC_REQUIRE(a->ints[2] == k && a->ints[4] == n && a->ints[5] == m && a->ints[6] == n,
              "gemm_bias_f32_cuda: shapes must be x[M,K] wt[K,N] b[N] out[M,N]");
  LKC_REQUIRE(k * 4 <= 48 * 1024 && m <= 65535, "gemm_bias_f32_cuda: K or M too large for this kernel");
  if (m * n == 0) return 0;
  return gemmBias(F(a, 0), F(a, 1), F(a, 2), O(a, 3), m, k, n, S(stream));
}
