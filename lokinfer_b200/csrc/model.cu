// Whole-model calls: the generator's forward, the decoder's forward and one AdaINResBlock1 as ONE call each (host code; the
// kernels it queues are those of this library's entry points, and three of the decoder's own). What they replace is the
// op-by-op compositions in generator.py and decoder.py, whose 110 and 48 calls through Python (argument checks, argument
// packing, one allocation per result, stream switches) took 5 and 1.7 ms of host time per forward whatever its length, two to
// ten times what the GPU needs below 10 s of audio.
//
// A forward is written once as a sequence of alloc / use / join / launch steps over an Exec and runs in two modes. In
// plan mode nothing is launched: every tensor's allocation and uses are recorded with the vector clock of the stream
// they happen on, and lkc_plan_memory turns that into offsets inside one workspace (the branches run on side streams,
// so a byte range is reused only where a join orders its uses before the new allocation). In run mode the same
// sequence takes its tensors from the workspace and queues its kernels. The plan depends on the length alone; the last
// few are kept with the model (a plan costs about 40 us).
#include <algorithm>
#include <list>
#include <memory>
#include <mutex>
#include <new>
#include <vector>

#include "lkc_common.h"

namespace lkc {
namespace {

constexpr int kStreams = 5;  // the caller's stream and four side streams
// Events of the joins, used in turn. A generator forward makes 17 joins, a decoder's 13: an event may be recorded again as soon
// as the wait on it has been queued, which is the case when join() returns.
constexpr int kEvents = 12;
constexpr size_t kPlans = 16;
constexpr float kEps = 1e-5f;  // AdaIN
// Percent of the SMs that one launch may spread over, as other branches run beside it (on one stream too, so that both
// ways add the same partial sums): [stage] the k = 3, 7, 11 resblocks, and the two noise branches. What runs beside each
// other may add up to more than 100: launches of branches rarely coincide for long, and clusters that find no room start
// when others end. The longer a branch's chain, the more it gets; the first noise branch is waited for one stage earlier than
// the second. us per forward as a graph, T = 24 / 80 / 121 / 200 / 320 / 640 / 2080 frames: as below 302 / 465 / 506 / 640 / 750 / 1347 /
// 3936; [stage 0 | stage 1 | noise] 26, 36, 70 | 26, 36, 50 | 70, 40: 302 / 464 / 504 / 703 / 815 / 1342 / 3954; 33 each, noise 50: 304 /
// 464 / 528 / 657 / 752 / 1340 / 3990; k = 11 at 90 in stage 0: 300 / 475 / 519 / 651 / 772 / 1338 / 3971. No splitting at all, with an
// earlier build: 877 at T = 24, 934 at 121.
// A resblock whose tiles its share leaves whole gets the other share, with which more lengths are split: a whole tile's chain
// of 16 channel chunks is then the branch's time. T = 72 / 80 / 90 / 100 / 110 / 121 / 140 / 160 / 320 / 640: 26 and 36 for k = 3 and 7 of
// stage 0 at every length 442 / 467 / 479 / 476 / 489 / 503 / 541 / 615 / 751 / 1340; 40 for both 441 / 471 / 488 / 485 / 501 / 507 / 566 /
// 619 / 751 / 1342; as below 444 / 465 / 473 / 473 / 488 / 506 / 572 / 620 / 750 / 1347. (It was drawn before the convs started early
// beside other launches: T = 121 / 140 / 160 586 / 604 / 691 with 26 and 36, 552 / 573 / 658 as below.)
struct Share {
  int split, whole;
};
constexpr Share kBranchSms[2][3] = {{{26, 40}, {36, 40}, {60, 60}}, {{26, 26}, {36, 36}, {50, 50}}};
constexpr int kNoiseSms[2] = {60, 50};

// Channels of the two stages, of what goes into their upsamplers, and the upsampling factors.
constexpr int64_t kCh[2] = {256, 128}, kChIn[2] = {512, 256}, kUp[2] = {10, 6};

// Percent of the SMs of resblock `branch` (k = 3, 7, 11) of a stage whose rows have l columns.
int branchSms(int stage, int branch, int64_t l, int sms, const int32_t* clusters) {
  const Share s = kBranchSms[stage][branch];
  return convTcSplitRule(kCh[stage], kCh[stage], l, sms * s.split / 100, clusters) ? s.split : s.whole;
}

struct Plan {
  int64_t key = 0, bytes = 0, unplanned = 0;
  std::vector<int64_t> offsets;
};

// A tensor of the workspace, or (id < 0) one of the caller's.
struct Buf {
  float* p = nullptr;
  int64_t pitch = 0;
  int id = -1;
};

class Exec {
 public:
  // plan mode
  explicit Exec(bool concurrent) : concurrent_(concurrent) {}
  // run mode
  Exec(bool concurrent, const Plan& plan, char* base, cudaStream_t main, const cudaStream_t* side, cudaEvent_t* events)
      : concurrent_(concurrent), plan_(&plan), base_(base), events_(events) {
    streams_[0] = main;
    for (int i = 1; i < kStreams; ++i) streams_[i] = concurrent ? side[i - 1] : main;
  }

  bool running() const { return plan_ != nullptr; }
  cudaStream_t stream(int s) const { return streams_[s]; }

  Buf alloc(int s, int64_t floats, int64_t pitch = 0) {
    Buf b;
    b.pitch = pitch, b.id = next_++;
    if (running()) {
      b.p = reinterpret_cast<float*>(base_ + plan_->offsets[b.id]);
      return b;
    }
    const int l = lane(s);
    ++clock_[l][l];
    bytes_.push_back(floats * 4);
    for (int i = 0; i < kStreams; ++i) allocClock_.push_back(clock_[l][i]), lastUse_.push_back(0);
    lastUse_[size_t(b.id) * kStreams + l] = clock_[l][l];
    return b;
  }
  // f32[c, l] with rows on 16-byte boundaries
  Buf rows(int s, int64_t c, int64_t l) { return alloc(s, c * ((l + 3) & ~int64_t(3)), (l + 3) & ~int64_t(3)); }

  // One op on stream s that reads or writes `bufs`; fn() queues its kernel, or the two that some convs take, and returns 0 or an
  // error code.
  template <class Fn>
  void launch(int s, std::initializer_list<Buf> bufs, Fn fn) {
    if (running()) {
      if (rc != 0) return;
      const int64_t before = launchCount();
      rc = fn(streams_[s]);
      launches += launchCount() - before;
      return;
    }
    const int l = lane(s);
    const int64_t n = ++clock_[l][l];
    for (const Buf& b : bufs)
      if (b.id >= 0) lastUse_[size_t(b.id) * kStreams + l] = n;
  }

  // Nothing queued on `waiter` from here on starts before everything queued on `waited` so far has finished.
  void join(int waiter, int waited) {
    if (!concurrent_) return;
    if (!running()) {
      for (int i = 0; i < kStreams; ++i) clock_[waiter][i] = std::max(clock_[waiter][i], clock_[waited][i]);
      return;
    }
    if (rc != 0) return;
    const cudaError_t err = order(waiter, waited);
    if (err != cudaSuccess) rc = failCuda("model: stream join", err);
    else if (waited == 0) forked_[waiter] = true;
  }

  // After an error: what the side streams were given still uses the workspace, so the caller's stream waits for it like
  // after a whole forward (and a capture can end). The first error is the one that is reported.
  void joinForked() {
    for (int s = 1; s < kStreams; ++s)
      if (forked_[s]) order(0, s);
  }

  // overlay = false: every tensor gets bytes of its own.
  int finishPlan(Plan* out, bool overlay = true) {
    const int64_t n = int64_t(bytes_.size());
    out->offsets.assign(size_t(n), 0);
    const std::vector<int32_t> pinned(size_t(n), overlay ? 0 : 1);
    for (int64_t b : bytes_) out->unplanned += (b + 255) / 256 * 256;
    return lkc_plan_memory(n, kStreams, bytes_.data(), pinned.data(), allocClock_.data(), lastUse_.data(), 256,
                           out->offsets.data(), &out->bytes);
  }

  int rc = 0;
  int64_t launches = 0;

 private:
  cudaError_t order(int waiter, int waited) {
    cudaEvent_t e = events_[event_++ % kEvents];
    cudaError_t err = cudaEventRecord(e, streams_[waited]);
    if (err == cudaSuccess) err = cudaStreamWaitEvent(streams_[waiter], e, 0);
    if (err != cudaSuccess) cudaGetLastError();  // reported by the caller; the next launch's check must not see it
    return err;
  }
  int lane(int s) const { return concurrent_ ? s : 0; }

  const bool concurrent_;
  const Plan* plan_ = nullptr;
  char* base_ = nullptr;
  cudaStream_t streams_[kStreams] = {};
  cudaEvent_t* events_ = nullptr;
  bool forked_[kStreams] = {};
  int next_ = 0, event_ = 0;
  std::vector<int64_t> bytes_, allocClock_, lastUse_;
  int64_t clock_[kStreams][kStreams] = {};
};

const float* FP(const void* p) { return static_cast<const float*>(p); }

// One fused conv of the tensor-core family, stride 1: act((x - mean) * scale + beta) -> conv -> + bias [+ residual].
void conv(Exec& e, int s, Act act, Buf x, int64_t l, int64_t ci, int64_t co, int64_t k, int64_t d, int64_t pad,
          const void* w, const void* b, Buf affine, const void* alpha, float slope, const LkcConvState* state, Buf residual,
          Buf out, Buf stats, int smPercent) {
  e.launch(s, {x, affine, residual, out, stats}, [&](cudaStream_t st) {
    ConvFusedParams p;
    p.x = x.p, p.w = FP(w), p.bias = FP(b), p.affine = affine.p, p.alpha = FP(alpha), p.residual = residual.p;
    p.out = out.p, p.stats = stats.p;
    p.ci = ci, p.l = l, p.co = co, p.k = k, p.dilation = d, p.padding = pad, p.lo = l + 2 * pad - d * (k - 1);
    p.xPitch = x.pitch, p.resPitch = residual.pitch, p.outPitch = out.pitch;
    p.act = act, p.slope = slope, p.state = state, p.smPercent = smPercent;
    return convFused(p, st);
  });
}

// AdaIN -> Snake -> conv [+ residual] of a resblock, c -> c channels of the same length. gb = this AdaIN's (gamma | beta)
// inside the style bank. The affine is a launch of its own unless the conv's route folds the statistics itself; the
// plan reserves it either way, as the route may change between two calls (set_conv_path). statCols: columns per pair of
// `stats`; the return value is that of outStats, 128 unless `fine` allows others.
int adainConv(Exec& e, int s, Buf x, Buf stats, int statCols, int64_t l, int64_t c, int64_t k, int64_t d, const LkcResblock& w,
              int i, Buf bank, Buf residual, Buf out, Buf outStats, bool fine, int smPercent, bool urgent) {
  const Buf af = e.alloc(s, 3 * c);
  ConvFusedParams p;
  p.x = x.p, p.w = FP(w.w[i]), p.bias = FP(w.b[i]), p.affine = af.p, p.alpha = FP(w.alpha[i]), p.residual = residual.p;
  p.out = out.p, p.stats = outStats.p;
  p.ci = c, p.l = l, p.co = c, p.k = k, p.dilation = d, p.padding = d * (k - 1) / 2, p.lo = l;
  p.xPitch = x.pitch, p.resPitch = residual.pitch, p.outPitch = out.pitch;
  p.act = Act::Snake, p.state = w.state[i], p.smPercent = smPercent, p.fineStats = fine, p.urgent = urgent;
  const float* gb = bank.p + w.gb[i];
  if (e.running() && statCols == 128 && convFoldsAffine(p)) {
    p.statsIn = stats.p, p.gb = gb, p.eps = kEps;
  } else {
    e.launch(s, {stats, bank, af}, [&](cudaStream_t st) { return adainAffine(stats.p, gb, af.p, c, l, kEps, st, statCols, true); });
    p.behindAffine = true;
  }
  e.launch(s, {x, stats, bank, af, residual, out, outStats}, [&](cudaStream_t st) { return convFused(p, st); });
  return e.running() ? convStatCols(p) : 128;
}

Buf statsBuf(Exec& e, int s, int64_t c, int64_t l, int64_t cols = 128) { return e.alloc(s, c * ceilDiv(l, cols) * 2); }

Buf channelStatsOf(Exec& e, int s, Buf x, int64_t c, int64_t l) {
  Buf st = statsBuf(e, s, c, l);
  e.launch(s, {x, st}, [&](cudaStream_t cs) { return channelStats(x.p, st.p, c, l, x.pitch, statChunks(l), cs); });
  return st;
}

// What the last conv of a block adds: its running x, or what `make` (called with that x before the block's last
// iteration) returns; `ready` is called just before the last conv is queued.
struct PlainResidual {
  Buf make(Buf x) const { return x; }
  void ready() const {}
};

// AdaINResBlock1 (models/kokoro/model.py:235-247): three times {affine, Snake conv (dilation 1, 3, 5), affine, Snake conv
// + residual}. `out` / `outStats` receive the result: the caller's memory where they come with a pointer, else tensors
// allocated here. outStats = null: nobody asks for the result's statistics.
template <class Residual>
void resblock(Exec& e, int s, const LkcResblock& w, Buf x, Buf stats, int64_t l, Buf bank, Buf* out, Buf* outStats,
              Residual residual, int smPercent, bool urgent = true) {
  static const int64_t dil[3] = {1, 3, 5};
  const int64_t c = w.c, k = w.k;
  const Buf none;
  int statCols = 128;
  for (int j = 0; j < 3; ++j) {
    const int64_t d = dil[j];
    const int i1 = 2 * j, i2 = 2 * j + 1;
    const bool last = j == 2;
    const Buf res = last ? residual.make(x) : x;
    Buf xt = e.rows(s, c, l), st1 = statsBuf(e, s, c, l, 32);
    statCols = adainConv(e, s, x, stats, statCols, l, c, k, d, w, i1, bank, none, xt, st1, true, smPercent, urgent);
    Buf xn = last && out->p ? *out : e.rows(s, c, l), stn;
    if (!last) stn = statsBuf(e, s, c, l, 32);
    else if (outStats) stn = outStats->p ? *outStats : statsBuf(e, s, c, l);
    if (last) residual.ready();
    statCols = adainConv(e, s, xt, st1, statCols, l, c, k, 1, w, i2, bank, res, xn, stn, !last, smPercent, urgent);
    x = xn, stats = stn;
  }
  *out = x;
  if (outStats) *outStats = stats;
}

bool resblockOk(const LkcResblock& w) {
  if (w.c < 1 || w.k < 1 || w.k % 2 == 0) return false;
  for (int i = 0; i < 6; ++i)
    if (!w.w[i] || !w.b[i] || !w.alpha[i] || w.gb[i] < 0) return false;
  return true;
}

// The generator (models/kokoro/model.py:735-781), the op sequence of Generator.forward. Streams: 0 the caller's, 1 and 2
// the noise branches (they need only `har`), 3 and 4 the k = 7 and k = 3 resblocks of a stage.
void generator(Exec& e, const LkcGenerator& m, const LkcGeneratorIo& io) {
  const int64_t t = io.t, len[2] = {10 * t, 60 * t + 1};
  const Buf none;
  Buf x, har;
  x.p = const_cast<float*>(FP(io.x)), x.pitch = io.x_pitch;
  har.p = const_cast<float*>(FP(io.har)), har.pitch = io.har_pitch;
  int deviceSms = 0;
  const int32_t* clusters = nullptr;  // the plan does not ask how launches are spread
  if (e.running() && (e.rc = convTcDevice(&deviceSms, &clusters)) != 0) return;

  Buf bank = e.alloc(0, m.bank_n);
  e.join(1, 0), e.join(2, 0), e.join(3, 0);
  // the style bank beside the first convs: the noise branches need it for their first AdaIN
  e.launch(3, {bank}, [&](cudaStream_t st) { return gemmBias(FP(io.s), FP(m.bank_wt), FP(m.bank_b), bank.p, 1, 128, m.bank_n, st); });

  auto upsample = [&](int i, Buf in, int64_t lin, Buf res) {
    Buf u = e.rows(0, kCh[i], len[i]);
    e.launch(0, {in, res, u}, [&](cudaStream_t st) {
      ConvtParams p;
      p.x = in.p, p.bias = FP(m.ups_b[i]), p.res = res.p, p.out = u.p;
      p.ci = kChIn[i], p.l = lin, p.co = kCh[i], p.stride = kUp[i], p.padLeft = i, p.slope = 0.1f;
      p.xPitch = in.pitch, p.resPitch = res.pitch, p.outPitch = u.pitch;
      const ConvState* cs = reinterpret_cast<const ConvState*>(m.ups_state[i]);
      return convtTc(p, cs->wp, cs->f16, st);
    });
    return u;
  };

  // The first upsampler runs next to the first noise branch, the longer of the two; their sum is formed by that
  // branch's last conv, whose residual is (its own running x) + (the upsampled input). The sum and its chunk statistics
  // then leave one epilogue, and neither the upsampler nor a statistics pass stands between the branch and stage 0.
  const Buf u0 = upsample(0, x, t, none);
  struct AddUpsampled {
    Exec& e;
    Buf u;
    int64_t c, l;
    Buf make(Buf x) const {
      e.join(0, 1);
      Buf r = e.rows(0, c, l);
      e.launch(0, {x, u, r}, [&](cudaStream_t st) { return addRows(x.p, u.p, r.p, c * r.pitch, st); });
      return r;
    }
    void ready() const { e.join(1, 0); }
  };
  Buf noise[2], noiseStats;
  for (int i = 1; i >= 0; --i) {  // polyphase view of `har`, stride-1 conv, resblock
    const int s = 1 + i;
    const LkcNoiseConv& n = m.noise_conv[i];
    const int64_t ly = len[i] + n.taps - 1;
    Buf y = e.rows(s, n.rows, ly);
    e.launch(s, {har, y}, [&](cudaStream_t st) {
      return spaceToDepth(har.p, y.p, 22, len[1], n.rows, ly, har.pitch, y.pitch, n.stride, n.padding, st);
    });
    Buf xs = e.rows(s, kCh[i], len[i]), xst = statsBuf(e, s, kCh[i], len[i]);
    conv(e, s, Act::None, y, ly, n.rows, kCh[i], n.taps, 1, 0, n.w, n.b, none, nullptr, 0.f, n.state, none, xs, xst,
         kNoiseSms[i]);
    e.join(s, 3);
    if (i == 0)
      resblock(e, s, m.noise_res[i], xs, xst, len[i], bank, &noise[i], &noiseStats, AddUpsampled{e, u0, kCh[0], len[0]}, kNoiseSms[i]);
    else
      resblock(e, s, m.noise_res[i], xs, xst, len[i], bank, &noise[i], nullptr, PlainResidual{}, kNoiseSms[i], false);
  }

  Buf in = noise[0], inStats = noiseStats, mean;
  for (int i = 0; i < 2; ++i) {
    const int64_t l = len[i], c = kCh[i];
    e.join(0, 1 + i);
    if (i == 1) {
      in = upsample(1, mean, len[0], noise[1]);
      inStats = channelStatsOf(e, 0, in, c, l);
    }
    e.join(3, 0), e.join(4, 0);
    Buf rb[3];
    for (int j = 2; j >= 0; --j)
      resblock(e, j == 2 ? 0 : (j == 1 ? 3 : 4), m.res[3 * i + j], in, inStats, l, bank, &rb[j], nullptr, PlainResidual{},
               e.running() ? branchSms(i, j, l, deviceSms, clusters) : 100);
    e.join(0, 3), e.join(0, 4);
    mean = e.rows(0, c, l);
    e.launch(0, {rb[0], rb[1], rb[2], mean}, [&](cudaStream_t cs) {
      return add3Scale(rb[0].p, rb[1].p, rb[2].p, mean.p, c * mean.pitch, 1.f / 3.f, cs);
    });
  }

  Buf post, ident;
  if (io.post) post.p = static_cast<float*>(io.post), post.pitch = io.post_pitch;
  else post = e.rows(0, 22, len[1]);
  ident.p = const_cast<float*>(FP(m.ident128));
  conv(e, 0, Act::Leaky, mean, len[1], 128, 22, 7, 1, 3, m.post_w, m.post_b, ident, nullptr, 0.01f, m.post_state, none, post, none,
       100);
  e.launch(0, {post}, [&](cudaStream_t st) {
    return istftLogits(post.p, static_cast<float*>(io.audio), len[1], post.pitch, 20, 5, st);
  });
}

// The decoder (models/kokoro/model.py:704-717), stream 1 for the shortcuts. A block's input is ONE buffer `cat` for the four
// decode blocks: rows [0, 1024) are what the block before wrote (a block reads them in its first conv and its shortcut, both
// before its second conv overwrites them), the others asr_res, F0, N and zero rows, written once. So nothing is concatenated
// between blocks, and the chunk statistics of the block's rows come from the epilogue that wrote them.
constexpr int64_t kDecIn[2] = {528, 1104}, kDecCh = 1024, kDecOut = 512;
constexpr float kDecSlope = 0.2f, kSqrtHalf = 0.7071067811865476f;
// Percent of the SMs (see kBranchSms) of the main convs and of the shortcuts beside them. At 100 each launch is planned, and
// started early, as if it ran alone; where two coincide, clusters wait for room, which for long inputs costs less than fewer CTAs
// per tile. Short ones have few clusters of many CTAs, of which the device holds few (15 of seven or eight, see countClusters), and
// gain when main convs and shortcuts leave each other room: the shares are the best pair measured for their number of tiles, on
// which the form of the launches depends. us per forward as a graph over three to six lengths of each row:
//   main, shortcuts | 65, 35  | 60, 40  | 100, 30 | 75, 25  | 100, 100
//   F = 8 to 64     | 171-186 | 197-214 | 173-187 | 179-194 | 194-208
//   F = 65 to 128   | 194-195 | 226-227 | 196-199 | 203-206 | 223-224
//   F = 129 to 256  | 293-299 | 254-259 | 276-281 | 275-282 | 265-271
//   F = 257 to 384  | 297-304 | 320-329 | 436-445 | 419-429 | 322-333
//   F = 385 to 512  | 469-475 | 492-501 | 456-463 | 466-472 | 349-354
//   F = 513 to 1040 | 511-569 | 511-571 | 500-706 | 537-576 | 432-568
struct DecSms {
  int main, shortcut;
};
DecSms decSms(int64_t frames) {
  static const DecSms few[] = {{65, 35}, {60, 40}, {65, 35}};  // by the 128-column tiles of a row
  const int64_t tiles = ceilDiv(frames, 128);
  return tiles <= 3 ? few[tiles - 1] : DecSms{100, 100};
}

void decoder(Exec& e, const LkcDecoder& m, const LkcDecoderIo& io) {
  const int64_t f = io.frames;
  const DecSms sms = decSms(f);
  const Buf none;
  auto from = [](Buf b, int64_t floats) {  // the same buffer from an offset on
    if (b.p) b.p += floats;
    return b;
  };
  Buf bank = e.alloc(0, m.bank_n), enc = e.rows(0, kDecIn[0], f), cat = e.rows(0, kDecIn[1], f);
  Buf encStats = statsBuf(e, 0, kDecIn[0], f), catStats = statsBuf(e, 0, kDecIn[1], f);
  const int64_t pitch = enc.pitch, chunkFloats = 2 * statChunks(f);
  e.join(1, 0);
  e.launch(1, {bank}, [&](cudaStream_t st) { return gemmBias(FP(io.s), FP(m.bank_wt), FP(m.bank_b), bank.p, 1, 128, m.bank_n, st); });
  e.launch(0, {enc, cat}, [&](cudaStream_t st) {
    return decoderInputs(FP(io.asr), io.asr_pitch, FP(io.f0), FP(io.n), FP(m.f0_w), FP(m.f0_b), FP(m.n_w), FP(m.n_b), enc.p,
                         kDecIn[0], cat.p, kDecCh + 64, kDecIn[1], f, pitch, st);
  });
  e.launch(0, {enc, encStats}, [&](cudaStream_t st) { return channelStats(enc.p, encStats.p, kDecIn[0], f, pitch, statChunks(f), st); });
  e.join(0, 1);  // the style bank
  e.join(1, 0);  // the block inputs
  conv(e, 1, Act::None, enc, f, 512, 64, 1, 1, 0, m.asr_w, m.asr_b, none, nullptr, 0.f, m.asr_state, none,
       from(cat, kDecCh * pitch), from(catStats, kDecCh * chunkFloats), sms.shortcut);
  e.launch(1, {cat, catStats}, [&](cudaStream_t st) {
    return channelStats(cat.p + (kDecCh + 64) * pitch, catStats.p + (kDecCh + 64) * chunkFloats, kDecIn[1] - kDecCh - 64, f,
                        pitch, statChunks(f), st);
  });

  // AdaIN -> leaky -> conv k 3 [+ residual, scaled]; see adainConv
  auto leakyConv = [&](Buf x, Buf stats, int64_t l, int64_t ci, int64_t co, const void* w, const void* b, const LkcConvState* state,
                       int64_t gbAt, Buf residual, Buf out, Buf outStats) {
    const Buf af = e.alloc(0, 3 * ci);
    ConvFusedParams p;
    p.x = x.p, p.w = FP(w), p.bias = FP(b), p.affine = af.p, p.residual = residual.p, p.out = out.p, p.stats = outStats.p;
    p.ci = ci, p.l = l, p.co = co, p.k = 3, p.padding = 1, p.lo = l;
    p.xPitch = x.pitch, p.resPitch = residual.pitch, p.outPitch = out.pitch;
    p.act = Act::Leaky, p.slope = kDecSlope, p.state = state, p.outScale = residual.pitch ? kSqrtHalf : 1.f;
    p.smPercent = sms.main;
    const float* gb = bank.p + gbAt;
    if (e.running() && convFoldsAffine(p))
      p.statsIn = stats.p, p.gb = gb, p.eps = kEps;
    else
      e.launch(0, {stats, bank, af}, [&](cudaStream_t st) { return adainAffine(stats.p, gb, af.p, ci, l, kEps, st); });
    e.launch(0, {x, stats, bank, af, residual, out, outStats}, [&](cudaStream_t st) { return convFused(p, st); });
  };

  for (int i = 0; i < 5; ++i) {
    const LkcDecoderBlock& b = m.block[i];
    const Buf x = i == 0 ? enc : cat, stats = i == 0 ? encStats : catStats;
    const int64_t l = b.up ? 2 * f : f;
    Buf h = e.rows(0, b.cout, l), hStats = statsBuf(e, 0, b.cout, l), sc = e.rows(0, b.cout, f);
    e.join(1, 0);
    conv(e, 1, Act::None, x, f, b.cin, b.cout, 1, 1, 0, b.w1x1, b.b1x1, none, nullptr, 0.f, b.state1x1, none, sc, none,
         sms.shortcut);
    if (!b.up) {
      leakyConv(x, stats, f, b.cin, b.cout, b.w1, b.b1, b.state1, b.gb1, none, h, hStats);
      e.join(0, 1);
      leakyConv(h, hStats, f, b.cout, b.cout, b.w2, b.b2, b.state2, b.gb2, sc, cat, catStats);
    } else {
      const Buf up = e.rows(1, b.cout, l);
      e.launch(1, {sc, up}, [&](cudaStream_t st) { return upsampleRows2(sc.p, up.p, b.cout, f, sc.pitch, up.pitch, st); });
      const Buf af = e.alloc(0, 3 * b.cin), r = e.rows(0, b.cin, l);
      e.launch(0, {stats, bank, af}, [&](cudaStream_t st) { return adainAffine(stats.p, bank.p + b.gb1, af.p, b.cin, f, kEps, st); });
      e.launch(0, {x, af, r}, [&](cudaStream_t st) {
        return adainLeakyPool(x.p, af.p, FP(b.pool_w), FP(b.pool_b), r.p, b.cin, f, x.pitch, r.pitch, kDecSlope, st);
      });
      conv(e, 0, Act::None, r, l, b.cin, b.cout, 3, 1, 1, b.w1, b.b1, none, nullptr, 0.f, b.state1, none, h, hStats, sms.main);
      e.join(0, 1);
      Buf out;
      out.p = static_cast<float*>(io.out), out.pitch = io.out_pitch;
      leakyConv(h, hStats, l, b.cout, b.cout, b.w2, b.b2, b.state2, b.gb2, up, out, none);
    }
  }
}

}  // namespace
}  // namespace lkc

using namespace lkc;

namespace {
bool isConcurrent(int64_t mode) { return mode != 0 && mode != LKC_UNPLANNED; }
}  // namespace

struct LkcModel {
  bool isDecoder = false;
  LkcGenerator w;
  LkcDecoder dec;
  cudaEvent_t events[kEvents] = {};
  std::mutex mutex;
  std::list<std::shared_ptr<const Plan>> plans;  // most recently used first

  // mode = LkcGeneratorIo.concurrent
  int plan(int64_t t, int64_t mode, std::shared_ptr<const Plan>* out) {
    const bool overlay = mode != LKC_UNPLANNED && mode != (LKC_UNPLANNED | 1), concurrent = isConcurrent(mode);
    const int64_t key = 4 * t + (overlay ? 2 : 0) + (concurrent ? 1 : 0);
    for (auto it = plans.begin(); it != plans.end(); ++it)
      if ((*it)->key == key) {
        plans.splice(plans.begin(), plans, it);
        *out = plans.front();
        return 0;
      }
    auto p = std::make_shared<Plan>();
    p->key = key;
    Exec e(concurrent);
    if (isDecoder) {
      LkcDecoderIo io{};
      io.frames = t;
      decoder(e, dec, io);
    } else {
      LkcGeneratorIo io{};
      io.t = t;
      generator(e, w, io);
    }
    if (int rc = e.finishPlan(p.get(), overlay)) return rc;
    plans.push_front(p);
    if (plans.size() > kPlans) plans.pop_back();
    *out = p;
    return 0;
  }
};

namespace {
// Whether a prepared state was made for this shape (conv: stride 0), as the sequence below assumes without looking again.
bool stateFits(const LkcConvState* state, int64_t co, int64_t ci, int64_t k, int64_t stride) {
  const ConvState* st = reinterpret_cast<const ConvState*>(state);
  return st && st->wp && st->co == co && st->ci == ci && st->k == k && st->stride == stride;
}
// A resblock of c channels whose AdaIN parameters lie inside a bank of bankN floats.
bool resblockFits(const LkcResblock& w, int64_t c, int64_t bankN) {
  if (!resblockOk(w) || w.c != c) return false;
  for (int i = 0; i < 6; ++i)
    if (w.gb[i] > bankN - 2 * c || (w.state[i] && !stateFits(w.state[i], c, c, w.k, 0))) return false;
  return true;
}
// The handle with its events, or null (and the handle gone).
LkcModel* withEvents(LkcModel* m) {
  for (cudaEvent_t& ev : m->events) {
    const cudaError_t err = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    if (err != cudaSuccess) {
      failCuda("model: cudaEventCreate", err);
      lkc_model_destroy(m);
      return nullptr;
    }
  }
  return m;
}
}  // namespace

extern "C" LKC_API LkcModel* lkc_generator_create(const LkcGenerator* w) {
  const char* bad = nullptr;
  if (!w) bad = "generator_create: null weights";
  if (!bad && (!w->bank_wt || !w->bank_b || w->bank_n < 1 || w->bank_n > 0x7fffffff || !w->post_w || !w->post_b || !w->ident128))
    bad = "generator_create: null weight";
  for (int i = 0; !bad && i < 8; ++i) {
    const LkcResblock& rb = i < 2 ? w->noise_res[i] : w->res[i - 2];
    if (!resblockFits(rb, kCh[i < 2 ? i : (i - 2) / 3], w->bank_n)) bad = "generator_create: bad resblock";
  }
  for (int i = 0; !bad && i < 2; ++i) {
    const LkcNoiseConv& n = w->noise_conv[i];
    if (!n.w || !n.b || n.stride < 1 || n.stride > 64 || n.padding < 0 || n.taps < 1 || n.rows < 22 * n.stride ||
        !stateFits(n.state, kCh[i], n.rows, n.taps, 0))
      bad = "generator_create: bad noise conv";
    else if (!w->ups_b[i] || !stateFits(w->ups_state[i], kCh[i], kChIn[i], 2 * kUp[i], kUp[i]))
      bad = "generator_create: bad upsampler";
  }
  if (!bad && w->post_state && !stateFits(w->post_state, 22, kCh[1], 7, 0)) bad = "generator_create: bad conv_post";
  LkcModel* m = bad ? nullptr : new (std::nothrow) LkcModel;
  if (!m) {
    fail(bad ? bad : "generator_create: out of host memory");
    return nullptr;
  }
  m->w = *w;
  return withEvents(m);
}

extern "C" LKC_API LkcModel* lkc_decoder_create(const LkcDecoder* w) {
  const char* bad = nullptr;
  if (!w) bad = "decoder_create: null weights";
  if (!bad && (!w->bank_wt || !w->bank_b || w->bank_n < 1 || w->bank_n > 0x7fffffff || !w->f0_w || !w->f0_b || !w->n_w ||
               !w->n_b || !w->asr_w || !w->asr_b || !stateFits(w->asr_state, 64, 512, 1, 0)))
    bad = "decoder_create: null weight or bad asr_res";
  for (int i = 0; !bad && i < 5; ++i) {
    const LkcDecoderBlock& b = w->block[i];
    const int64_t cin = kDecIn[i > 0], cout = i == 4 ? kDecOut : kDecCh;
    if (b.cin != cin || b.cout != cout || b.up != (i == 4) || !b.w1 || !b.b1 || !b.w2 || !b.b2 || !b.w1x1 || !b.b1x1 ||
        (b.up && (!b.pool_w || !b.pool_b)) || !stateFits(b.state1, cout, cin, 3, 0) || !stateFits(b.state2, cout, cout, 3, 0) ||
        !stateFits(b.state1x1, cout, cin, 1, 0) || b.gb1 < 0 || b.gb1 > w->bank_n - 2 * cin || b.gb2 < 0 ||
        b.gb2 > w->bank_n - 2 * cout)
      bad = "decoder_create: bad block";
  }
  LkcModel* m = bad ? nullptr : new (std::nothrow) LkcModel;
  if (!m) {
    fail(bad ? bad : "decoder_create: out of host memory");
    return nullptr;
  }
  m->isDecoder = true, m->dec = *w;
  return withEvents(m);
}

extern "C" LKC_API void lkc_model_destroy(LkcModel* m) {
  if (!m) return;
  for (cudaEvent_t ev : m->events)
    if (ev) cudaEventDestroy(ev);
  delete m;
}

extern "C" LKC_API int lkc_generator_branch_sms(int64_t t, int stage, int branch, int sms, const int32_t* clusters) {
  if (t < 1 || t >= (int64_t(1) << 24) || (stage | 1) != 1 || branch < 0 || branch > 2 || sms < 1 || sms > 65535 || !clusters) return 0;
  return branchSms(stage, branch, stage ? 60 * t + 1 : 10 * t, sms, clusters);
}

extern "C" LKC_API int lkc_generator_workspace(LkcModel* m, int64_t t, int concurrent, int64_t* bytes, int64_t* unplanned) {
  LKC_REQUIRE(m && bytes && !m->isDecoder, "generator_workspace: null argument or a decoder's handle");
  LKC_REQUIRE(t >= 1 && t < (int64_t(1) << 24), "generator_workspace: t out of range");
  return noThrow([&] {
    std::lock_guard<std::mutex> lock(m->mutex);
    std::shared_ptr<const Plan> p;
    if (int rc = m->plan(t, concurrent, &p)) return rc;
    *bytes = p->bytes;
    if (unplanned) *unplanned = p->unplanned;
    return 0;
  });
}

extern "C" LKC_API int lkc_generator_forward(LkcModel* m, LkcGeneratorIo* io, void* stream) {
  LKC_REQUIRE(m && io && io->x && io->har && io->s && io->audio && io->workspace, "generator_forward: null argument");
  LKC_REQUIRE(!m->isDecoder, "generator_forward: a decoder's handle");
  LKC_REQUIRE(io->t >= 1 && io->t < (int64_t(1) << 24), "generator_forward: t out of range");
  LKC_REQUIRE(io->x_pitch >= io->t && io->har_pitch >= 60 * io->t + 1 && (!io->post || io->post_pitch >= 60 * io->t + 1),
              "generator_forward: a row pitch is smaller than the row");
  LKC_REQUIRE((reinterpret_cast<uintptr_t>(io->workspace) & 255) == 0, "generator_forward: the workspace must be 256-byte aligned");
  // The events and the order of record and wait on them belong to one forward at a time; queueing is all that happens
  // under the lock.
  return noThrow([&] {
    std::lock_guard<std::mutex> lock(m->mutex);
    std::shared_ptr<const Plan> p;
    if (int rc = m->plan(io->t, io->concurrent, &p)) return rc;
    LKC_REQUIRE(io->workspace_bytes >= p->bytes, "generator_forward: the workspace is too small (lkc_generator_workspace)");
    Exec e(isConcurrent(io->concurrent), *p, static_cast<char*>(io->workspace), S(stream),
           reinterpret_cast<const cudaStream_t*>(io->side), m->events);
    generator(e, m->w, *io);
    if (e.rc != 0) e.joinForked();
    io->launches = e.launches;
    return e.rc;
  });
}

namespace {
// Whether `side` can be forked from `stream` and joined back: not while it is in a capture that `stream` is not in. A side
// stream stays in its caller's capture when that call returns, until the capture ends; a fork from outside would fail and
// invalidate the capture.
bool joinable(cudaStream_t stream, cudaStream_t side) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone, sd = cudaStreamCaptureStatusNone;
  unsigned long long idStream = 0, idSide = 0;
  if (cudaStreamGetCaptureInfo(side, &sd, &idSide) != cudaSuccess || sd == cudaStreamCaptureStatusInvalidated) {
    cudaGetLastError();
    return false;
  }
  if (sd == cudaStreamCaptureStatusNone) return true;
  if (cudaStreamGetCaptureInfo(stream, &st, &idStream) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return st == cudaStreamCaptureStatusActive && idStream == idSide;
}
}  // namespace

extern "C" LKC_API int lkc_decoder_workspace(LkcModel* m, int64_t frames, int64_t* bytes) {
  LKC_REQUIRE(m && bytes && m->isDecoder, "decoder_workspace: null argument or a generator's handle");
  LKC_REQUIRE(frames >= 1 && frames < (int64_t(1) << 24), "decoder_workspace: frames out of range");
  return noThrow([&] {
    std::lock_guard<std::mutex> lock(m->mutex);
    std::shared_ptr<const Plan> p;
    if (int rc = m->plan(frames, 1, &p)) return rc;
    *bytes = p->bytes;
    return 0;
  });
}

extern "C" LKC_API int lkc_decoder_forward(LkcModel* m, LkcDecoderIo* io, void* stream) {
  LKC_REQUIRE(m && io && io->asr && io->f0 && io->n && io->s && io->out && io->workspace && io->side,
              "decoder_forward: null argument");
  LKC_REQUIRE(m->isDecoder, "decoder_forward: a generator's handle");
  LKC_REQUIRE(io->frames >= 1 && io->frames < (int64_t(1) << 24), "decoder_forward: frames out of range");
  LKC_REQUIRE(io->asr_pitch >= io->frames && io->out_pitch >= 2 * io->frames, "decoder_forward: a row pitch is smaller than the row");
  LKC_REQUIRE((reinterpret_cast<uintptr_t>(io->workspace) & 255) == 0, "decoder_forward: the workspace must be 256-byte aligned");
  return noThrow([&] {  // as lkc_generator_forward
    std::lock_guard<std::mutex> lock(m->mutex);
    std::shared_ptr<const Plan> p;
    if (int rc = m->plan(io->frames, 1, &p)) return rc;
    LKC_REQUIRE(io->workspace_bytes >= p->bytes, "decoder_forward: the workspace is too small (lkc_decoder_workspace)");
    cudaStream_t side[kStreams - 1];
    for (cudaStream_t& s : side) s = joinable(S(stream), S(io->side)) ? S(io->side) : S(stream);
    Exec e(true, *p, static_cast<char*>(io->workspace), S(stream), side, m->events);
    decoder(e, m->dec, *io);
    if (e.rc != 0) e.joinForked();
    io->launches = e.launches;
    return e.rc;
  });
}

namespace {
// The sequence of lkc_resblock in both modes.
void resblockCall(Exec& e, const LkcResblock& w, const LkcResblockIo& io) {
  Buf x, st, bank, out, outStats;
  x.p = const_cast<float*>(FP(io.x)), x.pitch = io.x_pitch;
  bank.p = const_cast<float*>(FP(io.bank));
  out.p = static_cast<float*>(io.out), out.pitch = io.out_pitch;
  outStats.p = static_cast<float*>(io.out_stats);
  if (io.stats) st.p = const_cast<float*>(FP(io.stats));
  else st = channelStatsOf(e, 0, x, w.c, io.l);
  resblock(e, 0, w, x, st, io.l, bank, &out, &outStats, PlainResidual{}, 100);
}
}  // namespace

extern "C" LKC_API int lkc_resblock(const LkcResblock* w, LkcResblockIo* io, void* stream) {
  LKC_REQUIRE(w && io && resblockOk(*w) && io->l >= 1, "resblock: bad argument");
  LKC_REQUIRE(io->x && io->bank && io->out && io->out_stats, "resblock: null operand");
  LKC_REQUIRE(io->x_pitch >= io->l && io->out_pitch >= io->l, "resblock: a row pitch is smaller than the row");
  LKC_REQUIRE(w->c <= 65535, "resblock: too many channels");  // channel_stats: one grid row per channel
  LKC_REQUIRE(((reinterpret_cast<uintptr_t>(io->stats) | reinterpret_cast<uintptr_t>(io->out_stats)) & 7) == 0,
              "resblock: stats and out_stats must be 8-byte aligned");
  return noThrow([&] {
    Plan p;
    Exec plan(false);
    resblockCall(plan, *w, *io);
    if (int rc = plan.finishPlan(&p)) return rc;
    if (!io->workspace) {  // the size only
      io->workspace_bytes = p.bytes;
      return 0;
    }
    LKC_REQUIRE((reinterpret_cast<uintptr_t>(io->workspace) & 255) == 0 && io->workspace_bytes >= p.bytes,
                "resblock: the workspace must be 256-byte aligned and hold what the size call says");
    Exec e(false, p, static_cast<char*>(io->workspace), S(stream), nullptr, nullptr);
    resblockCall(e, *w, *io);
    io->launches = e.launches;
    return e.rc;
  });
}
