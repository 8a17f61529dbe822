"""The work whose speed is watched: what a user of this framework has it do, through its public entry points.

One weight set per process (random init, as in lokinfer_b200.synth) stands for the model a program loads once; inputs
are drawn from the case's seed. A generator frame is 12.5 ms of audio (300 samples at 24 kHz), so T frames are T / 80
seconds; the decoder in front of it works on F = T / 2 frames.

Kinds of cases:
  speak     Generator.synthesize: pinned host buffers in, waveform in a pinned host buffer out; the call of a program
            that says one utterance and waits for it.
  speak_f0  Generator.synthesize_f0: the same from the pitch curve (harmonic source with in-kernel noise and STFT on the
            device).
  stream    Generator.pipeline: a queue of utterances of one length from host buffers, two in flight; the throughput
            form of a server.
  forward   Generator.forward on device tensors, nothing captured: utterances whose length is new each time.
  decode    Decoder.forward: aligned text features, pitch and energy curves -> the generator's input.
  chain     Decoder.forward, Generator.har_from_f0, Generator.forward: text features to waveform on the device.
  resblock  the three AdaINResBlock1 of one generator stage, each called by itself on a contiguous [C, L] tensor.
  conv      one fused conv (affine -> Snake -> conv -> residual, chunk statistics) called as an op on contiguous tensors.
"""
from __future__ import annotations

import functools
import math

import torch

from lokinfer_b200 import ops, synth
from lokinfer_b200.decoder import Decoder
from lokinfer_b200.generator import RES_KERNELS, Generator

DEVICE = "cuda"
T_MIN, T_MAX = 16, 2080  # 0.2 s (one syllable) .. 26 s (a paragraph)


def listed():
    return [
        # one word (0.3 s): the smallest call, all latency
        {"name": "speak_T24", "kind": "speak", "T": 24},
        # one sentence (4 s)
        {"name": "speak_T320", "kind": "speak", "T": 320},
        # a paragraph (26 s): the repository's headline workload
        {"name": "speak_T2080", "kind": "speak", "T": 2080},
        # an odd length (9.3 s) from the pitch curve
        {"name": "speak_f0_T747", "kind": "speak_f0", "T": 747},
        # a server's queue: six utterances of 10 s each
        {"name": "stream_T800x6", "kind": "stream", "T": 800, "n": 6},
        # lengths that are not captured: a short utterance of odd length (1.5 s) and a long one (10 s)
        {"name": "forward_T121", "kind": "forward", "T": 121},
        {"name": "forward_T800", "kind": "forward", "T": 800},
        # the decoder of a 1.5 s and of a 26 s utterance
        {"name": "decode_F61", "kind": "decode", "F": 61},
        {"name": "decode_F1040", "kind": "decode", "F": 1040},
        # text features to waveform (4 s)
        {"name": "chain_F160", "kind": "chain", "F": 160},
        # stage-1 resblocks (C = 128) over 4 s, the odd row length that the reflect pad makes
        {"name": "resblock_C128_L19201", "kind": "resblock", "stage": 1, "L": 19201},
        # the widest conv of the operator sweep
        {"name": "conv_C512_L19200_k7", "kind": "conv", "C": 512, "L": 19200, "K": 7, "d": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["speak", "speak", "speak_f0", "stream", "forward", "forward", "decode", "chain", "resblock",
                       "conv"])
    if kind in ("speak", "speak_f0", "forward"):
        return {"kind": kind, "T": _log_int(rng, T_MIN, T_MAX)}
    if kind == "stream":
        return {"kind": kind, "T": _log_int(rng, 80, 800), "n": rng.randint(2, 6)}
    if kind in ("decode", "chain"):
        return {"kind": kind, "F": _log_int(rng, T_MIN // 2, T_MAX // 2)}
    if kind == "resblock":
        stage = rng.randint(0, 1)
        return {"kind": kind, "stage": stage, "L": _log_int(rng, 320, (20800, 124801)[stage])}
    c = rng.choice([128, 256, 512])
    return {"kind": kind, "C": c, "L": _log_int(rng, 320, 124801 * 128 // c), "K": rng.choice(RES_KERNELS),
            "d": rng.choice([1, 3, 5])}


# ------------------------------------------------------------------ the model and the inputs

@functools.lru_cache(maxsize=None)
def _generator():
    return Generator(synth.generator_weights(0), DEVICE)


@functools.lru_cache(maxsize=None)
def _decoder():
    return Decoder(synth.decoder_weights(0), DEVICE)


class _Draws:
    """Seeded device-side draws."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE)
        self.g.manual_seed(int(seed))

    def normal(self, *shape, scale=1.0):
        return torch.randn(*shape, generator=self.g, device=DEVICE) * scale

    def uniform(self, lo, hi, *shape):
        return torch.rand(*shape, generator=self.g, device=DEVICE) * (hi - lo) + lo


def _host(t):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out


def _utterance(r, t):
    """Host buffers of one utterance: x, har, style, and the waveform buffer."""
    return (_host(r.normal(512, t)), _host(r.normal(synth.N_BINS, synth.shapes(t)["L1"])), _host(r.normal(128)),
            torch.empty(synth.shapes(t)["S"], pin_memory=True))


def prepare(case, seed):
    kind, r = case["kind"], _Draws(seed)
    st = {"kind": kind, "gen": _generator()}
    if kind == "speak":
        st["utt"] = _utterance(r, case["T"])
        st["gen"].capture(case["T"])
    elif kind == "speak_f0":
        t = case["T"]
        st["x"], st["s"] = _host(r.normal(512, t)), _host(r.normal(128))
        st["f0"] = _host(torch.from_numpy(synth.f0_curve(t, seed)))
        st["seed"], st["audio"] = 1234 + seed, torch.empty(synth.shapes(t)["S"], pin_memory=True)
        st["gen"].capture(t)
    elif kind == "stream":
        st["utts"] = [_utterance(r, case["T"]) for _ in range(case["n"])]
        st["pipe"] = st["gen"].pipeline(case["T"])
    elif kind == "forward":
        st["x"], st["s"] = r.normal(512, case["T"]), r.normal(128)
        st["har"] = r.normal(synth.N_BINS, synth.shapes(case["T"])["L1"])
    elif kind in ("decode", "chain"):
        f = case["F"]
        st["dec"] = _decoder()
        st["asr"], st["s"], st["n"] = r.normal(512, f), r.normal(128), r.uniform(0.0, 4.0, 2 * f)
        st["f0"], st["seed"] = torch.from_numpy(synth.f0_curve(2 * f, seed)).to(DEVICE), 1234 + seed
    elif kind == "resblock":
        st["stage"], st["s"] = case["stage"], r.normal(128)
        st["x"] = r.normal((256, 128)[case["stage"]], case["L"])
    else:
        c, l, k, d = case["C"], case["L"], case["K"], case["d"]
        w = r.normal(c, c, k, scale=1.0 / math.sqrt(c * k))
        st["args"] = (r.normal(c, l), w, r.normal(c, scale=0.1),
                      torch.stack([r.normal(c, scale=0.5), r.uniform(0.5, 1.5, c), r.normal(c, scale=0.3)]),
                      r.uniform(0.5, 1.5, c))
        st["kw"] = {"residual": r.normal(c, l), "padding": d * (k - 1) // 2, "dilation": d,
                    "state": ops.conv1d_prepare_f32_cuda(w)}
    torch.cuda.synchronize()
    return st


# ------------------------------------------------------------------ one pass

def run(st):
    kind, gen = st["kind"], st["gen"]
    if kind == "speak":
        x, har, s, audio = st["utt"]
        return gen.synthesize(x, har, s, audio)
    if kind == "speak_f0":
        return gen.synthesize_f0(st["x"], st["f0"], st["seed"], st["s"], st["audio"])
    if kind == "stream":
        pipe = st["pipe"]
        tickets = [pipe.submit(*u) for u in st["utts"]]
        for k in tickets:
            pipe.wait(k)
        return [u[3] for u in st["utts"]]
    if kind == "forward":
        return gen.forward(st["x"], st["har"], st["s"])
    if kind == "decode":
        return st["dec"].forward(st["asr"], st["f0"], st["n"], st["s"])
    if kind == "chain":
        x = st["dec"].forward(st["asr"], st["f0"], st["n"], st["s"])
        return gen.forward(x, gen.har_from_f0(st["f0"], st["seed"]), st["s"])
    if kind == "resblock":
        gb = gen.style(st["s"])
        return [gen.adain_resblock1_fused(st["x"], gb, f"resblocks.{3 * st['stage'] + j}", k)
                for j, k in enumerate(RES_KERNELS)]
    return ops.conv1d_snake_f32_cuda(*st["args"], **st["kw"])


# ------------------------------------------------------------------ what a pass cannot do without

def _resblock_macs(c, k):
    return 6 * c * c * k  # per column: three iterations of two convs


def _generator_work(t):
    """(multiply-adds of the convolutions, weight floats) of one generator forward."""
    sh, macs, weights, ci = synth.shapes(t), 0, 0, 512
    for (c, ku, su, kn), k_noise, l_in, l in zip(synth.STAGES, (12, 1), (t, sh["L0"]), (sh["L0"], sh["L1"])):
        macs += ci * c * ku * l_in + synth.N_BINS * c * k_noise * l
        macs += sum(_resblock_macs(c, k) for k in (kn, *RES_KERNELS)) * l
        weights += ci * c * ku + synth.N_BINS * c * k_noise + sum(_resblock_macs(c, k) + 12 * c * 128
                                                                  for k in (kn, *RES_KERNELS))
        ci = c
    macs += 128 * synth.N_BINS * 7 * sh["L1"]
    return macs, weights + 128 * synth.N_BINS * 7


def _decoder_work(f):
    macs, weights = 512 * 64 * f, 512 * 64
    for _, cin, cout, up in synth.DECODER_BLOCKS:
        w = 3 * cout * (cin + cout) + (cin * cout if cin != cout else 0)
        macs += w * f * (2 if up else 1)
        weights += w + 2 * 128 * (cin + cout)
    return macs, weights


def work(case):
    kind = case["kind"]
    if kind in ("speak", "speak_f0", "stream", "forward"):
        t, n = case["T"], case.get("n", 1)
        macs, weights = _generator_work(t)
        har = t if kind == "speak_f0" else synth.N_BINS * synth.shapes(t)["L1"]
        return {"bytes": 4.0 * (weights + n * (512 * t + har + 128 + 300 * t)), "flops": 2.0 * macs * n}
    if kind in ("decode", "chain"):
        f = case["F"]
        macs, weights = _decoder_work(f)
        io = 512 * f + 4 * f + 128 + 512 * 2 * f
        if kind == "chain":
            gm, gw = _generator_work(2 * f)
            macs, weights, io = macs + gm, weights + gw, 512 * f + 4 * f + 128 + 600 * f
        return {"bytes": 4.0 * (weights + io), "flops": 2.0 * macs}
    if kind == "resblock":
        c, l = (256, 128)[case["stage"]], case["L"]
        per = sum(_resblock_macs(c, k) for k in RES_KERNELS)
        return {"bytes": 4.0 * (per + 3 * 12 * c * 128 + 4 * c * l), "flops": 2.0 * per * l}
    c, l, k = case["C"], case["L"], case["K"]
    return {"bytes": 4.0 * (c * c * k + 3 * c * l), "flops": 2.0 * c * c * k * l}


def tolerance(case):
    # Float32 throughout. One conv or one block: the rounding of 32-bit sums. A whole generator: that rounding through
    # some twenty convolutions, normalisations and Snakes in a row, then exp.
    return {"rel": 1e-5 if case["kind"] in ("conv", "resblock", "decode") else 2e-5}
