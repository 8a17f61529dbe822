"""The host logic around the decoder's whole-forward call, on CPU tensors with a stand-in for the library: what several
threads and streams of one Decoder hand to it."""
import contextlib
import ctypes
import threading
import time
import types

import pytest
import torch

from lokinfer_b200 import _lib, ops
from lokinfer_b200 import decoder as D
from lokinfer_b200.synth import DECODER_BLOCKS

FRAMES = 4


class Library:
    """lkc_decoder_workspace / _forward: keeps (the caller's stream, its side stream) of every call."""

    def __init__(self):
        self.calls = []

    def lkc_decoder_workspace(self, handle, frames, size):
        ctypes.cast(size, ctypes.POINTER(ctypes.c_int64))[0] = 256
        return 0

    def lkc_decoder_forward(self, handle, io, stream):
        self.calls.append((stream, ctypes.cast(io, ctypes.POINTER(_lib.LkcDecoderIo))[0].side))
        return 0


@pytest.fixture
def dec(monkeypatch):
    """A decoder on CPU tensors (weights unset) with stand-ins for the prepared states, the library, the model's handle and the
    streams: thread-local current stream `lib.at.stream`, new ones numbered from 1000, each slow to make."""
    d = D.Decoder.__new__(D.Decoder)
    d.device, d.w, d.state, d.gb_pad, d.bank_off = torch.device("cpu"), {}, {}, {}, {}
    off = 0

    def conv(name, co, ci, k):
        d.w[name + ".weight"], d.w[name + ".bias"] = torch.empty(co, ci, k), torch.empty(co)
        d.state[name] = types.SimpleNamespace(handle=4096, shape=(co, ci, k))

    conv("decoder.asr_res.0", 64, 512, 1)
    for c in ("F0_conv", "N_conv"):
        d.w[f"decoder.{c}.weight"], d.w[f"decoder.{c}.bias"] = torch.empty(1, 1, 3), torch.empty(1)
    for name, cin, cout, up in DECODER_BLOCKS:
        ci = D._pad16(cin)
        d.gb_pad[name] = ci - cin
        conv(name + ".conv1", cout, ci, 3), conv(name + ".conv2", cout, cout, 3), conv(name + ".conv1x1", cout, ci, 1)
        if up:
            d.w[name + ".pool.weight"], d.w[name + ".pool.bias"] = torch.empty(ci, 1, 3), torch.empty(ci)
        for fc, n in ((".norm1.fc", 2 * ci), (".norm2.fc", 2 * cout)):
            d.bank_off[name + fc] = (off, n)
            off += n
    d.bank_wt, d.bank_b = torch.empty(128, off), torch.empty(off)
    D.Decoder._init_calls(d)

    lib, made = Library(), iter(range(1000, 9999))
    lib.at = threading.local()

    def stream(*a, **k):
        n = next(made)
        time.sleep(0.02)
        return types.SimpleNamespace(cuda_stream=n)

    monkeypatch.setattr(D, "_Model", lambda struct, held, create: types.SimpleNamespace(held=held, handle=1))
    monkeypatch.setattr(_lib, "lib", lambda: lib)
    monkeypatch.setattr(torch.cuda, "device", lambda *a: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "Stream", stream)
    monkeypatch.setattr(ops, "_stream", lambda: getattr(lib.at, "stream", 0))
    d.library = lib
    return d


def call(d):
    return d.forward(torch.zeros(512, FRAMES), torch.zeros(2 * FRAMES), torch.zeros(2 * FRAMES), torch.zeros(128))


def in_threads(*jobs):
    errors = []

    def run(job):
        try:
            job()
        except Exception as e:  # a thread's exception would be lost
            errors.append(repr(e))

    threads = [threading.Thread(target=run, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors


def test_first_use_from_several_threads(dec):
    """A thread that finds the model made finds everything that the call needs."""

    def late():
        while dec._model is None:
            time.sleep(0.001)
        call(dec)

    in_threads(lambda: call(dec), late, late)
    assert len(dec.library.calls) == 3 and all(side for _, side in dec.library.calls)


def test_every_calling_stream_has_a_side_stream_of_its_own(dec):
    """Also when the new stream that torch hands out is one that a caller uses already."""

    def on(stream):
        def job():
            dec.library.at.stream = stream
            for _ in range(3):
                call(dec)
        return job

    in_threads(*(on(s) for s in (0, 7, 1000, 1002)))
    sides = {}
    for stream, side in dec.library.calls:
        assert sides.setdefault(stream, side) == side != stream
    assert len(sides) == len(set(sides.values())) == 4
    in_threads(*(on(s) for s in range(10, 50)))  # many short-lived callers: the store stays bounded
    assert len(dec._sides) == dec._MAX_SIDES
