"""lkc_generator_create: everything that the forward's sequence takes for granted is checked once, on the host. Pointers
here are never dereferenced; prepared states are real (host objects)."""
import ctypes

import pytest
import torch

from lokinfer_b200 import _lib

ADDR, BANK_N = 4096, 100000


class Weights:
    def __init__(self):
        self.lib, self.states, self.m = _lib.lib(), [], _lib.LkcGenerator()
        m = self.m
        m.bank_wt = m.bank_b = m.post_w = m.post_b = m.ident128 = ADDR
        m.bank_n = BANK_N
        m.post_state = self.conv(22, 128, 7)
        for i, (c, ci, up, rows, taps, stride) in enumerate(((256, 512, 10, 144, 2, 6), (128, 256, 6, 32, 1, 1))):
            n = m.noise_conv[i]
            n.w = n.b = ADDR
            n.state, n.stride, n.padding, n.taps, n.rows = self.conv(c, rows, taps), stride, 0, taps, rows
            m.ups_b[i], m.ups_state[i] = ADDR, self.convt(ci, c, up)
            for blk, k in ((m.noise_res[i], (7, 11)[i]), *((m.res[3 * i + j], k) for j, k in enumerate((3, 7, 11)))):
                blk.c, blk.k = c, k
                for j in range(6):
                    blk.w[j] = blk.b[j] = blk.alpha[j] = ADDR
                    blk.state[j], blk.gb[j] = self.conv(c, c, k), BANK_N - 2 * c

    def conv(self, co, ci, k):
        self.states.append(self.lib.lkc_conv1d_state_create_as(ADDR, co, ci, k, 0))
        return self.states[-1]

    def convt(self, ci, co, up):
        self.states.append(self.lib.lkc_convt_state_create_as(ADDR, ci, co, 2 * up, up, up // 2, 0))
        return self.states[-1]

    def create(self):
        """None where the weights were accepted, else the message."""
        handle = self.lib.lkc_generator_create(ctypes.byref(self.m))
        if handle:
            self.lib.lkc_model_destroy(handle)
            return None
        return None if "cudaEventCreate" in _lib.last_error() else _lib.last_error()  # the first step after the checks

    def __del__(self):
        for st in self.states:
            self.lib.lkc_conv1d_state_destroy(st)


def test_weights_that_fit_are_accepted():
    w = Weights()
    assert w.create() is None
    w.m.res[2].state[3] = None  # the CUDA-core kernel serves that conv
    w.m.post_state = None
    assert w.create() is None


def _set(path, value):
    def change(w):
        obj = w.m
        for p in path[:-1]:
            obj = obj[p] if isinstance(p, int) else getattr(obj, p)
        if isinstance(path[-1], int):
            obj[path[-1]] = value(w) if callable(value) else value
        else:
            setattr(obj, path[-1], value(w) if callable(value) else value)
    return change


@pytest.mark.parametrize("change,message", [
    (_set(("res", 0, "c"), 128), "bad resblock"),  # stage 0 has 256 channels
    (_set(("noise_res", 1, "c"), 256), "bad resblock"),
    (_set(("res", 4, "gb", 5), BANK_N - 2 * 128 + 1), "bad resblock"),  # one float past the bank
    (_set(("res", 4, "gb", 0), -1), "bad resblock"),
    (_set(("bank_n",), BANK_N - 1), "bad resblock"),
    (_set(("res", 5, "state", 2), lambda w: w.conv(128, 128, 7)), "bad resblock"),  # k = 11 here
    (_set(("res", 5, "state", 2), lambda w: w.conv(128, 64, 11)), "bad resblock"),
    (_set(("noise_conv", 0, "state"), lambda w: w.conv(256, 144, 3)), "bad noise conv"),
    (_set(("noise_conv", 0, "state"), lambda w: w.conv(128, 144, 2)), "bad noise conv"),
    (_set(("noise_conv", 1, "rows"), 48), "bad noise conv"),  # not what the state was made for
    (_set(("noise_conv", 0, "stride"), 7), "bad noise conv"),
    (_set(("noise_conv", 0, "padding"), -1), "bad noise conv"),
    (_set(("ups_state", 0), lambda w: w.convt(512, 128, 10)), "bad upsampler"),
    (_set(("ups_state", 0), lambda w: w.convt(256, 256, 10)), "bad upsampler"),
    (_set(("ups_state", 1), lambda w: w.convt(256, 128, 10)), "bad upsampler"),
    (_set(("ups_state", 1), lambda w: w.conv(128, 256, 12)), "bad upsampler"),  # a conv's state
    (_set(("ups_state", 1), None), "bad upsampler"),
    (_set(("post_state",), lambda w: w.conv(22, 128, 5)), "bad conv_post"),
    (_set(("ident128",), None), "null weight"),
])
def test_weights_that_do_not_fit_are_refused(change, message):
    w = Weights()
    change(w)
    assert message in (w.create() or "")


def test_decoder_weights_are_checked():
    """lkc_decoder_create: states of the five blocks' shapes, AdaIN parameters inside the bank."""
    lib, states = _lib.lib(), []

    def conv(co, ci, k):
        states.append(lib.lkc_conv1d_state_create_as(ADDR, co, ci, k, 0))
        return states[-1]

    def create(change=lambda d: None):
        d = _lib.LkcDecoder()
        d.bank_wt = d.bank_b = d.f0_w = d.f0_b = d.n_w = d.n_b = d.asr_w = d.asr_b = ADDR
        d.bank_n, d.asr_state = BANK_N, conv(64, 512, 1)
        for i, b in enumerate(d.block):
            b.cin, b.cout, b.up = (528, 1104)[i > 0], 512 if i == 4 else 1024, int(i == 4)
            b.w1 = b.b1 = b.w2 = b.b2 = b.w1x1 = b.b1x1 = b.pool_w = b.pool_b = ADDR
            b.state1, b.state2, b.state1x1 = conv(b.cout, b.cin, 3), conv(b.cout, b.cout, 3), conv(b.cout, b.cin, 1)
            b.gb1, b.gb2 = BANK_N - 2 * b.cin, BANK_N - 2 * b.cout
        change(d)
        handle = lib.lkc_decoder_create(ctypes.byref(d))
        if handle:
            lib.lkc_model_destroy(handle)
            return None
        return None if "cudaEventCreate" in _lib.last_error() else _lib.last_error()

    def setter(path, value):
        def change(d):
            *head, last = path
            for p in head:
                d = d[p] if isinstance(p, int) else getattr(d, p)
            setattr(d, last, value)
        return change

    assert create() is None
    for path, value in ((("asr_state",), None), (("bank_n",), 100), (("block", 0, "cin"), 1104), (("block", 4, "up"), 0),
                        (("block", 2, "w1x1"), None), (("block", 4, "pool_w"), None), (("block", 1, "gb1"), BANK_N - 2207),
                        (("block", 3, "gb2"), -1), (("block", 1, "state2"), states[0])):
        assert "decoder_create" in (create(setter(path, value)) or ""), path
    for st in states:
        lib.lkc_conv1d_state_destroy(st)
