"""The decoder AdainResBlk1d stack in front of the generator (models/kokoro/model.py:158-221, 704-717) on the GPU
against the CPU oracle: its three extra ops, each block type (basic and fused), and the whole stack's output dec_x."""
import math

import numpy as np
import pytest
import torch

from lokinfer_b200 import synth
from oracle import kokoro_oracle as O
from util import REL_L2, rel_l2, t32, t64

pytestmark = pytest.mark.gpu


def dev(cuda, *arrs):
    from lokinfer_b200 import ops
    return [ops.to_cuda(a, cuda) for a in arrs]


def test_decoder_side_ops(cuda):
    from lokinfer_b200 import ops
    r = np.random.default_rng(3)
    # depthwise ConvTranspose1d: (C, L, K, stride, padding, output_padding), incl. the pool of the upsampling block
    for c, l, k, s, p, op in [(1090, 37, 3, 2, 1, 1), (5, 1, 3, 2, 1, 1), (8, 33, 4, 2, 1, 0), (3, 10, 5, 3, 0, 2),
                              (16, 700, 3, 1, 1, 0)]:
        x = r.standard_normal((c, l)).astype(np.float32)
        w = r.standard_normal((c, 1, k)).astype(np.float32)
        b = r.standard_normal(c).astype(np.float32)
        got = ops.conv_transpose1d_dw_f32_cuda(*dev(cuda, x, w, b), stride=s, padding=p, output_padding=op).cpu().numpy()
        ref = O.conv_transpose1d_dw(t64(x), t64(w), t64(b), stride=s, padding=p, output_padding=op).numpy()
        assert got.shape == ref.shape == (c, (l - 1) * s - 2 * p + k + op)
        np.testing.assert_allclose(got, ref, atol=1e-5, rtol=1e-5)
    for c, l, sc in [(7, 13, 2), (1104, 40, 2), (3, 5, 1), (2, 9, 3)]:
        x = r.standard_normal((c, l)).astype(np.float32)
        got = ops.upsample_nearest1d_f32_cuda(dev(cuda, x)[0], sc).cpu().numpy()
        np.testing.assert_array_equal(got, O.upsample_nearest1d(t32(x), sc).numpy())
    parts = [r.standard_normal((n, 21)).astype(np.float32) for n in (1024, 64, 1, 1, 14)]
    got = ops.concat_rows_f32_cuda(*dev(cuda, *parts)).cpu().numpy()
    np.testing.assert_array_equal(got, np.concatenate(parts, 0))
    with pytest.raises(ops.OpError):
        ops.concat_rows_f32_cuda(dev(cuda, parts[0])[0])


@pytest.mark.parametrize("frames", [9, 40, 160])
@pytest.mark.parametrize("fused", [True, False])
def test_decoder_vs_oracle(cuda, frames, fused):
    """dec_x [512, 2F] (the generator's input) for F frames. Ten chained convs of 514 .. 1090 input channels: the
    per-op bar compounds, the float64 oracle is the arbiter (GPU error within 2x the float32 oracle's own)."""
    from lokinfer_b200 import Decoder, ops
    sd = synth.decoder_weights(0)
    inp = synth.decoder_inputs(frames, 5 + frames)
    dec = Decoder(sd, cuda)
    a = dev(cuda, inp["asr"], inp["f0"], inp["n"], inp["s"])
    got = dec.forward(*a, fused=fused).cpu().numpy()
    assert got.shape == (512, 2 * frames)
    r32 = O.decoder(sd, *[O.T(inp[k]) for k in ("asr", "f0", "n", "s")], fused=fused).numpy()
    dt = torch.float64
    r64 = O.decoder(sd, *[O.T(inp[k], dt) for k in ("asr", "f0", "n", "s")], fused=fused).numpy()
    assert rel_l2(got, r32) <= 10 * REL_L2
    assert rel_l2(got, r64) <= 2 * rel_l2(r32, r64) + 1e-6
    assert ops.conv_tc_status() == 0
    if fused:  # every conv of the fused stack has a prepared tensor-core state (padded input channels)
        assert all(st is not None for st in dec.state.values())


def test_decoder_feeds_generator(cuda):
    """dec_x goes straight into the generator: decoder -> generator on the device equals the oracle's chain."""
    from lokinfer_b200 import Decoder, Generator, ops
    frames = 8
    dsd, gsd = synth.decoder_weights(0), synth.generator_weights(0)
    inp = synth.decoder_inputs(frames, 2)
    gin = synth.generator_inputs(2 * frames, 4)
    dec, gen = Decoder(dsd, cuda), Generator(gsd, cuda)
    x = dec.forward(*dev(cuda, inp["asr"], inp["f0"], inp["n"], inp["s"]))
    audio = gen.forward(x, *dev(cuda, gin["har"], inp["s"])).cpu().numpy()
    rx = O.decoder(dsd, *[O.T(inp[k]) for k in ("asr", "f0", "n", "s")])
    ref = O.generator(gsd, rx, O.T(gin["har"]), O.T(inp["s"])).numpy()
    assert audio.shape == ref.shape == (600 * frames,)
    assert np.abs(audio - ref).max() <= 1e-4


@pytest.fixture(scope="module")
def dec(cuda):
    from lokinfer_b200 import Decoder
    return Decoder(synth.decoder_weights(0), cuda)


def _composed(dec, *a):
    """The op-by-op form: a result allocator of one's own makes the whole call stand back."""
    from lokinfer_b200 import ops
    with ops.use_allocator(lambda shape, device: torch.empty(shape, dtype=torch.float32, device=device)):
        return dec.forward(*a)


def _args(cuda, frames, seed):
    inp = synth.decoder_inputs(frames, seed)
    return dev(cuda, inp["asr"], inp["f0"], inp["n"], inp["s"])


@pytest.mark.parametrize("frames", [1, 2, 3, 61, 64, 127, 129, 300, 1040])
def test_whole_decoder_agrees_with_the_composition(cuda, dec, frames):
    """The whole call differs from the op-by-op form in who computes the statistics and in how partial sums are split, not
    beyond rounding: within the 1e-5 of one op. Against float64 it is no further off than the composition is, within 1e-5 but at
    two columns, where the variance of two samples in front of 1 / sqrt(var + eps) magnifies the rounding of both alike."""
    from lokinfer_b200 import ops
    inp = synth.decoder_inputs(frames, 30 + frames)
    a = dev(cuda, inp["asr"], inp["f0"], inp["n"], inp["s"])
    got, want = dec.forward(*a), _composed(dec, *a)
    assert got.shape == want.shape == (512, 2 * frames) and got.is_contiguous()
    assert rel_l2(got.cpu().numpy(), want.cpu().numpy()) <= REL_L2
    assert torch.equal(got, dec.forward(*a)) and ops.conv_tc_status() == 0
    r64 = O.decoder(synth.decoder_weights(0), *[O.T(inp[k], torch.float64) for k in ("asr", "f0", "n", "s")]).numpy()
    err, err_ops = rel_l2(got.cpu().numpy(), r64), rel_l2(want.cpu().numpy(), r64)
    assert err <= 1.2 * err_ops + 1e-7 and (err <= REL_L2 or frames == 2)


@pytest.mark.parametrize("frames", [32, 33, 65, 128, 256, 257, 384, 385])
def test_whole_decoder_at_other_tile_counts(cuda, dec, frames):
    """The lengths where the width of the tiles and the shares of the SMs change."""
    test_whole_decoder_agrees_with_the_composition(cuda, dec, frames)


def test_whole_decoder_takes_row_pitches_and_leaves_the_rest(cuda, dec):
    """A view of wider rows, a stream of the caller's, replaced weights; operands that the call cannot take by their
    addresses go op by op or are refused as before."""
    from lokinfer_b200 import Decoder, ops
    a = _args(cuda, 50, 7)
    want = dec.forward(*a)
    wide = torch.full((512, 56), float("nan"), device=cuda)
    wide[:, :50] = a[0]
    with ops.padded_rows():
        got = dec.forward(wide[:, :50], *a[1:])
    assert torch.equal(got, want)
    with torch.cuda.stream(torch.cuda.Stream(device=cuda)):
        torch.cuda.current_stream().wait_stream(torch.cuda.default_stream(cuda))
        got = dec.forward(*a)
        torch.cuda.current_stream().synchronize()
    assert torch.equal(got, want)
    for bad in ([a[0][:, :49], *a[1:]], [a[0].cpu(), *a[1:]], [a[0].double(), *a[1:]], [a[0], a[1][:-1], a[2], a[3]]):
        with pytest.raises((ops.OpError, RuntimeError)):
            dec.forward(*bad)
    other = Decoder(synth.decoder_weights(0), cuda)
    other.forward(*a)
    other.w["decoder.encode.conv2.bias"] = other.w["decoder.encode.conv2.bias"] + 1.0
    got, want2 = other.forward(*a), _composed(other, *a)
    assert rel_l2(got.cpu().numpy(), want2.cpu().numpy()) <= REL_L2 and rel_l2(got.cpu().numpy(), want.cpu().numpy()) > 1e-3


@pytest.mark.parametrize("cold", [False, True])
def test_one_decoder_in_several_threads(cuda, dec, cold):
    """cold: the threads are the decoder's first users."""
    import threading

    from lokinfer_b200 import Decoder
    jobs = [_args(cuda, f, f) for f in (5, 61, 200)]
    want = [dec.forward(*j).clone() for j in jobs]
    torch.cuda.synchronize()
    user = Decoder(synth.decoder_weights(0), cuda) if cold else dec
    start, right, errors = threading.Barrier(3), [0, 0, 0], []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream(device=cuda)):
                start.wait(60)
                for _ in range(10):
                    right[i] += torch.equal(user.forward(*jobs[i]), want[i])
        except Exception as e:  # a thread's exception would be lost
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and right == [10, 10, 10]


def test_whole_decoder_in_a_graph(cuda, dec):
    a = _args(cuda, 61, 3)
    want = dec.forward(*a).clone()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = dec.forward(*a)
    out.zero_()
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)


@pytest.mark.parametrize("one_side", [False, True])
def test_a_capture_beside_a_call_of_another_thread(cuda, dec, monkeypatch, one_side):
    """While one thread captures a forward, another runs one: the call works and the capture stays valid. one_side: both are
    handed the same side stream, which is then in the first one's capture."""
    import threading
    a, b = _args(cuda, 61, 3), _args(cuda, 200, 4)
    want = [dec.forward(*x).clone() for x in (a, b)]
    streams = [torch.cuda.Stream(device=cuda) for _ in range(2)]
    if one_side:
        side = torch.cuda.Stream(device=cuda)
        monkeypatch.setattr(dec, "_side_stream", lambda caller: side.cuda_stream)
    torch.cuda.synchronize()
    captured, done = threading.Event(), threading.Event()
    got, errors = [], []

    def other():
        try:
            assert captured.wait(60)
            with torch.cuda.stream(streams[1]):
                got.append(dec.forward(*b))
        except Exception as e:  # a thread's exception would be lost
            errors.append(repr(e))
        finally:
            done.set()

    t, g = threading.Thread(target=other), torch.cuda.CUDAGraph()
    t.start()
    with torch.cuda.graph(g, stream=streams[0], capture_error_mode="thread_local"):
        out = dec.forward(*a)
        captured.set()
        assert done.wait(60)
        again = dec.forward(*a)  # the same capture a second time
    t.join()
    torch.cuda.synchronize()
    assert not errors and torch.equal(got[0], want[1])
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want[0]) and torch.equal(again, want[0])
