"""Convs whose tiles fill some rounds of the device and a little of one more: the columns that are over go as a launch of their own,
split over clusters (fullRounds in csrc/conv_tc.cu)."""
import ctypes

import pytest
import torch

from lokinfer_b200 import _lib, synth

pytestmark = pytest.mark.gpu

# c, l, k, d: tiles of one CTA and (512 channels, K = 5 and 11) of pairs, one column and many over, rows that the TMA unit cannot address
CASES = [(128, 37889, 11, 1), (128, 38000, 11, 5), (256, 18945, 11, 5), (256, 19201, 11, 1), (512, 9500, 7, 3), (512, 9600, 5, 1),
         (512, 9473, 11, 1), (640, 7700, 7, 1)]


def full_rounds(c, lo, k):
    """Columns of the first of two launches by the library's rule on this device, or 0."""
    sms, clusters = ctypes.c_int(0), (ctypes.c_int32 * 9)()
    assert _lib.lib().lkc_conv1d_tc_device(ctypes.byref(sms), clusters) == 0
    return _lib.lib().lkc_conv1d_tc_full_rounds(c, c, lo, k, sms.value, clusters)


def _reference(x, w, b, affine, alpha, res, k, d):
    """The conv in float64 and, for error bounds, the same sums of magnitudes."""
    pad, l = d * (k - 1) // 2, x.shape[1]
    mean, scale, beta = affine.double()[:, :, None]
    v = (x.double() - mean) * scale + beta
    a = alpha.double()[:, None]
    v = torch.nn.functional.pad(v + torch.sin(a * v) ** 2 / a, (pad, pad))
    ref, size = res.double() + b.double()[:, None], res.double().abs() + b.double().abs()[:, None]
    for i in range(k):
        win, wi = v[:, i * d:i * d + l], w[:, :, i].double()
        ref += wi @ win
        size += wi.abs() @ win.abs()
    return ref, size


def _check(out, stats, ref, size):
    c, l = out.shape
    # a product's halves lose 2^-22 of it, a chain of up to 24 MMAs 2^-23 of its sum at each, the activation a few 2^-23 of its value
    assert (out.double() - ref).abs().le(2.0 ** -18 * size).all()
    n = (l + 127) // 128
    o = torch.nn.functional.pad(out.double(), (0, n * 128 - l)).view(c, n, 128)
    live = (torch.arange(n * 128, device=out.device) < l).view(1, n, 128)
    m = o.sum(2) / live.sum(2)
    m2 = ((o - m[:, :, None]) ** 2 * live).sum(2)
    rms = (o ** 2).sum(2)  # what 128 additions in f32 may lose of it
    assert (stats[..., 0].double() - m).abs().le(2.0 ** -16 * (1 + rms.sqrt())).all()
    assert (stats[..., 1].double() - m2).abs().le(2.0 ** -16 * (1 + rms)).all()


@pytest.mark.parametrize("plain", [False, True])
@pytest.mark.parametrize("c,l,k,d", CASES)
def test_conv_in_two_launches(cuda, c, l, k, d, plain):
    from lokinfer_b200 import ops
    x, w, b, affine, alpha, res = (torch.from_numpy(v).to(cuda) for v in synth.conv_case(c, c, l, k, c + l + k))
    state = ops.conv1d_prepare_f32_cuda(w)
    pad = d * (k - 1) // 2
    ops.set_conv_io("plain" if plain else "tma")
    try:
        with ops.Profile(time_kernels=False) as prof:
            out, stats = ops.conv1d_snake_f32_cuda(x, w, b, affine, alpha, residual=res, padding=pad, dilation=d, state=state)
    finally:
        ops.set_conv_io("tma")
    assert full_rounds(c, l, k) > 0 and prof.count == 2
    assert ops.conv_tc_status() == 0
    _check(out, stats, *_reference(x, w, b, affine, alpha, res, k, d))


# c, l, cut, k, d: a first part of two launches (pairs and one CTA's tiles) and a second one of pairs or one CTA's tiles; pairs in both
@pytest.mark.parametrize("c,l,cut,k,d,two", [(512, 14800, 9600, 5, 1, True), (256, 34000, 19200, 11, 5, True),
                                             (256, 20001, 9472, 3, 1, False), (512, 15001, 9856, 11, 5, True)])
@pytest.mark.parametrize("pitch", [0, 1])  # rows on 16-byte boundaries, and not
def test_windows_in_two_launches_and_in_pairs(cuda, c, l, cut, k, d, two, pitch):
    """A row in two parts as the time-sharded path holds it: each part a window with real columns of its neighbour beside it, what lies
    beyond the utterance not zero, its statistics a slice of the whole row's."""
    from lokinfer_b200 import ops
    x, w, b, affine, alpha, res = (torch.from_numpy(v).to(cuda) for v in synth.conv_case(c, c, l, k, c + l + k))
    state = ops.conv1d_prepare_f32_cuda(w)
    pad, m, n, p = d * (k - 1) // 2, 64, -(-l // 128), (l + 3) // 4 * 4 + pitch
    assert (full_rounds(c, cut, k) > 0) == two
    rows = lambda t: torch.nn.functional.pad(t, (0, p - t.shape[1]))
    out, stats, dres = torch.full((c, p), 9.0, device=cuda), torch.full((c, n + 3, 2), 9.0, device=cuda), rows(res)
    filler = torch.full((c, m), 3.0, device=cuda)
    for lo, hi in ((0, cut), (cut, l)):
        left, right = (filler if lo == 0 else x[:, lo - m:lo]), (filler if hi == l else x[:, hi:hi + m])
        buf = torch.cat([left, x[:, lo:hi], right], 1)
        width = buf.shape[1]
        buf = torch.nn.functional.pad(buf, (0, -width % 4 + pitch), value=5.0)[:, :width]
        with ops.Profile(time_kernels=False) as prof:
            ops._run("conv1d_snake_res_f32_cuda", [buf, w, b, affine, alpha, dres[:, lo:hi]],
                     [out[:, lo:hi], stats[:, lo // 128:-(-hi // 128)]], attrs_int=[d, pad, ops.conv_tile(c, k)], state=state.handle,
                     window=[n + 3, m, m if lo == 0 else 0, m + hi - lo if hi == l else width])
        assert prof.count == (2 if full_rounds(c, hi - lo, k) else 1)
    assert ops.conv_tc_status() == 0
    _check(out[:, :l], stats[:, :n], *_reference(x, w, b, affine, alpha, res, k, d))
    assert (stats[:, n:] == 9).all()


def test_both_launches_are_counted(cuda):
    from lokinfer_b200 import ops
    from lokinfer_b200.generator import Generator
    x, w, b, affine, alpha, res = (torch.from_numpy(v).to(cuda) for v in synth.conv_case(256, 256, 19201, 11, 1))
    state = ops.conv1d_prepare_f32_cuda(w)
    with ops.Profile(time_kernels=False) as one:
        ops.conv1d_snake_f32_cuda(x[:, :9472].contiguous(), w, b, affine, alpha, padding=5, state=state)
    with ops.Profile(time_kernels=False) as two:
        ops.conv1d_snake_f32_cuda(x, w, b, affine, alpha, residual=res, padding=5, state=state)
    assert (one.count, two.count) == (1, 2)
    gen = Generator(synth.generator_weights(3), cuda)
    gb = gen.style(torch.zeros(128, device=cuda))
    counts = []
    for l in (19201, 18944):
        with ops.Profile(time_kernels=False) as prof:
            gen.adain_resblock1_fused(x[:, :l].contiguous(), gb, "resblocks.2", 11)
        counts.append(prof.count)
    assert counts == [14, 13]  # statistics, six affines and convs; the last one, whose statistics are per 128 columns, in two launches
