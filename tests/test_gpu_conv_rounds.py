"""Convs whose tiles fill some rounds of the device and a little of one more: the columns that are over go as a launch of their own,
split over clusters (fullRounds in csrc/conv_tc.cu)."""
import pytest
import torch

from lokinfer_b200 import synth

pytestmark = pytest.mark.gpu

# c, l, k, d: tiles of one CTA and of pairs, one column and many over, rows that the TMA unit cannot address
CASES = [(128, 37889, 11, 1), (128, 38000, 11, 5), (256, 9473, 11, 5), (256, 19201, 11, 1), (512, 9500, 7, 3), (640, 7700, 7, 1)]


@pytest.mark.parametrize("plain", [False, True])
@pytest.mark.parametrize("c,l,k,d", CASES)
def test_conv_in_two_launches(cuda, c, l, k, d, plain):
    from lokinfer_b200 import ops
    x, w, b, affine, alpha, res = (torch.from_numpy(v).to(cuda) for v in synth.conv_case(c, c, l, k, c + l + k))
    state = ops.conv1d_prepare_f32_cuda(w)
    pad = d * (k - 1) // 2
    ops.set_conv_io("plain" if plain else "tma")
    try:
        out, stats = ops.conv1d_snake_f32_cuda(x, w, b, affine, alpha, residual=res, padding=pad, dilation=d, state=state)
    finally:
        ops.set_conv_io("tma")
    assert ops.conv_tc_status() == 0

    mean, scale, beta = affine.double()[:, :, None]
    v = (x.double() - mean) * scale + beta
    a = alpha.double()[:, None]
    v = torch.nn.functional.pad(v + torch.sin(a * v) ** 2 / a, (pad, pad))
    ref, size = res.double() + b.double()[:, None], res.double().abs() + b.double().abs()[:, None]
    for i in range(k):
        win, wi = v[:, i * d:i * d + l], w[:, :, i].double()
        ref += wi @ win
        size += wi.abs() @ win.abs()
    # a product's halves lose 2^-22 of it, a chain of up to 24 MMAs 2^-23 of its sum at each, the activation a few 2^-23 of its value
    assert (out.double() - ref).abs().le(2.0 ** -18 * size).all()
    n = (l + 127) // 128
    o = torch.nn.functional.pad(out.double(), (0, n * 128 - l)).view(c, n, 128)
    live = (torch.arange(n * 128, device=cuda) < l).view(1, n, 128)
    m = o.sum(2) / live.sum(2)
    m2 = ((o - m[:, :, None]) ** 2 * live).sum(2)
    rms = (o ** 2).sum(2)  # what 128 additions in f32 may lose of it
    assert (stats[..., 0].double() - m).abs().le(2.0 ** -16 * (1 + rms.sqrt())).all()
    assert (stats[..., 1].double() - m2).abs().le(2.0 ** -16 * (1 + rms)).all()


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
