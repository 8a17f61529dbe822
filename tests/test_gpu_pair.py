"""Convs on CTA pairs (csrc/conv_pair.cu): whole pairs of output-channel blocks, 16-byte aligned rows, too many tiles to be split.

The form is a matter of speed alone. At 128 columns the products, drains and order of sums are those of the form of one CTA, which
the 4-byte route takes: results are bit-identical to those, which the other tests hold to the oracle. At 160 columns residuals are
added behind other drains and statistics are per 32 columns: results agree to rounding."""
import ctypes

import pytest
import torch

from lokinfer_b200 import _lib, synth

pytestmark = pytest.mark.gpu



def pair_cols(ci, co, lo, k, d, act=1, fine=False, behind=False):
    """Columns per pair tile that the library's rule gives on this device, or 0."""
    sms, clusters = ctypes.c_int(0), (ctypes.c_int32 * 9)()
    assert _lib.lib().lkc_conv1d_tc_device(ctypes.byref(sms), clusters) == 0
    return _lib.lib().lkc_conv1d_tc_pair_cols(ci, co, lo, k, d, d * (k - 1) // 2, act, fine, behind, 100, sms.value, clusters)


# ci, co, l, k, d of convs that take pairs with any activation: one chunk, a chunk for one of the two groups of producer warps, tiles of
# 128 columns with whole, one-column and empty last halves, rounds of pairs that are full, two and three rounds, the widest window, K
# of one and two tap groups and more than eight
TAKEN = [(16, 256, 4737, 3, 1), (16, 256, 9472, 11, 5), (32, 256, 9472, 16, 1), (48, 256, 4737, 7, 3), (64, 768, 3000, 9, 1),
         (128, 256, 20100, 2, 3), (128, 512, 9537, 7, 5), (256, 256, 4864, 3, 1), (256, 256, 9472, 11, 5)]
# With Snake: two and three rounds of few chunks, a pointwise conv, whole rounds
TAKEN_SNAKE = [(48, 256, 19201, 5, 3), (64, 256, 28000, 3, 1), (256, 256, 9600, 1, 1), (512, 512, 9472, 5, 1), (1104, 1024, 2368, 1, 1),
               (256, 256, 18944, 3, 1)]
# Wherever the rule draws its line: also these, in one form or the other
CASES = [(16, 256, 9600, 3, 1), (48, 256, 4737, 7, 3), (256, 256, 4864, 3, 1), (256, 256, 9472, 11, 5), (256, 256, 9473, 11, 1),
         (128, 512, 9537, 7, 5), (256, 256, 9600, 1, 1), (32, 256, 20100, 2, 3), (64, 768, 6000, 9, 1), (32, 256, 9500, 16, 1)]


def _case(cuda, ci, co, l, k):
    from lokinfer_b200 import ops
    x, w, b, affine, alpha, res = (torch.from_numpy(v).to(cuda) for v in synth.conv_case(ci, co, l, k, ci + co + l + k))
    state = ops.conv1d_prepare_f32_cuda(w)
    assert state is not None
    return x, w, b, affine, alpha, res, state


@pytest.mark.parametrize("variant", ["snake", "snake_res", "leaky_res_scaled", "affine"])
@pytest.mark.parametrize("ci,co,l,k,d", TAKEN + TAKEN_SNAKE + [c for c in CASES if c not in TAKEN + TAKEN_SNAKE])
def test_pair_form_changes_no_bit(cuda, ci, co, l, k, d, variant):
    from lokinfer_b200 import ops
    x, w, b, affine, alpha, res, state = _case(cuda, ci, co, l, k)

    def call(xx, rr):
        kw = dict(padding=d * (k - 1) // 2, dilation=d, state=state)
        if variant == "affine":
            return ops.conv1d_affine_f32_cuda(xx, w, b, affine, **kw)
        if variant == "leaky_res_scaled":
            return ops.conv1d_leaky_f32_cuda(xx, w, b, affine, slope=0.2, residual=rr, out_scale=0.7071067811865476, **kw)
        return ops.conv1d_snake_f32_cuda(xx, w, b, affine, alpha, residual=rr if variant == "snake_res" else None, **kw)

    lo = l + 2 * (d * (k - 1) // 2) - d * (k - 1)
    act = {"affine": 0, "leaky_res_scaled": 2}.get(variant, 1)
    if (ci, co, l, k, d) in TAKEN or act == 1 and (ci, co, l, k, d) in TAKEN_SNAKE:
        assert pair_cols(ci, co, lo, k, d, act) == 128
    res = res[:, :lo].contiguous()
    ops.set_conv_io("plain")
    try:
        ref, ref_stats = call(x, res)
    finally:
        ops.set_conv_io("tma")
    with ops.padded_rows():
        px, pres = ops.to_cuda(x.cpu().numpy(), cuda, rows=True), ops.to_cuda(res.cpu().numpy(), cuda, rows=True)
        out, stats = call(px, pres)
    assert ops.conv_tc_status() == 0
    assert torch.equal(out, ref)
    assert torch.equal(stats, ref_stats)


@pytest.mark.parametrize("k", [3, 7, 11])
@pytest.mark.parametrize("l", [4737, 4800, 9601, 11840, 11841, 20801])
def test_pair_form_in_a_resblock(cuda, l, k):
    """Tiles of 160 columns with a pair of statistics per 32, which only whole-block calls take. Every element is looked at: a column
    that is wrong at an edge of a tile or of its halves is lost in the norm."""
    for d in (1, 3, 5):
        assert pair_cols(256, 256, l, k, d, fine=True, behind=True) == (160 if l != 11841 or k == 3 else 0)
    import numpy as np
    from lokinfer_b200 import ops
    from lokinfer_b200.generator import Generator
    gen = Generator(synth.generator_weights(3), cuda)
    r = np.random.default_rng(l)
    with ops.padded_rows():
        x = ops.to_cuda(r.standard_normal((256, l), dtype=np.float32), cuda, rows=True)
        gb = gen.style(torch.from_numpy(r.standard_normal(128, dtype=np.float32)).to(cuda))
        out, _ = gen.adain_resblock1_fused(x, gb, f"resblocks.{k // 4}", k)
        ops.set_conv_io("plain")
        try:
            ref, _ = gen.adain_resblock1_fused(x, gb, f"resblocks.{k // 4}", k)
        finally:
            ops.set_conv_io("tma")
    assert ops.conv_tc_status() == 0
    # the order in which 6 convs' residuals and statistics are added: a few units of the last place each
    assert torch.linalg.vector_norm(out - ref) <= 2e-6 * torch.linalg.vector_norm(ref)
    # an element: eight times that share of its row's root mean square
    assert ((out - ref).abs() <= 16e-6 * ref.square().mean(1, keepdim=True).sqrt()).all()


@pytest.mark.parametrize("ci,l", [(16, 4737), (48, 9473)])
def test_pairs_leave_nothing_behind_for_the_next_launch(cuda, ci, l):
    """A pair's CTAs leave when every signal for their shared memory has come, the second CTA's last ones to the first too. Launches back
    to back whose last tiles have one column, so that the two CTAs are far apart when they end, in turn with another form that takes
    over the shared memory; all give the bits of the first."""
    from lokinfer_b200 import ops
    x, w, b, affine, _, _, state = _case(cuda, ci, 256, l, 3)
    few = ops.to_cuda(x[:, :300].cpu().numpy(), cuda)  # split over clusters
    with ops.padded_rows():
        px = ops.to_cuda(x.cpu().numpy(), cuda, rows=True)
        kw = dict(padding=1, state=state)
        outs = [(ops.conv1d_affine_f32_cuda(px, w, b, affine, **kw), ops.conv1d_affine_f32_cuda(few, w, b, affine, **kw))
                for _ in range(60)]
    assert ops.conv_tc_status() == 0
    for pair, split in outs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(pair + split, outs[0][0] + outs[0][1]))
