"""Operand formats of weight packs without a GPU: a format asked for is an argument down to the pack, and the process-wide
conv path stays as it is."""
import contextlib

import pytest
import torch

from lokinfer_b200 import _lib, decoder, ops, synth


@pytest.fixture
def no_gpu(monkeypatch):
    """Weight packs on CPU tensors: the launch is left out, sizes and states are the library's."""
    packs = []

    def run(name, operands, outs, attrs_int=(), **kw):
        packs.append((name, tuple(operands[0].shape), outs[0].numel(), tuple(attrs_int)))

    monkeypatch.setattr(ops, "_run", run)
    monkeypatch.setattr(ops, "conv_tc_status", lambda: 0)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    return packs


def test_decoder_leaves_the_conv_path_alone(no_gpu, monkeypatch):
    """The decoder's pointwise convs are packed in the tf32 format, the others in the current one, with no switch of the
    path on the way: another thread's packs and launches never see one."""
    switched = []
    monkeypatch.setattr(ops, "set_conv_path", lambda mode: switched.append(mode))
    dec = decoder.Decoder(synth.decoder_weights(0), "cpu")
    assert switched == [] and ops._conv_path == "auto"
    fmt = {n: st.fmt for n, st in dec.state.items()}
    assert {n for n, f in fmt.items() if f == "tf32"} == {n for n in fmt if n.endswith("conv1x1") or "asr_res" in n}
    assert all(f in ("f16", "tf32") for f in fmt.values())


def test_decoder_of_the_blocks_alone(no_gpu):
    """adain_resblk* need the blocks' weights only; asr_res, F0_conv and N_conv are forward()'s."""
    sd = synth.decoder_weights(0)
    dec = decoder.Decoder({n: v for n, v in sd.items() if n.startswith(("decoder.encode.", "decoder.decode."))}, "cpu")
    assert set(dec.state) == set(decoder.Decoder(sd, "cpu").state) - {"decoder.asr_res.0"}


def test_weight_beyond_f16_is_packed_again_without_a_switch(no_gpu, monkeypatch):
    switched = []
    monkeypatch.setattr(ops, "set_conv_path", lambda mode: switched.append(mode))
    monkeypatch.setattr(ops, "conv_tc_status", lambda: ops.STATUS_F16_WEIGHTS)
    assert ops.conv1d_prepare_f32_cuda(torch.zeros(32, 16, 3)).fmt == "tf32"
    assert ops.conv_transpose1d_prepare_f32_cuda(torch.zeros(32, 16, 12), 6, 3).fmt == "tf32"
    assert ops.conv1d_prepare_f32_cuda(torch.zeros(32, 16, 3), "f16").fmt == "f16"  # asked for: not second-guessed
    assert switched == []


def test_formats_of_a_pack():
    """Sizes by argument equal those of the path that stands for the format; unknown formats are refused."""
    lib = _lib.lib()
    for path, fmt in (("auto", 0), ("tf32", 2)):
        ops.set_conv_path(path)
        try:
            want = lib.lkc_conv1d_tc_pack_floats(200, 48, 5), lib.lkc_convt_tc_pack_floats(32, 40, 12, 6, 3)
        finally:
            ops.set_conv_path("auto")
        assert want == (lib.lkc_conv1d_tc_pack_floats_as(200, 48, 5, fmt), lib.lkc_convt_tc_pack_floats_as(32, 40, 12, 6, 3, fmt))
        assert min(want) > 0
    assert lib.lkc_conv1d_tc_pack_floats_as(200, 48, 5, 1) == 0 and lib.lkc_convt_tc_pack_floats_as(32, 40, 12, 6, 3, 1) == 0
    assert not lib.lkc_conv1d_state_create_as(4096, 200, 48, 5, 1)
    with pytest.raises(ops.OpError, match="fmt must be"):
        ops.conv1d_prepare_f32_cuda(torch.zeros(32, 16, 3), "bf16")
