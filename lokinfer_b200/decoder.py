"""The decoder in front of the Kokoro generator, wired from `ops.*_cuda`: five AdainResBlk1d blocks that turn the
aligned text features, the pitch curve and the energy curve into the generator's input x [512, 2F]
(models/kokoro/model.py:158-221 the blocks, :704-717 the stack). Same op sequence as the reference's CPU graph, fused
(stats -> adain_affine -> conv1d_leaky, :205-221) or basic (:158-174). forward() is one library call that works on block
inputs in place (lkc_decoder_forward); the composition from single ops, which concatenates them, stands behind it.

Its convs have 514 / 1090 / 1024 input channels and kernel size 3. The tensor-core kernel stages 16 input channels at
a time, so the two odd counts are padded: the block inputs get zero rows up to the next multiple of 16 and the weights /
AdaIN parameters, once, when they are uploaded, zero columns to match. A zero row has mean 0 and variance 0, its activation is the finite AdaIN bias, and it meets a zero weight:
the padding contributes exact zeros and every conv of the stack runs on tcgen05.
"""
from __future__ import annotations

import ctypes
import operator
import threading

import numpy as np
import torch

from . import _lib, ops
from .generator import _Held, _Model
from .synth import DECODER_BLOCKS

SQRT1_2 = 0.7071067811865476


def _pad16(c: int) -> int:
    return -(-c // 16) * 16


class Decoder:
    def __init__(self, sd: dict, device="cuda"):
        self.device = torch.device(device)
        w = {k: ops.to_cuda(np.ascontiguousarray(v, dtype=np.float32), self.device) for k, v in sd.items()}
        self.w, self.state = w, {}
        self.gb_pad = {}  # block -> channels appended to norm1's (gamma, beta)
        for name, cin, cout, up in DECODER_BLOCKS:
            cp = _pad16(cin)
            if cp != cin:  # zero input channels / zero AdaIN parameters for the appended rows
                z = cp - cin
                w[name + ".conv1.weight"] = torch.cat(
                    [w[name + ".conv1.weight"], torch.zeros(cout, z, 3, device=self.device)], 1).contiguous()
                if cin != cout:
                    w[name + ".conv1x1.weight"] = torch.cat(
                        [w[name + ".conv1x1.weight"], torch.zeros(cout, z, 1, device=self.device)], 1).contiguous()
                if up:
                    w[name + ".pool.weight"] = torch.cat(
                        [w[name + ".pool.weight"], torch.zeros(z, 1, 3, device=self.device)], 0).contiguous()
                    w[name + ".pool.bias"] = torch.cat([w[name + ".pool.bias"], torch.zeros(z, device=self.device)])
            self.gb_pad[name] = cp - cin
            for conv in (".conv1", ".conv2"):
                self.state[name + conv] = ops.conv1d_prepare_f32_cuda(w[name + conv + ".weight"])
            if cin != cout:
                self.state[name + ".conv1x1"] = ops.conv1d_prepare_f32_cuda(w[name + ".conv1x1.weight"], "tf32")
                w[name + ".conv1x1.bias"] = torch.zeros(cout, device=self.device)
        if "decoder.asr_res.0.weight" in w:  # only forward() needs it: a state dict of the blocks is enough for adain_resblk*
            self.state["decoder.asr_res.0"] = ops.conv1d_prepare_f32_cuda(w["decoder.asr_res.0.weight"], "tf32")
        # style bank: every `<name>.fc` of the decoder as one GEMV (models/kokoro/model.py:67-81, names sorted)
        names = sorted(k[: -len(".weight")] for k in w if k.endswith(".fc.weight"))
        # The (gamma | beta) of a norm1 carry their zeros for the appended rows: gamma, zeros, beta, zeros.
        self.bank_off, o, wt, bias = {}, 0, [], []
        for n in names:
            pad = self.gb_pad.get(n[: -len(".norm1.fc")], 0) if n.endswith(".norm1.fc") else 0
            for t, parts in ((w[n + ".weight"], wt), (w[n + ".bias"], bias)):
                c = int(t.shape[0]) // 2
                z = torch.zeros(pad, *t.shape[1:], device=self.device)
                parts += [t[:c], z, t[c:], z]
            self.bank_off[n] = (o, int(w[n + ".bias"].shape[0]) + 2 * pad)
            o += self.bank_off[n][1]
        self.bank_wt = torch.cat(wt).t().contiguous()
        self.bank_b = torch.cat(bias).contiguous()
        self._ident = {c: torch.stack([torch.zeros(c), torch.ones(c), torch.zeros(c)]).to(self.device).contiguous()
                       for c in {512} | {_pad16(cin) for _, cin, _, _ in DECODER_BLOCKS}}
        self._init_calls()

    def _init_calls(self):
        self._model = None  # _Model of the whole-forward call
        self._sides = {}  # calling stream -> the stream of its shortcuts (_side_stream)

    # The forward as one library call (lkc_decoder_forward). It computes what the composition in forward() computes with a
    # third of its launches (block inputs are never concatenated, statistics come from the convs that wrote the rows), the
    # shortcuts beside the convs, and no trip through Python per kernel: 48 op calls took 1.7 ms at any length. The
    # composition remains for single kernels (ops.Profile with timing, ops.tracing), the CUDA-core path, convs without a
    # tensor-core state and operands that the whole call would not check.

    _NAMES = tuple(["decoder.asr_res.0.weight", "decoder.asr_res.0.bias"]
                   + [f"decoder.{c}.{p}" for c in ("F0_conv", "N_conv") for p in ("weight", "bias")]
                   + [f"{name}.{p}" for name, _, _, up in DECODER_BLOCKS
                      for p in ["conv1.weight", "conv1.bias", "conv2.weight", "conv2.bias", "conv1x1.weight", "conv1x1.bias"]
                      + (["pool.weight", "pool.bias"] if up else [])])
    _STATES = tuple(["decoder.asr_res.0"]
                    + [f"{name}.{c}" for name, _, _, _ in DECODER_BLOCKS for c in ("conv1", "conv2", "conv1x1")])
    _GET_W, _GET_S = operator.itemgetter(*_NAMES), operator.itemgetter(*_STATES)

    def _is(self, t, *shape):
        return tuple(t.shape) == shape and t.dtype == torch.float32 and t.is_contiguous() and t.device == self.bank_b.device

    def _whole_model(self):
        """_Model of lkc_decoder_forward, or None when some conv has no tensor-core state."""
        try:
            ws, states = self._GET_W(self.w), self._GET_S(self.state)
        except KeyError:
            return None
        pieces = (*ws, *states, self.bank_wt, self.bank_b, self.bank_off)
        model = self._model
        if model is not None and model.held.current(pieces):
            return model
        w, st, n = dict(zip(self._NAMES, ws)), dict(zip(self._STATES, states)), int(self.bank_b.shape[0])

        def has(conv, co, ci, k):
            s = st[conv]
            return s is not None and s.shape == (co, ci, k) and self._is(w[conv + ".weight"], co, ci, k) and self._is(w[conv + ".bias"], co)

        ok = (self._is(self.bank_wt, 128, n) and self._is(self.bank_b, n) and has("decoder.asr_res.0", 64, 512, 1)
              and all(self._is(w[f"decoder.{c}.weight"], 1, 1, 3) and self._is(w[f"decoder.{c}.bias"], 1)
                      for c in ("F0_conv", "N_conv")))
        d = _lib.LkcDecoder()
        for b, (name, cin, cout, up) in zip(d.block, DECODER_BLOCKS):
            ci = _pad16(cin)
            ok = (ok and has(name + ".conv1", cout, ci, 3) and has(name + ".conv2", cout, cout, 3)
                  and has(name + ".conv1x1", cout, ci, 1)
                  and (not up or (self._is(w[name + ".pool.weight"], ci, 1, 3) and self._is(w[name + ".pool.bias"], ci)))
                  and not bool(up and self.gb_pad[name] != ci - cin))
            (b.gb1, n1), (b.gb2, n2) = self.bank_off[name + ".norm1.fc"], self.bank_off[name + ".norm2.fc"]
            if not (ok and n1 == 2 * ci and n2 == 2 * cout):
                return None
            b.cin, b.cout, b.up = ci, cout, int(up)
            b.w1, b.b1 = w[name + ".conv1.weight"].data_ptr(), w[name + ".conv1.bias"].data_ptr()
            b.w2, b.b2 = w[name + ".conv2.weight"].data_ptr(), w[name + ".conv2.bias"].data_ptr()
            b.w1x1, b.b1x1 = w[name + ".conv1x1.weight"].data_ptr(), w[name + ".conv1x1.bias"].data_ptr()
            if up:
                b.pool_w, b.pool_b = w[name + ".pool.weight"].data_ptr(), w[name + ".pool.bias"].data_ptr()
            b.state1, b.state2, b.state1x1 = (st[name + c].handle for c in (".conv1", ".conv2", ".conv1x1"))
        d.bank_wt, d.bank_b, d.bank_n = self.bank_wt.data_ptr(), self.bank_b.data_ptr(), n
        d.f0_w, d.f0_b = w["decoder.F0_conv.weight"].data_ptr(), w["decoder.F0_conv.bias"].data_ptr()
        d.n_w, d.n_b = w["decoder.N_conv.weight"].data_ptr(), w["decoder.N_conv.bias"].data_ptr()
        d.asr_w, d.asr_b = w["decoder.asr_res.0.weight"].data_ptr(), w["decoder.asr_res.0.bias"].data_ptr()
        d.asr_state = st["decoder.asr_res.0"].handle
        with torch.cuda.device(self.bank_b.device):
            model = _Model(d, _Held(pieces), "lkc_decoder_create")
        self._model = model  # complete: another thread may take it from here on
        return model

    _MAX_SIDES = 16
    _SIDES_LOCK = threading.Lock()

    def _side_stream(self, caller):
        """The handle of the stream for the shortcuts of a call on stream `caller`: one per calling stream, so that callers on
        different streams do not wait for each other, nor one for a capture of another. Its own, as far as torch's pool of 32
        goes: none of another caller and no calling stream seen so far. The last callers' are kept; a stream that was handed out
        twice in the end costs overlap, not results (lkc_decoder_forward leaves out one that is in another capture)."""
        with self._SIDES_LOCK:
            side = self._sides.pop(caller, None)
            if side is None:
                taken = {caller, *self._sides, *(s.cuda_stream for s in self._sides.values())}
                for _ in range(64):
                    side = torch.cuda.Stream(self.bank_b.device)
                    if side.cuda_stream not in taken:
                        break
                while len(self._sides) >= self._MAX_SIDES:
                    del self._sides[next(iter(self._sides))]
            self._sides[caller] = side  # the last one used at the end
            return side.cuda_stream

    def _takes(self, asr, f0, n_curve, s):
        """Whether the whole call may have these operands, whose addresses go to the kernels unchecked."""
        dev = self.bank_b.device
        return (all(isinstance(t, torch.Tensor) and t.device == dev and t.dtype == torch.float32 for t in (asr, f0, n_curve, s))
                and asr.shape[1] >= 1 and asr.stride(1) == 1 and asr.stride(0) >= asr.shape[1]
                and all(t.is_contiguous() for t in (f0, n_curve, s)) and s.numel() == 128)

    def _forward_whole(self, model, asr, f0, n_curve, s):
        dev, frames, lib = self.bank_b.device, int(asr.shape[1]), _lib.lib()
        size = ctypes.c_int64(0)
        with torch.cuda.device(dev):
            out = ops.empty_rows(512, 2 * frames, dev)
            rc = lib.lkc_decoder_workspace(model.handle, frames, ctypes.byref(size))
            if rc == 0:
                ws = torch.empty(size.value, dtype=torch.uint8, device=dev)
                io = _lib.LkcDecoderIo()
                io.asr, io.f0, io.n, io.s = asr.data_ptr(), f0.data_ptr(), n_curve.data_ptr(), s.data_ptr()
                io.out, io.frames, io.asr_pitch, io.out_pitch = out.data_ptr(), frames, asr.stride(0), out.stride(0)
                stream = ops._stream()
                io.workspace, io.workspace_bytes, io.side = ws.data_ptr(), size.value, self._side_stream(stream)
                rc = lib.lkc_decoder_forward(model.handle, ctypes.byref(io), stream)
        if rc != 0:
            raise _lib.LkcError("decoder forward: " + _lib.last_error())
        ops.count_launches(io.launches)
        return out

    def _style(self, s):
        bank = ops.gemm_bias_f32_cuda(s.reshape(1, -1), self.bank_wt, self.bank_b).reshape(-1)

        def gb(name):
            o, n = self.bank_off[name]
            return bank[o: o + n]

        return gb

    def _conv1x1(self, x, name):
        """Pointwise conv on the tensor cores (K = 1, identity affine), 42-99 us at 61 to 1040 columns. The input is raw
        features, so the operands are tf32 halves: the f16 halves of the other convs would limit its range. Error against
        float64 0.38-0.75 of that of the CUDA cores' f32 sums over 512 to 1104 channels."""
        w = self.w
        return ops.conv1d_affine_f32_cuda(x, w[name + ".weight"], w[name + ".bias"], self._ident[int(x.shape[0])],
                                          state=self.state[name])[0]

    def _concat(self, parts, cin):
        """concat_rows of the block input, with zero rows up to the next multiple of 16 channels."""
        z = _pad16(cin) - cin
        if z:
            parts = list(parts) + [torch.zeros(z, parts[0].shape[1], device=self.device)]
        return ops.concat_rows_f32_cuda(*parts)

    def adain_resblk(self, x, gb, name, cin, cout, upsample):
        """AdainResBlk1d through the basic ops (models/kokoro/model.py:158-174). x carries the padded rows."""
        w = self.w
        r = ops.leaky_relu_f32_cuda(ops.adain1d_f32_cuda(x, gb(name + ".norm1.fc")), slope=0.2)
        if upsample:
            r = ops.conv_transpose1d_dw_f32_cuda(r, w[name + ".pool.weight"], w[name + ".pool.bias"], stride=2,
                                                 padding=1, output_padding=1)
        r = ops.conv1d_f32_cuda(r, w[name + ".conv1.weight"], w[name + ".conv1.bias"], padding=1)
        r = ops.leaky_relu_f32_cuda(ops.adain1d_f32_cuda(r, gb(name + ".norm2.fc")), slope=0.2)
        r = ops.conv1d_f32_cuda(r, w[name + ".conv2.weight"], w[name + ".conv2.bias"], padding=1)
        sc = ops.upsample_nearest1d_f32_cuda(x, scale=2) if upsample else x
        if cin != cout:
            sc = ops.conv1d_nobias_f32_cuda(sc, w[name + ".conv1x1.weight"])
        return ops.scale_f32_cuda(ops.add_f32_cuda(r, sc), scale=SQRT1_2)

    def adain_resblk_fused(self, x, gb, name, cin, cout, upsample):
        """The block through the fused conv kernels (models/kokoro/model.py:205-221)."""
        w = self.w
        gb1 = gb(name + ".norm1.fc")
        af = ops.adain_affine_f32_cuda(ops.channel_stats_f32_cuda(x), gb1, length=int(x.shape[1]))
        if upsample:
            r = ops.leaky_relu_f32_cuda(ops.adain1d_f32_cuda(x, gb1), slope=0.2)
            r = ops.conv_transpose1d_dw_f32_cuda(r, w[name + ".pool.weight"], w[name + ".pool.bias"], stride=2,
                                                 padding=1, output_padding=1)
            h, st = ops.conv1d_affine_f32_cuda(r, w[name + ".conv1.weight"], w[name + ".conv1.bias"],
                                               self._ident[int(x.shape[0])], padding=1,
                                               state=self.state[name + ".conv1"])
        else:
            h, st = ops.conv1d_leaky_f32_cuda(x, w[name + ".conv1.weight"], w[name + ".conv1.bias"], af, slope=0.2,
                                              padding=1, state=self.state[name + ".conv1"])
        af = ops.adain_affine_f32_cuda(st, gb(name + ".norm2.fc"), length=int(h.shape[1]))
        sc = self._conv1x1(x, name + ".conv1x1") if cin != cout else x
        if upsample:  # nearest neighbour: the same values on either side of a pointwise conv, at half the columns
            sc = ops.upsample_nearest1d_f32_cuda(sc, scale=2)
        out, _ = ops.conv1d_leaky_f32_cuda(h, w[name + ".conv2.weight"], w[name + ".conv2.bias"], af, slope=0.2,
                                           residual=sc, out_scale=SQRT1_2, padding=1,
                                           state=self.state[name + ".conv2"])
        return out

    def forward(self, asr, f0, n_curve, s, fused=True):
        """asr f32[512, F], f0 / n_curve f32[2F], s f32[128] (cuda tensors) -> x f32[512, 2F], the generator's input
        (models/kokoro/model.py:704-717)."""
        w = self.w
        ops.check(asr.dim() == 2 and asr.shape[0] == 512, "asr must be f32[512, F]")
        frames = int(asr.shape[1])
        ops.check(tuple(f0.shape) == (2 * frames,) and tuple(n_curve.shape) == (2 * frames,),
                  "f0 and n_curve must be f32[2F]")
        if fused and not ops.op_by_op() and self._takes(asr, f0, n_curve, s):
            model = self._whole_model()
            if model is not None:
                return self._forward_whole(model, asr, f0, n_curve, s)
        gb = self._style(s)
        f0d = ops.conv1d_f32_cuda(f0.reshape(1, -1), w["decoder.F0_conv.weight"], w["decoder.F0_conv.bias"], stride=2,
                                  padding=1)
        nd = ops.conv1d_f32_cuda(n_curve.reshape(1, -1), w["decoder.N_conv.weight"], w["decoder.N_conv.bias"],
                                 stride=2, padding=1)
        blk = self.adain_resblk_fused if fused else self.adain_resblk
        name, cin, cout, up = DECODER_BLOCKS[0]
        x = blk(self._concat([asr, f0d, nd], cin), gb, name, cin, cout, up)
        if fused:
            asr_res = self._conv1x1(asr, "decoder.asr_res.0")
        else:
            asr_res = ops.conv1d_f32_cuda(asr, w["decoder.asr_res.0.weight"], w["decoder.asr_res.0.bias"])
        for name, cin, cout, up in DECODER_BLOCKS[1:]:
            x = blk(self._concat([x, asr_res, f0d, nd], cin), gb, name, cin, cout, up)
        return x
