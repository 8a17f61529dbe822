"""The Kokoro iSTFTNet generator wired from `ops.*_cuda`: the `cuda`-device twin of the generator part of the
reference graph builder (models/kokoro/model.py:735-781) with its building blocks adain_resblock1_fused (:235-247),
adain_resblock1 (:250-260) and the style bank (:67-81, 135-144). The graph structure is the reference's; only the
kernel-name suffix differs.

Generator(sd) uploads a state dict once (weights become device constants, the ConvTranspose weights are packed once,
the AdaIN `fc` layers are concatenated into one style-bank GEMV). forward() runs one utterance on torch's current
stream. capture(t) records the fused graph for one input length into a CUDA graph with static input/output
buffers, so a replay costs one launch.
"""
from __future__ import annotations

import ctypes
import operator

import numpy as np
import torch

from . import _lib, ops
from .synth import shapes

DILATIONS = (1, 3, 5)
RES_KERNELS = (3, 7, 11)


class _NullCtx:
    def __enter__(self):
        return None

    def __exit__(self, *exc):
        return False


class StyleBank:
    """fc(style) of every AdaIN as views into one style-bank GEMV (model.py:135-144): bank(name) -> f32[2C]."""

    def __init__(self, bank, off):
        self.bank, self.off = bank, off

    def __call__(self, name):
        o, n = self.off[name]
        return self.bank[o: o + n]


class _Held:
    """The objects whose addresses a library struct holds, and where its tensors were. The references keep the memory; the
    struct is made anew when one of them was replaced in the generator or moved (`t.data = ...`)."""

    def __init__(self, objs):
        self.objs = objs
        self.tensors = [o for o in objs if isinstance(o, torch.Tensor)]
        self.ptrs = list(map(torch.Tensor.data_ptr, self.tensors))

    def current(self, objs):
        return (len(objs) == len(self.objs) and all(map(operator.is_, self.objs, objs))
                and list(map(torch.Tensor.data_ptr, self.tensors)) == self.ptrs)


class _Model:
    """Handle of lkc_generator_create (or lkc_decoder_create); a call in flight in another thread keeps the one it was given."""

    def __init__(self, struct, held, create="lkc_generator_create"):
        self.held = held
        self.handle = getattr(_lib.lib(), create)(ctypes.byref(struct))
        if not self.handle:
            raise _lib.LkcError(_lib.last_error())

    def __del__(self):
        try:
            if self.handle:
                _lib.lib().lkc_model_destroy(self.handle)
                self.handle = None
        except Exception:
            pass


class Generator:
    def __init__(self, sd: dict, device="cuda"):
        self.device = torch.device(device)
        self.w = {k: ops.to_cuda(np.ascontiguousarray(v, dtype=np.float32), self.device) for k, v in sd.items()}
        for k in list(self.w):
            if ".alpha" in k:  # Snake alpha (1, C, 1) -> (C,)   (model.py:_flat_alpha)
                self.w[k] = self.w[k].reshape(-1).contiguous()
        # Style bank: every `<name>.fc` as one [128, total] weight + bias, names sorted (model.py:67-81).
        names = sorted(k[: -len(".weight")] for k in self.w if k.endswith(".fc.weight"))
        self.bank_wt = torch.cat([self.w[n + ".weight"].t() for n in names], dim=1).contiguous()
        self.bank_b = torch.cat([self.w[n + ".bias"] for n in names]).contiguous()
        self.bank_off, o = {}, 0
        for n in names:
            self.bank_off[n] = (o, self.w[n + ".bias"].shape[0])
            o += self.bank_off[n][1]
        # Polyphase packs of the two upsamplers (model.py:788-793), run once on constants.
        self.ups_wp = None
        if "ups.0.weight" in self.w:  # a state dict of resblocks only is enough for adain_resblock1*
            self.ups_wp = [ops.convt_poly_weights_cuda(self.w["ups.0.weight"], 10, 5),
                           ops.convt_poly_weights_cuda(self.w["ups.1.weight"], 6, 3)]
            self.ups_state = [ops.conv_transpose1d_prepare_f32_cuda(self.w["ups.0.weight"], 10, 5),
                              ops.conv_transpose1d_prepare_f32_cuda(self.w["ups.1.weight"], 6, 3)]
        self.ident128 = torch.stack([torch.zeros(128), torch.ones(128), torch.zeros(128)]).to(self.device).contiguous()
        # Prepared state of every fused-conv weight the tensor-core kernel accepts (packed once, at init).
        self.conv_state = {}
        for k in self.w:
            if k.endswith(".weight") and (".convs1." in k or ".convs2." in k or k == "conv_post.weight"):
                st = ops.conv1d_prepare_f32_cuda(self.w[k])
                if st is not None:
                    self.conv_state[k[: -len(".weight")]] = st
        # The two noise convs (22 -> 256, k 12, stride 6, padding 3; 22 -> 128, k 1) as stride-1 convs over the
        # polyphase view of `har` (ops.space_to_depth_f32_cuda), channels padded to a multiple of 16: the shape the
        # tensor-core conv takes. Packed once, like every other weight.
        self.noise_tc = {}
        for i, (stride, pad) in enumerate(((6, 3), (1, 0))):
            key = f"noise_convs.{i}"
            if key + ".weight" not in sd:
                continue
            wn = np.ascontiguousarray(sd[key + ".weight"], dtype=np.float32)
            rows = -(-wn.shape[1] * stride // 16) * 16
            wp = ops.to_cuda(ops.polyphase_conv_weights(wn, stride, rows), self.device)
            state = ops.conv1d_prepare_f32_cuda(wp)
            if state is not None:
                ident = torch.stack([torch.zeros(rows), torch.ones(rows), torch.zeros(rows)]).to(self.device).contiguous()
                self.noise_tc[i] = (wp, state, ident, stride, pad, wn.shape[2] // stride, rows)
        self._graphs = {}
        self._streams = None
        self._blocks = {}  # prefix -> (LkcResblock, the getters of its weights and states, _Held)
        self._model = None  # (getters of its weights and states, _Model) of the whole-forward call

    # ------------------------------------------------------------------ building blocks

    def _noise_conv(self, har, i, keep):
        """noise_convs[i](har) -> (xs, chunk statistics of xs or None); temporaries go to `keep`. On the tensor cores when the polyphase pack
        exists (and the conv path is not "simt"): space-to-depth of har, then a stride-1 conv with an identity
        affine, whose epilogue also gives the statistics the following resblock needs."""
        w = self.w
        if i in self.noise_tc and ops._conv_path != "simt":
            wp, state, ident, stride, pad, taps, rows = self.noise_tc[i]
            y = ops.space_to_depth_f32_cuda(har, stride, pad, taps, rows)
            keep.append(y)
            return ops.conv1d_affine_f32_cuda(y, wp, w[f"noise_convs.{i}.bias"], ident, state=state)
        if i == 0:
            return ops.conv1d_f32_cuda(har, w["noise_convs.0.weight"], w["noise_convs.0.bias"], stride=6, padding=3), None
        return ops.conv1d_f32_cuda(har, w["noise_convs.1.weight"], w["noise_convs.1.bias"]), None

    def style(self, s):
        """fc(style) of every AdaIN as views into one style-bank GEMV (model.py:135-144): name -> f32[2C]."""
        return StyleBank(ops.gemm_bias_f32_cuda(s.reshape(1, -1), self.bank_wt, self.bank_b).reshape(-1), self.bank_off)

    # One resblock and one forward as single library calls (lkc_resblock, lkc_generator_forward), queued without a trip
    # through Python per kernel. The compositions below compute the same in single ops, not launch for launch: the whole
    # forward adds the first upsampled input in the noise block's last conv, takes stage 0's statistics from that conv's
    # epilogue and gives each branch a share of the SMs, and in both calls split convs fold the statistics themselves. So the
    # last bits differ, and timings of single kernels (ops.Profile) are those of the composition. It remains for what
    # looks at single kernels (ops.Profile with timing, ops.tracing, the stage outputs), for the CUDA-core path, for shapes
    # that have no tensor-core state and for operands that a whole call would not check.

    def _is(self, t, *shape):
        """A tensor the kernels can take by its address alone."""
        return tuple(t.shape) == shape and t.dtype == torch.float32 and t.is_contiguous() and t.device == self.bank_b.device

    def _block(self, prefix, k):
        """LkcResblock of the weights under `prefix`, or None when a conv of it has no prepared state."""
        entry = self._blocks.get(prefix)
        try:
            if entry is not None:
                blk, get_w, get_s, held = entry
                if held.current(get_w(self.w) + get_s(self.conv_state) + (self.bank_off,)):
                    return blk if blk.k == k else None
            convs = [f"{prefix}.convs{n}.{j}" for j in range(3) for n in (1, 2)]
            get_w = operator.itemgetter(*[c + ".weight" for c in convs], *[c + ".bias" for c in convs],
                                        *[f"{prefix}.alpha{n}.{j}" for j in range(3) for n in (1, 2)])
            get_s = operator.itemgetter(*convs)
            ws, states = get_w(self.w), get_s(self.conv_state)
            gb = [self.bank_off[f"{prefix}.adain{n}.{j}.fc"] for j in range(3) for n in (1, 2)]
        except KeyError:
            return None
        c = int(ws[0].shape[0])
        if not (all(st is not None and st.shape == (c, c, k) for st in states) and all(n == 2 * c for _, n in gb)
                and all(self._is(t, c, c, k) for t in ws[:6]) and all(self._is(t, c) for t in ws[6:])):
            return None
        blk, ptrs = _lib.LkcResblock(), [t.data_ptr() for t in ws]
        blk.c, blk.k = c, k
        blk.w[:], blk.b[:], blk.alpha[:] = ptrs[:6], ptrs[6:12], ptrs[12:]
        blk.state[:], blk.gb[:] = [st.handle for st in states], [o for o, _ in gb]
        self._blocks[prefix] = (blk, get_w, get_s, _Held(ws + states + (self.bank_off,)))
        return blk

    _BLOCKS = [(f"noise_res.{i}", k) for i, k in enumerate((7, 11))] + [
        (f"resblocks.{3 * i + j}", k) for i in (0, 1) for j, k in enumerate(RES_KERNELS)]
    _OTHER_NAMES = ("noise_convs.0.bias", "noise_convs.1.bias", "ups.0.bias", "ups.1.bias", "conv_post.weight",
                    "conv_post.bias")
    _OTHERS = operator.itemgetter(*_OTHER_NAMES)

    def _pieces(self, get_w, get_s):
        """Everything that the whole-forward struct points to."""
        return (*get_w(self.w), *get_s(self.conv_state), *self.noise_tc.values(), *(n[0] for n in self.noise_tc.values()),
                *self.ups_state, self.bank_wt, self.bank_b, self.ident128, self.bank_off)

    def _whole_model(self):
        """_Model of lkc_generator_forward, or None when some conv has no tensor-core state."""
        if self.ups_wp is None:
            return None
        try:
            if self._model is not None:
                get_w, get_s, model = self._model
                if model.held.current(self._pieces(get_w, get_s)):
                    return model
            blocks = [self._block(prefix, k) for prefix, k in self._BLOCKS]
            if None in blocks:
                return None
            others = self._OTHERS(self.w)
            noise, ups, post = (self.noise_tc[0], self.noise_tc[1]), tuple(self.ups_state), self.conv_state["conv_post"]
        except KeyError:
            return None
        n = int(self.bank_b.shape[0])
        tensors = zip((*others, self.bank_wt, self.bank_b, self.ident128),
                      ((256,), (128,), (256,), (128,), (22, 128, 7), (22,), (128, n), (n,), (3, 128)))
        states = zip((noise[0][1], noise[1][1], *ups, post),
                     ((256, noise[0][6], noise[0][5]), (128, noise[1][6], noise[1][5]), (512, 256, 20, 10),
                      (256, 128, 12, 6), (22, 128, 7)))
        if not (all(self._is(t, *sh) for t, sh in tensors) and all(st is not None and st.shape == sh for st, sh in states)):
            return None
        m = _lib.LkcGenerator()
        m.noise_res[:], m.res[:] = blocks[:2], blocks[2:]
        m.bank_wt, m.bank_b, m.bank_n = self.bank_wt.data_ptr(), self.bank_b.data_ptr(), n
        for i, (wp, state, _, stride, pad, taps, rows) in enumerate(noise):
            nc = m.noise_conv[i]
            nc.w, nc.b, nc.state = wp.data_ptr(), others[i].data_ptr(), state.handle
            nc.stride, nc.padding, nc.taps, nc.rows = stride, pad, taps, rows
            m.ups_b[i], m.ups_state[i] = others[2 + i].data_ptr(), ups[i].handle
        m.post_w, m.post_b = others[4].data_ptr(), others[5].data_ptr()
        m.ident128, m.post_state = self.ident128.data_ptr(), post.handle
        with torch.cuda.device(self.bank_b.device):
            names = [n for prefix, _ in self._BLOCKS for n in self.w if n.startswith(prefix + ".") and ".adain" not in n]
            get_w = operator.itemgetter(*names, *self._OTHER_NAMES)
            get_s = operator.itemgetter(*(n for n in self.conv_state))
            model = _Model(m, _Held(self._pieces(get_w, get_s)))
        self._model = (get_w, get_s, model)
        return model

    @staticmethod
    def _workspace_bytes(model, t, concurrent, planned=True):
        """(bytes of the workspace, bytes without a plan) of the intermediates of one forward of length t."""
        b, u = ctypes.c_int64(0), ctypes.c_int64(0)
        mode = int(concurrent) if planned else int(concurrent) | _lib.LKC_UNPLANNED
        if _lib.lib().lkc_generator_workspace(model.handle, t, mode, ctypes.byref(b), ctypes.byref(u)) != 0:
            raise _lib.LkcError(_lib.last_error())
        return b.value, u.value

    def _forward_whole(self, model, x, har, s, outputs, concurrent, workspace=None, planned=True):
        """planned=False: every intermediate has bytes of its own in the workspace."""
        t, dev = int(x.shape[1]), self.device
        sh = shapes(t)
        if workspace is None:
            workspace = torch.empty(self._workspace_bytes(model, t, concurrent, planned)[0], dtype=torch.uint8, device=dev)
        io = _lib.LkcGeneratorIo()
        res = {"audio": torch.empty(sh["S"], dtype=torch.float32, device=dev)}
        if "post" in outputs:
            with ops.padded_rows():
                res["post"] = ops.empty_rows(22, sh["L1"], dev)
            io.post, io.post_pitch = res["post"].data_ptr(), res["post"].stride(0)
        io.x, io.har, io.s, io.audio = x.data_ptr(), har.data_ptr(), s.data_ptr(), res["audio"].data_ptr()
        io.t, io.x_pitch, io.har_pitch = t, x.stride(0), har.stride(0)
        io.workspace, io.workspace_bytes = workspace.data_ptr(), workspace.numel()
        io.concurrent = int(concurrent) if planned else int(concurrent) | _lib.LKC_UNPLANNED
        if concurrent:
            io.side[:] = [st.cuda_stream for st in self._side_streams()]
        if _lib.lib().lkc_generator_forward(model.handle, ctypes.byref(io), ops._stream()) != 0:
            raise _lib.LkcError("generator forward: " + _lib.last_error())
        ops.count_launches(io.launches)
        out = tuple(res[o] for o in outputs)
        return out[0] if len(out) == 1 else out

    def _resblock_whole(self, blk, x, gb, x_stats):
        c, n = int(x.shape[0]), int(x.shape[1])
        out = ops.empty_rows(c, n, x.device)
        stats = ops._alloc((c, ops.ceildiv(n, ops.STAT_CHUNK), 2), x.device)
        io, fn = _lib.LkcResblockIo(), _lib.lib().lkc_resblock
        io.x, io.bank, io.out, io.out_stats = x.data_ptr(), gb.bank.data_ptr(), out.data_ptr(), stats.data_ptr()
        io.stats = None if x_stats is None else x_stats.data_ptr()
        io.l, io.x_pitch, io.out_pitch = n, x.stride(0), out.stride(0)
        rc = fn(ctypes.byref(blk), ctypes.byref(io), None)  # sizes the workspace
        if rc == 0:
            ws = torch.empty(io.workspace_bytes, dtype=torch.uint8, device=x.device)
            io.workspace = ws.data_ptr()
            with torch.cuda.device(x.device):
                rc = fn(ctypes.byref(blk), ctypes.byref(io), ops._stream())
        if rc != 0:
            raise _lib.LkcError("resblock: " + _lib.last_error())
        ops.count_launches(io.launches)
        return out, stats

    def _takes_block(self, x, gb, x_stats):
        """Whether the whole-block call may have these operands, whose addresses go to the kernels unchecked. Everything
        else is left to the composition, op by op with its checks: a style bank of another generator (the block's offsets
        are this one's), one that is too short, operands on another device than the weights, an empty x, statistics that
        are not 8-byte aligned (the kernels read them in pairs)."""
        if not (isinstance(gb, StyleBank) and gb.off is self.bank_off):
            return False
        bank, dev = gb.bank, self.bank_b.device
        return (x.is_cuda and x.device == dev and x.dim() == 2 and x.shape[1] >= 1
                and bank.device == dev and bank.dtype == torch.float32 and bank.shape == self.bank_b.shape
                and bank.is_contiguous()
                and (x_stats is None or (x_stats.device == dev and x_stats.data_ptr() % 8 == 0)))

    def _snake_conv(self, x, af, alpha_key, conv, k, d, residual=None):
        w = self.w
        return ops.conv1d_snake_f32_cuda(x, w[conv + ".weight"], w[conv + ".bias"], af, w[alpha_key],
                                         residual=residual, padding=d * (k - 1) // 2, dilation=d,
                                         state=self.conv_state.get(conv))

    def adain_resblock1_fused(self, x, gb, prefix, k, x_stats=None):
        n = x.shape[1]
        if not ops.op_by_op() and self._takes_block(x, gb, x_stats):
            blk = self._block(prefix, k)
            ops._f32(x, *([] if x_stats is None else [x_stats]))
            if blk is not None and tuple(x.shape) == (blk.c, n) and (
                    x_stats is None or tuple(x_stats.shape) == (blk.c, ops.ceildiv(n, ops.STAT_CHUNK), 2)):
                return self._resblock_whole(blk, x, gb, x_stats)
        st = ops.channel_stats_f32_cuda(x) if x_stats is None else x_stats
        for j, d in enumerate(DILATIONS):
            af = ops.adain_affine_f32_cuda(st, gb(f"{prefix}.adain1.{j}.fc"), length=n)
            xt, st1 = self._snake_conv(x, af, f"{prefix}.alpha1.{j}", f"{prefix}.convs1.{j}", k, d)
            af = ops.adain_affine_f32_cuda(st1, gb(f"{prefix}.adain2.{j}.fc"), length=n)
            x, st = self._snake_conv(xt, af, f"{prefix}.alpha2.{j}", f"{prefix}.convs2.{j}", k, 1, residual=x)
        return x, st

    def adain_resblock1(self, x, gb, prefix, k):
        w = self.w
        for j, d in enumerate(DILATIONS):
            xt = ops.adain1d_f32_cuda(x, gb(f"{prefix}.adain1.{j}.fc"))
            xt = ops.snake_f32_cuda(xt, w[f"{prefix}.alpha1.{j}"])
            xt = ops.conv1d_f32_cuda(xt, w[f"{prefix}.convs1.{j}.weight"], w[f"{prefix}.convs1.{j}.bias"],
                                     padding=d * (k - 1) // 2, dilation=d)
            xt = ops.adain1d_f32_cuda(xt, gb(f"{prefix}.adain2.{j}.fc"))
            xt = ops.snake_f32_cuda(xt, w[f"{prefix}.alpha2.{j}"])
            xt = ops.conv1d_f32_cuda(xt, w[f"{prefix}.convs2.{j}.weight"], w[f"{prefix}.convs2.{j}.bias"],
                                     padding=(k - 1) // 2)
            x = ops.add_f32_cuda(xt, x)
        return x

    # ------------------------------------------------------------------ the graph

    def har_from_f0(self, f0, noise):
        """The generator's `har` input from the F0 curve, as the reference graph computes it before the generator
        (models/kokoro/model.py:720-726): harmonic source (9 harmonics, x300, Linear 9 -> 1, tanh) then STFT(n_fft 20,
        hop 5) -> cat(magnitude, phase). f0 f32[T] (one value per frame of x); noise = f32[300 T, 9] (the normal draw
        as an operand) or an int seed (drawn in the kernel, models/kokoro/model.py:721-722) -> f32[22, 60 T + 1]."""
        ops.check("m_source.l_linear.weight" in self.w, "the state dict has no m_source.l_linear weights")
        w9 = self.w["m_source.l_linear.weight"].reshape(9)
        bias = self.w["m_source.l_linear.bias"].reshape(1)
        if isinstance(noise, int):  # a seed: the noise is drawn in the kernel (the variant the reference graph ships)
            src = ops.harmonic_source_rng_f32_cuda(f0, w9, bias, noise)
        else:
            src = ops.harmonic_source_f32_cuda(f0, noise, w9, bias)
        return ops.stft_magphase_f32_cuda(src, n_fft=20, hop=5)

    def forward(self, x, har, s, fused=True, outputs=("audio",), concurrent=True, pad_rows=True):
        """x f32[512, T], har f32[22, 60 T + 1], s f32[128] (cuda tensors) -> the named outputs
        ("audio" f32[300 T], "post" f32[22, 60 T + 1]; with pad_rows the 2-D outputs are [:, :L] views of buffers
        whose rows are padded to a multiple of 4 floats).

        The op sequence is the reference's (model.py:735-781). With concurrent=True (fused graph only) the branches
        that do not depend on each other are queued on side streams, forked from and joined back to torch's current
        stream: the two noise branches (they only need `har`) and, per stage, the three resblocks (they share their
        input). The results are the same; independent persistent conv kernels then fill the SMs that the tail of
        another one leaves idle (a stage-0 conv of the 26 s case has 164 tiles for 148 SMs)."""
        w = self.w
        ops.check(x.dim() == 2 and x.shape[0] == 512, "x must be f32[512, T]")
        sh = shapes(int(x.shape[1]))
        ops.check(tuple(har.shape) == (22, sh["L1"]), f"har must be f32[22, {sh['L1']}]")
        if fused and pad_rows and not ops._pad_rows and ops._conv_path != "simt":
            # the generator owns every intermediate: rows padded to 16 bytes, so that the tensor-core kernels move
            # them with the TMA unit (values do not depend on the pitch)
            with ops.padded_rows():
                return self.forward(x, har, s, fused, outputs, concurrent, pad_rows)
        whole = fused and set(outputs) <= {"audio", "post"} and not ops.op_by_op() and ops._pad_rows
        model = self._whole_model() if whole else None
        if model is not None:
            ops._f32(x, har, s)
            dev = self.bank_b.device
            ops.check(all(v.is_cuda and v.device == dev for v in (x, har, s)) and s.numel() == 128,
                      f"x, har and s must live on the generator's device ({dev}), s must be f32[128]")
            with torch.cuda.device(dev):
                return self._forward_whole(model, x, har, s.contiguous(), outputs, concurrent)
        gb = self.style(s)
        cur = torch.cuda.current_stream(self.device)
        par = fused and concurrent
        side = self._side_streams() if par else None

        def on(stream):
            return torch.cuda.stream(stream) if par else _NullCtx()

        keep = []  # every intermediate stays referenced until all streams are joined
        st = {}
        rb = None
        noise = [None, None]
        if par:
            for i in (0, 1):
                ops.join(side[i], cur)
        for i, (_, _, k_noise) in enumerate(((20, 10, 7), (12, 6, 11))):
            if not fused:
                break
            with on(side[i] if par else None):
                xs, xs_stats = self._noise_conv(har, i, keep)
                noise[i], _ = self.adain_resblock1_fused(xs, gb, f"noise_res.{i}", k_noise, x_stats=xs_stats)
                keep += [xs, xs_stats] if xs_stats is not None else [xs]
        for i, (k_up, u, k_noise) in enumerate(((20, 10, 7), (12, 6, 11))):
            if fused:
                if par:
                    ops.join(cur, side[i])
                if i == 0:
                    xin = x
                else:
                    # resblock mean as its own pass (13 us of HBM time at T = 2080), so that the upsampler takes the
                    # tensor-core path; conv_transpose1d_poly(..., mean3=...) is the fused CUDA-core alternative
                    xin = ops.add3_scale_f32_cuda(rb[0], rb[1], rb[2], scale=1.0 / 3.0)
                    keep.append(xin)
                x = ops.conv_transpose1d_poly_f32_cuda(
                    xin, self.ups_wp[i], w[f"ups.{i}.bias"], noise[i], stride=u, padding=(k_up - u) // 2,
                    taps=k_up // u, slope=0.1, pad_left=1 if i == 1 else 0, state=self.ups_state[i])
                xst = ops.channel_stats_f32_cuda(x)
                keep += [x, xst, *(rb or [])]
                new_rb = [None, None, None]
                if par:
                    ops.join(side[2], cur)
                    ops.join(side[3], cur)
                # the k = 11 block is the longest: it stays on the current stream
                for j, stream in ((2, None), (1, side[2] if par else None), (0, side[3] if par else None)):
                    with on(stream):
                        new_rb[j] = self.adain_resblock1_fused(x, gb, f"resblocks.{3 * i + j}", RES_KERNELS[j], xst)[0]
                if par:
                    ops.join(cur, side[2])
                    ops.join(cur, side[3])
                rb = new_rb
            else:
                if i == 0:
                    xs = ops.conv1d_f32_cuda(har, w["noise_convs.0.weight"], w["noise_convs.0.bias"], stride=6, padding=3)
                else:
                    xs = ops.conv1d_f32_cuda(har, w["noise_convs.1.weight"], w["noise_convs.1.bias"])
                xs = self.adain_resblock1(xs, gb, f"noise_res.{i}", k_noise)
                x = ops.leaky_relu_f32_cuda(x, slope=0.1)
                x = ops.conv_transpose1d_f32_cuda(x, w[f"ups.{i}.weight"], w[f"ups.{i}.bias"], stride=u,
                                                  padding=(k_up - u) // 2, output_padding=0)
                if i == 1:
                    x = ops.pad_reflect1d_f32_cuda(x, left=1, right=0)
                x = ops.add_f32_cuda(x, xs)
                rb = [self.adain_resblock1(x, gb, f"resblocks.{3 * i + j}", kk) for j, kk in enumerate(RES_KERNELS)]
                x = ops.add3_scale_f32_cuda(rb[0], rb[1], rb[2], scale=1.0 / 3.0)
            st[f"stage{i}"] = rb if fused else x
        if fused:
            # resblock mean, then the direct fused conv (model.py:774-776): on this device the extra pass over the
            # mean costs ~40 us of HBM time, and the conv then runs on the tensor cores (Co = 22 padded to 128 rows)
            xm = ops.add3_scale_f32_cuda(rb[0], rb[1], rb[2], scale=1.0 / 3.0)
            post, _ = ops.conv1d_leaky_f32_cuda(xm, w["conv_post.weight"], w["conv_post.bias"], self.ident128,
                                                slope=0.01, padding=3, state=self.conv_state.get("conv_post"))
        else:
            x = ops.leaky_relu_f32_cuda(x, slope=0.01)
            post = ops.conv1d_f32_cuda(x, w["conv_post.weight"], w["conv_post.bias"], padding=3)
        st["post"] = post
        st["audio"] = ops.istft_logits_f32_cuda(post, n_fft=20, hop=5)
        if par:
            # tensors made on a side stream are consumed on the current one: tell the allocator
            for t in keep + noise + list(rb):
                if isinstance(t, torch.Tensor):
                    t.record_stream(cur)
        res = tuple(st[o] for o in outputs)
        return res[0] if len(res) == 1 else res

    def _side_streams(self):
        if self._streams is None:
            self._streams = [torch.cuda.Stream(device=self.device) for _ in range(4)]
        return self._streams

    def _warm_stream(self):
        """The stream capture() runs its warm-up and traced forwards on: one per generator, and never the same CUDA
        stream as a side stream. torch hands streams out of a pool of 32 round-robin, so a stream made later can BE an
        earlier one; a traced forward whose main stream coincided with a side stream would look more serial than the
        captured one is, and the memory plan made from it would overlay tensors of branches that run concurrently."""
        if getattr(self, "_warm", None) is None:
            taken = {s.cuda_stream for s in self._side_streams()}
            for _ in range(64):
                s = torch.cuda.Stream(device=self.device)
                if s.cuda_stream not in taken:
                    self._warm = s
                    break
            else:
                raise RuntimeError("no CUDA stream distinct from the side streams")
        return self._warm

    # ------------------------------------------------------------------ CUDA graph replay

    def capture(self, t: int, planned: bool = True):
        """Records forward(fused=True) for input length t into a CUDA graph (once per t). Returns a dict with the
        static buffers `x`, `har`, `s`, `audio` and the `graph`; fill the inputs, then graph.replay().

        planned=True (default): the forward's intermediates live in a planned arena, ONE device buffer in which tensors
        that are never alive together (judged by the fork / join structure of the streams, not by program order) overlay
        each other (`arena_bytes`; `unplanned_bytes` is what keeping every intermediate would take). The plan is the
        whole-forward call's own; the op-by-op forward of the CUDA-core path is traced and planned by arena.py.
        planned=False: every intermediate has memory of its own, in the graph's pool."""
        if t in self._graphs:
            return self._graphs[t]
        from .arena import PlannedArena, Tracer
        sh = shapes(t)
        dev = self.device
        pitch = -(-t // ops.ROW_ALIGN) * ops.ROW_ALIGN  # rows of x start on 16-byte boundaries for any t
        bufs = {"x": torch.zeros(512, pitch, device=dev)[:, :t], "har": torch.zeros(22, sh["L1"], device=dev),
                "s": torch.zeros(128, device=dev)}
        model = None if ops.op_by_op() else self._whole_model()
        whole = model is not None
        if whole and planned:
            bufs["arena_bytes"], bufs["unplanned_bytes"] = self._workspace_bytes(model, t, True)
            bufs["arena"] = torch.empty(bufs["arena_bytes"], dtype=torch.uint8, device=dev)
        side = self._warm_stream()
        side.wait_stream(torch.cuda.current_stream(dev))
        arena = None
        with torch.cuda.stream(side):
            for _ in range(1 if whole else 2):  # warm-up outside capture: lazy module loading, function attributes
                ref = self.forward(bufs["x"], bufs["har"], bufs["s"])
            if planned and not whole:
                with ops.tracing(Tracer()) as tr:
                    tr.pin(self.forward(bufs["x"], bufs["har"], bufs["s"]))
                arena = PlannedArena(tr, dev)
                del tr
                arena.begin()
                with ops.use_allocator(arena.allocator):
                    again = self.forward(bufs["x"], bufs["har"], bufs["s"])
                torch.cuda.synchronize(dev)
                ops.check(torch.equal(again, ref), "the planned arena changed the result of the forward")
        torch.cuda.current_stream(dev).wait_stream(side)
        torch.cuda.synchronize(dev)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            if whole:
                bufs["audio"] = self._forward_whole(model, bufs["x"], bufs["har"], bufs["s"], ("audio",), True,
                                                    bufs.get("arena"), planned)
            elif arena is not None:
                arena.begin()
                with ops.use_allocator(arena.allocator):
                    bufs["audio"] = self.forward(bufs["x"], bufs["har"], bufs["s"])
            else:
                bufs["audio"] = self.forward(bufs["x"], bufs["har"], bufs["s"])
        bufs["graph"], bufs["model"] = g, model  # the model keeps the weights that the graph reads, whatever replaces them
        if arena is not None:
            bufs["arena"], bufs["arena_bytes"], bufs["unplanned_bytes"] = arena, arena.nbytes, arena.unplanned_bytes
        self._graphs[t] = bufs
        return bufs

    def synthesize_f0(self, x_host, f0_host, seed, s_host, audio_host=None):
        """End-to-end call with HOST buffers that starts one step earlier than synthesize(): the `har` input is
        computed on the device from the F0 curve f32[T] (harmonic source with in-kernel noise from `seed`, then the
        STFT), as the reference graph does before its generator (models/kokoro/model.py:720-726)."""
        t = int(x_host.shape[1])
        b = self.capture(t)
        f0 = torch.empty(t, dtype=torch.float32, device=self.device)
        f0.copy_(f0_host, non_blocking=True)
        b["x"].copy_(x_host, non_blocking=True)
        b["s"].copy_(s_host, non_blocking=True)
        b["har"].copy_(self.har_from_f0(f0, int(seed)))
        b["graph"].replay()
        return self._collect(b, audio_host)

    def _collect(self, b, audio_host):
        """Waveform and status word to the host in stream order, one synchronisation. (The status as a call of its own behind
        the synchronisation cost 5 to 10 us: T = 24 373 -> 364, T = 320 964 -> 957.)"""
        if audio_host is None:
            audio_host = torch.empty(b["audio"].shape, dtype=torch.float32, pin_memory=True)
        audio_host.copy_(b["audio"], non_blocking=True)
        word = torch.empty(1, dtype=torch.int32, pin_memory=True)
        with torch.cuda.device(self.device):
            ops.conv_tc_status_async(word)
            torch.cuda.current_stream().synchronize()
            if int(word[0]) == 0:
                return audio_host
            ops.conv_tc_status()  # clears it
        raise RuntimeError(f"tensor-core conv kernels reported status {int(word[0]):#x} "
                           "(0x10000 = activation beyond the f16 range; else role << 8 | wait that gave up)")

    def pipeline(self, t: int, depth: int = 2):
        """Host-buffer synthesis with `depth` utterances of `t` frames in flight (see SynthesisPipeline)."""
        return SynthesisPipeline(self, t, depth)

    def synthesize(self, x_host, har_host, s_host, audio_host=None):
        """End-to-end call with HOST buffers (pinned torch tensors for async copies): host -> device copies, one
        graph replay, device -> host copy of the waveform. Returns the host waveform tensor. Raises if the tensor-core
        kernels reported a problem during the call (a bounded wait that gave up, or an activation beyond the f16
        range of the split operands, which overflows there and makes the waveform wrong)."""
        b = self.capture(int(x_host.shape[1]))
        b["x"].copy_(x_host, non_blocking=True)
        b["har"].copy_(har_host, non_blocking=True)
        b["s"].copy_(s_host, non_blocking=True)
        b["graph"].replay()
        return self._collect(b, audio_host)


class SynthesisPipeline:
    """Throughput form of Generator.synthesize for a stream of utterances of one length: the host -> device copies of
    utterance i + 1 and the device -> host copy of utterance i - 1 run on the two copy engines while the captured graph
    computes utterance i. One graph and one arena; per slot a set of staging tensors (inputs and waveform), so the
    graph's static buffers are only touched by device-side copies on the compute stream.

        pipe = gen.pipeline(t)
        tickets = [pipe.submit(x, har, s, out) for (x, har, s, out) in batch]   # pinned host tensors
        for k in tickets: pipe.wait(k)                                          # out is complete after wait

    submit() blocks only when all `depth` slots are in flight (it then waits for the oldest). wait() raises if the
    tensor-core kernels reported a problem up to and including that utterance (the status word is read stream-ordered
    after each utterance, not cleared)."""

    def __init__(self, gen, t: int, depth: int = 2):
        ops.check(depth >= 1, "depth must be >= 1")
        self.gen, self.t, self.depth = gen, int(t), int(depth)
        dev = gen.device
        self.b = gen.capture(self.t)
        self.h2d, self.d2h = torch.cuda.Stream(device=dev), torch.cuda.Stream(device=dev)
        self.compute = torch.cuda.current_stream(dev)  # the graph replays on the stream current at construction
        self.slots = []
        for _ in range(self.depth):
            self.slots.append({
                "x": torch.empty_like(self.b["x"]), "har": torch.empty_like(self.b["har"]),
                "s": torch.empty_like(self.b["s"]), "audio": torch.empty_like(self.b["audio"]),
                "status": torch.zeros(1, dtype=torch.int32).pin_memory(),
                "in_ready": torch.cuda.Event(), "in_free": None, "computed": torch.cuda.Event(),
                "out_done": None, "ticket": -1})
        self.n = 0

    def submit(self, x_host, har_host, s_host, audio_host):
        slot = self.slots[self.n % self.depth]
        if slot["ticket"] >= 0:
            self.wait(slot["ticket"])  # the slot's previous utterance has left the device
        b = self.b
        with torch.cuda.stream(self.h2d):
            if slot["in_free"] is not None:
                self.h2d.wait_event(slot["in_free"])
            slot["x"].copy_(x_host, non_blocking=True)
            slot["har"].copy_(har_host, non_blocking=True)
            slot["s"].copy_(s_host, non_blocking=True)
            slot["in_ready"].record(self.h2d)
        with torch.cuda.stream(self.compute):
            self.compute.wait_event(slot["in_ready"])
            b["x"].copy_(slot["x"]), b["har"].copy_(slot["har"]), b["s"].copy_(slot["s"])
            slot["in_free"] = torch.cuda.Event()
            slot["in_free"].record(self.compute)
            b["graph"].replay()
            slot["audio"].copy_(b["audio"])
            ops.conv_tc_status_async(slot["status"])
            slot["computed"].record(self.compute)
        with torch.cuda.stream(self.d2h):
            self.d2h.wait_event(slot["computed"])
            audio_host.copy_(slot["audio"], non_blocking=True)
            slot["out_done"] = torch.cuda.Event()
            slot["out_done"].record(self.d2h)
        slot["ticket"] = self.n
        self.n += 1
        return slot["ticket"]

    def wait(self, ticket: int) -> None:
        slot = self.slots[ticket % self.depth]
        if slot["ticket"] != ticket:
            return  # already waited for (its slot has been reused or released)
        slot["out_done"].synchronize()
        slot["ticket"] = -1
        status = int(slot["status"].item())
        if status != 0:
            raise RuntimeError(f"tensor-core conv kernels reported status {status:#x} "
                               "(0x10000 = activation beyond the f16 range; else role << 8 | wait that gave up)")
