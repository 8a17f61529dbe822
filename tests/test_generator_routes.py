"""Which calls take the whole-resblock / whole-forward library calls and which go through the op-by-op composition, with
its checks: the host logic in front of the launches, on CPU tensors that claim to live on a GPU."""
import contextlib
import ctypes
import types

import pytest
import torch

from lokinfer_b200 import _lib, ops
from lokinfer_b200 import generator as G

C, N, K = 16, 300, 3


class OnGpu(torch.Tensor):
    """A CPU tensor whose device reads cuda:`index`."""

    index = 0
    is_cuda = property(lambda self: True)
    device = property(lambda self: torch.device("cuda", self.index))


def on_gpu(t, index=0):
    t = t.as_subclass(OnGpu)
    t.index = index
    return t


class Composition(Exception):
    pass


@pytest.fixture
def gen(monkeypatch):
    """A generator of one resblock whose whole call answers "whole" and whose composition raises."""
    g = G.Generator.__new__(G.Generator)
    g.device, g.w, g._blocks, g._model = torch.device("cuda:0"), {}, {}, None
    g.bank_off = {"rb.adain1.0.fc": (0, 2 * C)}
    g.bank_b = on_gpu(torch.zeros(12 * C))
    blk = type("Blk", (), {"c": C, "k": K})()
    monkeypatch.setattr(g, "_block", lambda prefix, k: blk)
    monkeypatch.setattr(g, "_resblock_whole", lambda *a: "whole")

    def composed(*a, **k):
        raise Composition

    monkeypatch.setattr(ops, "channel_stats_f32_cuda", composed)
    monkeypatch.setattr(ops, "adain_affine_f32_cuda", composed)
    return g


def bank(g, n=12 * C, index=0, off=None):
    return G.StyleBank(on_gpu(torch.zeros(n), index), g.bank_off if off is None else off)


def stats():
    return on_gpu(torch.zeros(C, 3, 2))


def test_own_operands_take_the_whole_call(gen):
    x = on_gpu(torch.zeros(C, N))
    assert gen.adain_resblock1_fused(x, bank(gen), "rb", K) == "whole"
    assert gen.adain_resblock1_fused(x, bank(gen), "rb", K, x_stats=stats()) == "whole"


def test_a_bank_of_another_generator_goes_by_its_own_offsets(gen):
    x = on_gpu(torch.zeros(C, N))
    foreign = bank(gen, 24 * C, off={"rb.adain1.0.fc": (5, 2 * C)})
    with pytest.raises(Composition):
        gen.adain_resblock1_fused(x, foreign, "rb", K)


@pytest.mark.parametrize("what", ["x on another GPU", "stats on the CPU", "stats on another GPU", "stats not 8-byte aligned",
                                  "bank on the CPU", "bank on another GPU", "short bank", "strided bank", "f64 bank",
                                  "empty x"])
def test_operands_the_whole_call_would_not_check(gen, what):
    x, b, st = on_gpu(torch.zeros(C, N)), bank(gen), None
    if what == "x on another GPU":
        x = on_gpu(torch.zeros(C, N), 1)
    elif what == "stats on the CPU":
        st = torch.zeros(C, 3, 2)
    elif what == "stats on another GPU":
        st = on_gpu(torch.zeros(C, 3, 2), 1)
    elif what == "stats not 8-byte aligned":
        flat = torch.zeros(C * 6 + 1)
        st = on_gpu(flat[1 if flat.data_ptr() % 8 == 0 else 0:][:C * 6].view(C, 3, 2))
    elif what == "empty x":
        x = on_gpu(torch.zeros(C, 0))
    else:
        b.bank = {"bank on the CPU": torch.zeros(12 * C), "bank on another GPU": on_gpu(torch.zeros(12 * C), 1),
                  "short bank": on_gpu(torch.zeros(12 * C - 1)), "strided bank": on_gpu(torch.zeros(24 * C)[::2]),
                  "f64 bank": on_gpu(torch.zeros(12 * C, dtype=torch.float64))}[what]
    with pytest.raises(Composition):
        gen.adain_resblock1_fused(x, b, "rb", K, x_stats=st)


def test_resblock_call_rejects_what_its_kernels_cannot_take():
    """lkc_resblock from C: refused on the host, before anything is queued (no pointer here is a device address)."""
    blk = _lib.LkcResblock()
    blk.c, blk.k = C, K
    blk.w[:], blk.b[:], blk.alpha[:] = [4096] * 6, [4096] * 6, [4096] * 6

    def call(**kw):
        io = _lib.LkcResblockIo()
        io.x = io.bank = io.out = io.out_stats = 4096
        io.l = io.x_pitch = io.out_pitch = N
        for k, v in kw.items():
            setattr(io, k, v)
        return _lib.lib().lkc_resblock(ctypes.byref(blk), ctypes.byref(io), None), io

    rc, io = call()  # without a workspace: its size only
    assert rc == 0 and io.workspace_bytes > 0
    for kw in ({"stats": 4100}, {"out_stats": 4100}):
        assert call(**kw)[0] != 0 and "8-byte aligned" in _lib.last_error()
    blk.c = 65536
    assert call()[0] != 0 and "too many channels" in _lib.last_error()


@pytest.mark.parametrize("index", [(1, 1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1)])
def test_forward_refuses_operands_on_another_gpu(gen, monkeypatch, index):
    monkeypatch.setattr(gen, "_whole_model", lambda: object())
    monkeypatch.setattr(gen, "_forward_whole", lambda *a, **k: "whole")
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    t = 4
    args = [torch.zeros(512, t), torch.zeros(22, 60 * t + 1), torch.zeros(128)]
    assert gen.forward(*[on_gpu(a) for a in args]) == "whole"
    with pytest.raises(ops.OpError, match="the generator's device"):
        gen.forward(*[on_gpu(a, i) for a, i in zip(args, index)])


@pytest.fixture
def block():
    """A generator of one resblock on CPU tensors, with stand-ins for the prepared states: its pointer struct needs no GPU."""
    g = G.Generator.__new__(G.Generator)
    g.device, g.w, g.conv_state, g.bank_off, g._blocks, g._model = torch.device("cpu"), {}, {}, {}, {}, None
    for j in range(3):
        for n in (1, 2):
            conv = f"rb.convs{n}.{j}"
            g.w[conv + ".weight"], g.w[conv + ".bias"] = torch.zeros(C, C, K), torch.zeros(C)
            g.w[f"rb.alpha{n}.{j}"] = torch.ones(C)
            g.conv_state[conv] = types.SimpleNamespace(handle=4096 + 2 * j + n, shape=(C, C, K))
            g.bank_off[f"rb.adain{n}.{j}.fc"] = (2 * C * (2 * j + n - 1), 2 * C)
    g.bank_b = torch.zeros(12 * C)
    return g


def test_block_follows_its_weights(block):
    """A weight that was replaced, or moved in place, is the one that the next call uses."""
    first = block._block("rb", K)
    assert first is not None and block._block("rb", K) is first and block._block("rb", K + 2) is None
    new = torch.ones(C)
    block.w["rb.convs2.1.bias"] = new
    assert block._block("rb", K).b[3] == new.data_ptr()
    moved = torch.ones(C)
    block.w["rb.alpha1.2"].data = moved
    assert block._block("rb", K).alpha[4] == moved.data_ptr()
    block.conv_state["rb.convs1.0"] = types.SimpleNamespace(handle=77, shape=(C, C, K))
    assert block._block("rb", K).state[0] == 77
    again = block._block("rb", K)
    assert block._block("rb", K) is again


def test_block_leaves_odd_weights_to_the_composition(block):
    """Weights that the ops would refuse do not reach the kernels by address, also when they come later."""
    keep = dict(block.w), dict(block.conv_state)
    for name, t in (("rb.convs1.1.bias", torch.zeros(C - 1)), ("rb.alpha2.0", torch.zeros(C, dtype=torch.float64)),
                    ("rb.convs2.2.weight", torch.zeros(C, C, K + 2)), ("rb.convs2.2.bias", torch.zeros(2 * C)[::2]),
                    ("rb.convs2.2.bias", torch.zeros(C, device="meta"))):
        assert block._block("rb", K) is not None
        block.w[name] = t
        assert block._block("rb", K) is None, name
        block.w.update(keep[0])
    del block.w["rb.alpha1.0"]
    assert block._block("rb", K) is None
    block.w.update(keep[0])
    block.conv_state["rb.convs2.0"] = None
    assert block._block("rb", K) is None
    block.conv_state.update(keep[1])
    assert block._block("rb", K) is not None
