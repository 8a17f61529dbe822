"""Which calls take the whole-resblock / whole-forward library calls and which go through the op-by-op composition, with
its checks: the host logic in front of the launches, on CPU tensors that claim to live on a GPU."""
import pytest
import torch

from lokinfer_b200 import generator as G
from lokinfer_b200 import ops

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
