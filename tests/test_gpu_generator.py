"""Whole-path parity: one AdaINResBlock1, the full generator (fused and basic graphs) against the CPU oracle and the
committed golden fixture, CUDA-graph replay, and size-independent properties at the full 26 s size."""
import numpy as np
import pytest
import torch

from lokinfer_b200 import synth
from oracle import kokoro_oracle as O
from util import REL_L2, WAVE_MAXABS, check_stats, rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gen(cuda):
    from lokinfer_b200 import Generator
    return Generator(synth.generator_weights(0), cuda)


def _inputs(cuda, t, seed=1):
    from lokinfer_b200 import ops
    inp = synth.generator_inputs(t, seed)
    return inp, [ops.to_cuda(inp[k], cuda) for k in ("x", "har", "s")]


@pytest.mark.parametrize("c,l,k", [(16, 300, 7), (128, 1201, 3), (128, 2000, 11), (256, 640, 7), (80, 5700, 3)])
def test_resblock(cuda, c, l, k):
    """Config 0 at reduced length: one AdaINResBlock1 (kernel k, dilations 1/3/5) through the fused ops."""
    from lokinfer_b200 import Generator, ops
    sd, x, s = synth.resblock_case(c, l, k, 100 + c + k)
    g = Generator(sd, cuda)
    out, st = g.adain_resblock1_fused(ops.to_cuda(x, cuda), g.style(ops.to_cuda(s, cuda)), "rb", k)
    sd32 = {n: O.T(v) for n, v in sd.items()}
    ref, rst = O.adain_resblock1_fused(O.T(x), O.style_bank(sd32, O.T(s)), sd32, "rb", k)
    sd64 = {n: O.T(v, torch.float64) for n, v in sd.items()}
    ref64, _ = O.adain_resblock1_fused(O.T(x, torch.float64), O.style_bank(sd64, O.T(s, torch.float64)), sd64, "rb", k)
    got = out.cpu().numpy()
    # six chained convs: the per-op bar compounds; the float64 golden is the arbiter
    assert rel_l2(got, ref.numpy()) <= 6 * REL_L2
    assert rel_l2(got, ref64.numpy()) <= 2 * rel_l2(ref.numpy(), ref64.numpy()) + 1e-6
    np.testing.assert_allclose(st.cpu().numpy()[..., 0], rst.numpy()[..., 0], atol=1e-4, rtol=1e-4)


def test_generator_golden(cuda, gen):
    from pathlib import Path
    gold = np.load(Path(__file__).resolve().parent / "golden" / "kokoro_golden.npz")
    _, d = _inputs(cuda, 4)
    post, audio = gen.forward(*d, outputs=("post", "audio"))
    assert tuple(audio.shape) == (1200,) and tuple(post.shape) == (22, 241)
    assert np.abs(audio.cpu().numpy() - gold["gen_audio_f32"]).max() <= WAVE_MAXABS
    assert np.abs(audio.cpu().numpy() - gold["gen_audio_f64"]).max() <= WAVE_MAXABS
    assert rel_l2(post.cpu().numpy(), gold["gen_post_f64"]) <= 1e-4


@pytest.mark.parametrize("t", [1, 7, 16])
@pytest.mark.parametrize("fused", [True, False])
def test_generator_vs_oracle(cuda, gen, t, fused):
    inp, d = _inputs(cuda, t, seed=3 + t)
    audio = gen.forward(*d, fused=fused).cpu().numpy()
    sd = synth.generator_weights(0)
    ref32 = O.generator(sd, O.T(inp["x"]), O.T(inp["har"]), O.T(inp["s"]), fused=fused).numpy()
    dt = torch.float64
    ref64 = O.generator(sd, O.T(inp["x"], dt), O.T(inp["har"], dt), O.T(inp["s"], dt), fused=fused).numpy()
    sh = synth.shapes(t)
    assert audio.shape == (sh["S"],) == ref32.shape
    assert np.abs(audio - ref32).max() <= WAVE_MAXABS
    assert np.abs(audio - ref64).max() <= WAVE_MAXABS


def _oracle_stages(inp, dt, fused=True):
    sd = synth.generator_weights(0)
    return O.generator(sd, O.T(inp["x"], dt), O.T(inp["har"], dt), O.T(inp["s"], dt), fused=fused, stages=True)


@pytest.mark.parametrize("t", [320, 333, 797])
def test_generator_baseline_configs_vs_oracle(cuda, gen, t):
    """BASELINE config 1 (the 4 s sentence case, T = 320) and two utterance lengths of config 3 (T in 120..800, one
    odd: odd T makes every row pitch of stage 0 odd as well) against the CPU oracle in float32 and float64:
    the eager forward with concurrent streams, the same forward on one stream, and the captured-graph path with
    host buffers (Generator.synthesize). Bars: waveform max-abs <= 1e-4, conv_post logits rel-L2, and the GPU's
    error against float64 within 2x the float32 oracle's own."""
    inp, d = _inputs(cuda, t, seed=40 + t)
    post, audio = gen.forward(*d, outputs=("post", "audio"))
    audio_1s = gen.forward(*d, concurrent=False)
    host = [torch.from_numpy(inp[k]).pin_memory() for k in ("x", "har", "s")]
    audio_graph = gen.synthesize(*host).numpy().copy()
    sh = synth.shapes(t)
    assert tuple(audio.shape) == (sh["S"],) and tuple(post.shape) == (22, sh["L1"])
    r32, r64 = _oracle_stages(inp, torch.float32), _oracle_stages(inp, torch.float64)
    a32, a64 = r32["audio"].numpy(), r64["audio"].numpy()
    got = audio.cpu().numpy()
    assert np.abs(got - a32).max() <= WAVE_MAXABS
    assert np.abs(got - a64).max() <= WAVE_MAXABS
    np.testing.assert_array_equal(audio_1s.cpu().numpy(), got)
    np.testing.assert_array_equal(audio_graph, got)
    p = post.cpu().numpy()
    e_gpu, e_cpu = rel_l2(p, r64["post"].numpy()), rel_l2(r32["post"].numpy(), r64["post"].numpy())
    assert rel_l2(p, r32["post"].numpy()) <= 48 * REL_L2  # 48 chained fused convs
    assert e_gpu <= 2 * e_cpu + 1e-6
    assert rel_l2(got, a64) <= 2 * rel_l2(a32, a64) + 1e-6
    from lokinfer_b200 import ops
    assert ops.conv_tc_status() == 0


@pytest.mark.parametrize("k", [3, 7, 11])
@pytest.mark.parametrize("l", [19200, 19201])
def test_resblock_config0_full_length(cuda, k, l):
    """BASELINE config 0 at its full length: one AdaINResBlock1 at C = 128, L = 19200 (and 19201, the generator's
    real stage-1 length for T = 320) for each kernel size, against the float32 and float64 oracle."""
    from lokinfer_b200 import Generator, ops
    sd, x, s = synth.resblock_case(128, l, k, 300 + k)
    g = Generator(sd, cuda)
    with ops.padded_rows():
        out, st = g.adain_resblock1_fused(ops.to_cuda(x, cuda, rows=True), g.style(ops.to_cuda(s, cuda)), "rb", k)
    plain, st_plain = g.adain_resblock1_fused(ops.to_cuda(x, cuda), g.style(ops.to_cuda(s, cuda)), "rb", k)
    assert torch.equal(out, plain) and torch.equal(st, st_plain)  # padded rows (TMA) and contiguous rows agree
    sd32 = {n: O.T(v) for n, v in sd.items()}
    ref, rst = O.adain_resblock1_fused(O.T(x), O.style_bank(sd32, O.T(s)), sd32, "rb", k)
    sd64 = {n: O.T(v, torch.float64) for n, v in sd.items()}
    ref64, _ = O.adain_resblock1_fused(O.T(x, torch.float64), O.style_bank(sd64, O.T(s, torch.float64)), sd64, "rb", k)
    got = out.cpu().numpy()
    assert got.shape == (128, l)
    assert rel_l2(got, ref.numpy()) <= 6 * REL_L2
    assert rel_l2(got, ref64.numpy()) <= 2 * rel_l2(ref.numpy(), ref64.numpy()) + 1e-6
    np.testing.assert_allclose(st.cpu().numpy()[..., 0], rst.numpy()[..., 0], atol=1e-4, rtol=1e-4)
    assert ops.conv_tc_status() == 0


def test_generator_config2_stages_vs_oracle(cuda, gen):
    """BASELINE config 2 (the 26 s paragraph case, T = 2080) against the float32 oracle run once on the CPU: the
    three resblock outputs of each stage, the conv_post logits and the waveform."""
    t = 2080
    inp, d = _inputs(cuda, t, seed=5)
    post, audio, s0, s1 = gen.forward(*d, outputs=("post", "audio", "stage0", "stage1"))
    ref = _oracle_stages(inp, torch.float32)
    for name, got_rb in (("stage0", s0), ("stage1", s1)):
        for j in range(3):
            assert rel_l2(got_rb[j].cpu().numpy(), ref[name][j].numpy()) <= 24 * REL_L2, (name, j)
    assert rel_l2(post.cpu().numpy(), ref["post"].numpy()) <= 48 * REL_L2
    assert np.abs(audio.cpu().numpy() - ref["audio"].numpy()).max() <= WAVE_MAXABS
    # stage0 / stage1 make the forward run op by op; without them it is one library call
    post, audio = gen.forward(*d, outputs=("post", "audio"))
    assert rel_l2(post.cpu().numpy(), ref["post"].numpy()) <= 48 * REL_L2
    assert np.abs(audio.cpu().numpy() - ref["audio"].numpy()).max() <= WAVE_MAXABS
    from lokinfer_b200 import ops
    assert ops.conv_tc_status() == 0


def test_graph_replay_matches_eager(cuda, gen):
    inp, d = _inputs(cuda, 9, seed=21)
    eager = gen.forward(*d).cpu().numpy()
    host = [torch.from_numpy(inp[k]).pin_memory() for k in ("x", "har", "s")]
    a1 = gen.synthesize(*host).numpy().copy()
    a2 = gen.synthesize(*host).numpy().copy()
    np.testing.assert_array_equal(a1, eager)
    np.testing.assert_array_equal(a1, a2)


def test_planned_arena(cuda):
    """The captured forward lives in a planned arena: identical samples to a capture without the plan (every intermediate
    has memory of its own) and to the eager forward, in well under the memory of keeping every intermediate."""
    from lokinfer_b200 import Generator, ops
    t = 416
    inp = synth.generator_inputs(t, 9)
    g1, g2 = Generator(synth.generator_weights(0), cuda), Generator(synth.generator_weights(0), cuda)
    d = [ops.to_cuda(inp[k], cuda) for k in ("x", "har", "s")]
    eager = g1.forward(*d)
    b1, b2 = g1.capture(t), g2.capture(t, planned=False)
    assert "arena" in b1 and "arena" not in b2
    assert b1["arena_bytes"] <= 0.55 * b1["unplanned_bytes"]
    for b in (b1, b2):
        for k, v in zip(("x", "har", "s"), d):
            b[k].copy_(v)
        for _ in range(3):
            b["graph"].replay()
    torch.cuda.synchronize()
    assert torch.equal(b1["audio"], eager) and torch.equal(b2["audio"], eager)
    assert ops.conv_tc_status() == 0


def test_many_captures_keep_their_plans_valid(cuda):
    """One generator captures more lengths than torch's stream pool has streams (32): a stream made for a later
    capture can be the same CUDA stream as one of the generator's side streams. The memory plan must still be made
    for the concurrency the captured graph really has: every replay equals the eager forward."""
    from lokinfer_b200 import Generator, ops
    g = Generator(synth.generator_weights(0), cuda)
    lengths = list(range(40, 40 + 36))
    worst = 0.0
    for i, t in enumerate(lengths):
        inp = synth.generator_inputs(t, 500 + i)
        d = [ops.to_cuda(inp[k], cuda) for k in ("x", "har", "s")]
        eager = g.forward(*d)
        unplanned = g._forward_whole(g._whole_model(), *d, ("audio",), True, planned=False)
        assert torch.equal(unplanned, eager), (i, t)
        b = g.capture(t)
        for k, v in zip(("x", "har", "s"), d):
            b[k].copy_(v)
        for _ in range(2):
            b["graph"].replay()
        torch.cuda.synchronize()
        assert torch.equal(b["audio"], eager), (i, t)
        worst = max(worst, eager.abs().max().item())
    assert ops.conv_tc_status() == 0 and worst > 0


def test_full_size_properties(cuda, gen):
    """The 26 s case (T = 2080: L0 = 20800, L1 = 124801, 624000 samples), too large for the CPU oracle in a test:
    exact shapes, run-to-run determinism, agreement of the fused graph with the basic-kernel graph (two independent
    kernel sets), and the iSTFT tail against torch.istft on the same logits."""
    t = 2080
    sh = synth.shapes(t)
    _, d = _inputs(cuda, t, seed=5)
    post, audio = gen.forward(*d, outputs=("post", "audio"))
    assert tuple(post.shape) == (22, sh["L1"]) == (22, 124801) and tuple(audio.shape) == (624000,)
    audio2 = gen.forward(*d)
    assert torch.equal(audio, audio2)
    assert torch.isfinite(audio).all()
    basic = gen.forward(*d, fused=False)
    assert (audio - basic).abs().max().item() <= 2 * WAVE_MAXABS
    ref = O.istft_logits_torch(post)  # torch's own CUDA iSTFT
    assert (audio - ref).abs().max().item() <= 1e-5 * ref.abs().max().item()
    from lokinfer_b200 import ops
    assert ops.conv_tc_status() == 0
    # the tensor-core and CUDA-core conv kernels give the same waveform
    ops.set_conv_path("simt")
    try:
        simt = gen.forward(*d)
    finally:
        ops.set_conv_path("auto")
    assert (audio - simt).abs().max().item() <= WAVE_MAXABS


def test_synthesis_pipeline_matches_synthesize(cuda, gen):
    """Generator.pipeline (two utterances in flight, copies overlapping compute) returns, for every utterance of a
    stream of different inputs, exactly what Generator.synthesize returns for it alone."""
    t = 200
    hosts, want = [], []
    for i in range(5):
        inp, _ = _inputs(cuda, t, seed=70 + i)
        h = [torch.from_numpy(inp[k]).pin_memory() for k in ("x", "har", "s")]
        hosts.append(h)
        want.append(gen.synthesize(*h).numpy().copy())
    pipe = gen.pipeline(t, depth=2)
    outs = [torch.empty(want[0].shape, dtype=torch.float32).pin_memory() for _ in hosts]
    tickets = [pipe.submit(*h, o) for h, o in zip(hosts, outs)]
    for k in tickets:
        pipe.wait(k)
    for o, w in zip(outs, want):
        np.testing.assert_array_equal(o.numpy(), w)
    assert not np.array_equal(want[0], want[1])


def test_style_bank_of_another_generator(cuda, gen):
    """A block of a generator made from a subset of the state dict, with the full model's style bank: the offsets are the
    bank's own. Same bits as the block run op by op."""
    from lokinfer_b200 import Generator, ops
    full = synth.generator_weights(0)
    part = Generator({n: v for n, v in full.items() if n.startswith("resblocks.4.")}, cuda)
    s, x = torch.randn(128, device=cuda), torch.randn(128, 1201, device=cuda)
    bank = gen.style(s)
    assert part.bank_off["resblocks.4.adain1.0.fc"] != bank.off["resblocks.4.adain1.0.fc"]
    out, st = part.adain_resblock1_fused(x, bank, "resblocks.4", 7)
    ref, rst = part.adain_resblock1_fused(x, lambda name: bank(name), "resblocks.4", 7)
    assert torch.equal(out, ref) and torch.equal(st, rst)
    own, _ = gen.adain_resblock1_fused(x, bank, "resblocks.4", 7)
    assert rel_l2(out.cpu().numpy(), own.cpu().numpy()) <= REL_L2


def test_resblock_with_statistics(cuda):
    """Chunk statistics of x handed in: the same bits as without. Statistics that the kernels could not read are refused
    before any launch, as are an x or a style bank that does not fit the block."""
    from lokinfer_b200 import Generator, _lib, ops
    sd, x, s = synth.resblock_case(48, 1201, 3, 11)  # three channel chunks: CTAs of a split tile with unequal shares
    g = Generator(sd, cuda)
    dx, bank = ops.to_cuda(x, cuda), g.style(ops.to_cuda(s, cuda))
    st = ops.channel_stats_f32_cuda(dx)
    out, ost = g.adain_resblock1_fused(dx, bank, "rb", 3)
    again, ast = g.adain_resblock1_fused(dx, bank, "rb", 3, x_stats=st)
    assert torch.equal(out, again) and torch.equal(ost, ast)
    sd32 = {n: O.T(v) for n, v in sd.items()}
    ref, _ = O.adain_resblock1_fused(O.T(x), O.style_bank(sd32, O.T(s)), sd32, "rb", 3)
    assert rel_l2(out.cpu().numpy(), ref.numpy()) <= 6 * REL_L2
    odd = torch.empty(st.numel() + 1, device=cuda)[1:].view(st.shape).copy_(st)
    short = type(bank)(bank.bank[:-1], bank.off)
    with ops.Profile(time_kernels=False) as prof:
        for a, kw in (((dx, bank), {"x_stats": st.cpu()}), ((dx, bank), {"x_stats": odd}), ((dx.cpu(), bank), {}),
                      ((dx[:, :0], bank), {})):
            with pytest.raises((ops.OpError, _lib.LkcError)):
                g.adain_resblock1_fused(*a, "rb", 3, **kw)
        assert prof.count <= 1
    last = max(bank.off, key=lambda n: bank.off[n][0])
    assert last in ("rb.adain2.2.fc",)
    with pytest.raises(ops.OpError):
        g.adain_resblock1_fused(dx, short, "rb", 3)
    assert ops.conv_tc_status() == 0


def test_replaced_weights_take_effect(cuda):
    """Biases and alphas written into Generator.w after the first call are the ones that the next call uses, also when the
    replaced tensors' memory has been given to someone else."""
    from lokinfer_b200 import Generator
    g, (_, d) = Generator(synth.generator_weights(0), cuda), _inputs(cuda, 9, seed=4)
    before = g.forward(*d)
    for name in ("conv_post.bias", "ups.0.bias", "noise_convs.1.bias", "resblocks.2.convs2.1.bias", "noise_res.0.alpha1.0"):
        g.w[name] = g.w[name] * 1.25 + 0.01
        filler = [torch.full_like(g.w[name], float("nan")) for _ in range(4)]
        after = g.forward(*d)
        assert torch.isfinite(after).all() and not torch.equal(after, before), name
        fresh = Generator(synth.generator_weights(0), cuda)
        fresh.w.update({k: v.clone() for k, v in g.w.items()})
        assert torch.equal(fresh.forward(*d), after), name
        before = after
        del filler


def test_error_inside_a_forward_joins_its_streams(cuda):
    """A conv in the middle of the forward is refused on the host (its prepared state says another channel count) after
    work has been queued on the side streams. The caller's stream is ordered behind that work: a capture can end (with a
    stream left unjoined it cannot), and the generator works on afterwards."""
    import ctypes
    from lokinfer_b200 import Generator, _lib, ops
    g, (_, d) = Generator(synth.generator_weights(0), cuda), _inputs(cuda, 9, seed=6)
    want = g.forward(*d)
    ci = ctypes.c_int64.from_address(g.conv_state["resblocks.3.convs2.1"].handle + 16)  # wp, co, ci, k, ...
    assert ci.value == 128
    ci.value = 64
    graph = torch.cuda.CUDAGraph()
    try:
        with ops.Profile(time_kernels=False), pytest.raises(_lib.LkcError, match="does not match the weight shape"):
            g.forward(*d)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            with pytest.raises(_lib.LkcError, match="does not match the weight shape"):
                g.forward(*d)
    finally:
        ci.value = 128
    torch.cuda.synchronize()
    assert torch.equal(g.forward(*d), want) and ops.conv_tc_status() == 0


@pytest.mark.parametrize("t", [1, 7, 24, 121, 320, 747, 801])
@pytest.mark.parametrize("concurrent", [True, False])
def test_memory_plan_changes_nothing(cuda, gen, t, concurrent):
    """The whole-forward call in its planned workspace against the same call with memory of its own for every intermediate:
    the same bits, from workspaces full of NaN, one and several forwards of different lengths in flight."""
    from lokinfer_b200 import ops
    inp, d = _inputs(cuda, t, seed=60 + t)
    model = gen._whole_model()
    got = []
    for planned in (False, True, True):
        n, unplanned = gen._workspace_bytes(model, t, concurrent, planned)
        assert n <= unplanned if planned else n == unplanned
        ws = torch.full((n,), 255, dtype=torch.uint8, device=cuda)  # every float a NaN
        got.append(gen._forward_whole(model, *d, ("post", "audio"), concurrent, ws, planned))
    torch.cuda.synchronize()
    for post, audio in got[1:]:
        assert torch.equal(post, got[0][0]) and torch.equal(audio, got[0][1])
    assert torch.isfinite(got[0][1]).all() and ops.conv_tc_status() == 0


@pytest.mark.parametrize("t", [5, 24, 121, 320])
def test_whole_forward_agrees_with_the_composition(cuda, gen, t):
    """The whole-forward call and the op-by-op form differ in where the upsampled input is added, in who folds the
    statistics and in how partial sums are split, not beyond rounding."""
    from lokinfer_b200 import ops
    _, d = _inputs(cuda, t, seed=80 + t)
    post, audio = gen.forward(*d, outputs=("post", "audio"))
    post2, audio2, _ = gen.forward(*d, outputs=("post", "audio", "stage0"))
    assert rel_l2(post.cpu().numpy(), post2.cpu().numpy()) <= 48 * REL_L2
    assert (audio - audio2).abs().max().item() <= WAVE_MAXABS


def test_one_generator_in_several_threads(cuda, gen):
    """Forwards of different lengths from four threads, each on its own stream: every result as from one thread."""
    import threading
    jobs = [(t, _inputs(cuda, t, seed=90 + t)[1]) for t in (9, 24, 61, 130)]
    want = [gen.forward(*d).clone() for _, d in jobs]
    torch.cuda.synchronize()
    wrong, errors = [], []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream(device=cuda)):
                for _ in range(10):
                    model = gen._whole_model()
                    out = gen._forward_whole(model, *jobs[i][1], ("audio",), True)
                    if not torch.equal(out, want[i]):
                        wrong.append(jobs[i][0])
        except Exception as e:  # a thread's exception would be lost
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    torch.cuda.synchronize()
    assert not errors and not wrong


def test_captured_forward_keeps_its_weights(cuda):
    """A weight replaced after a capture: the graph goes on with the weights it was made from, also once the next forward
    has taken the new one and the old tensor is gone from the generator."""
    from lokinfer_b200 import Generator
    g, (_, d) = Generator(synth.generator_weights(0), cuda), _inputs(cuda, 9, seed=8)
    want, b = g.forward(*d), g.capture(9)
    for k, v in zip(("x", "har", "s"), d):
        b[k].copy_(v)
    for name in ("conv_post.bias", "resblocks.0.convs1.0.bias", "noise_res.1.alpha2.2"):
        g.w[name] = g.w[name] + 0.5
    assert not torch.equal(g.forward(*d), want)
    filler = [torch.full((n,), float("nan"), device=cuda) for n in (22, 128, 256) for _ in range(20)]
    b["graph"].replay()
    torch.cuda.synchronize()
    assert torch.equal(b["audio"], want)
    del filler


@pytest.mark.parametrize("stage,l", [(1, 19201), (1, 24833), (1, 28417), (1, 20000), (0, 9601), (0, 12001), (0, 15000)])
@pytest.mark.parametrize("k", [3, 11])
def test_whole_resblock_at_other_tile_widths(cuda, gen, stage, l, k):
    """Lengths whose convs take tiles of 160, 192 or 224 columns inside the whole-block call (statistics per 32 columns):
    against the op-by-op form, whose tiles are 256 wide, within the rounding of six convs in a row; the last columns alone too,
    where a tile ends inside the row."""
    from lokinfer_b200 import ops
    x = torch.randn((256, 128)[stage], l, generator=torch.Generator(device=cuda).manual_seed(l), device=cuda)
    gb = gen.style(torch.randn(128, generator=torch.Generator(device=cuda).manual_seed(k), device=cuda))
    prefix = f"resblocks.{3 * stage + (0 if k == 3 else 2)}"
    out, st = gen.adain_resblock1_fused(x, gb, prefix, k)
    with ops.use_allocator(lambda shape, device: torch.empty(shape, dtype=torch.float32, device=device)):
        want, want_st = gen.adain_resblock1_fused(x, gb, prefix, k)
    assert rel_l2(out.cpu().numpy(), want.cpu().numpy()) <= 6 * REL_L2
    assert rel_l2(out[:, -256:].cpu().numpy(), want[:, -256:].cpu().numpy()) <= 6 * REL_L2
    assert rel_l2(st.cpu().numpy(), want_st.cpu().numpy()) <= 6 * REL_L2
    assert torch.equal(out, gen.adain_resblock1_fused(x, gb, prefix, k)[0]) and ops.conv_tc_status() == 0


# Both stages at their longest split row: 74 tiles, two CTAs each.
FEW_TILES = [(stage, l) for stage, longest in ((0, 4736), (1, 9472)) for l in (1, 2, 127, 128, 129, 1024, 1025, 4097, longest)]


@pytest.mark.parametrize("stage,l", FEW_TILES)
def test_whole_resblock_with_few_tiles(cuda, gen, stage, l):
    """Lengths whose convs are split among CTAs, which fold the statistics (1 to 37 pairs per channel in stage 0, to 74 in stage 1)
    themselves: against the op-by-op form with its adain_affine, within the rounding of six convs in a row; the statistics of
    the result against that result. Rows far from zero, constant ones, and some whose first pair lies far from the others (the
    fold's variance is taken relative to it)."""
    from lokinfer_b200 import ops
    r = torch.Generator(device=cuda).manual_seed(l)
    c = (256, 128)[stage]
    x = torch.randn(c, l, generator=r, device=cuda)
    x[::5] += 300.0
    x[::7] = -1234.5
    x[1::11, :128] += 1e4
    gb = gen.style(torch.randn(128, generator=r, device=cuda))
    prefix = f"resblocks.{3 * stage + 1}"
    out, st = gen.adain_resblock1_fused(x, gb, prefix, 7)
    with ops.use_allocator(lambda shape, device: torch.empty(shape, dtype=torch.float32, device=device)):
        want, want_st = gen.adain_resblock1_fused(x, gb, prefix, 7)
    # what the block adds; on the big rows x's own rounding hides it
    d, live = out - x, [i for i in range(c) if i % 5 and i % 7 and i % 11 != 1]
    assert rel_l2(d[live].cpu().numpy(), (want - x)[live].cpu().numpy()) <= 6 * REL_L2
    far = [i for i in range(1, c, 11) if i % 5 and i % 7]
    assert rel_l2(d[far, 128:].cpu().numpy(), (want - x)[far, 128:].cpu().numpy()) <= 6 * REL_L2
    assert rel_l2(out.cpu().numpy(), want.cpu().numpy()) <= 6 * REL_L2
    assert rel_l2(st[..., 0].cpu().numpy(), want_st[..., 0].cpu().numpy()) <= 6 * REL_L2
    check_stats(st.cpu().numpy(), out.cpu().numpy())
    assert torch.equal(out, gen.adain_resblock1_fused(x, gb, prefix, 7)[0]) and ops.conv_tc_status() == 0


@pytest.mark.parametrize("form", ["har", "f0"])
def test_synthesize_reports_the_status_once(cuda, gen, form):
    """An activation beyond the f16 range raises from the call that met it, with that status and no other; the next call is
    clean and right."""
    from lokinfer_b200 import ops
    inp, _ = _inputs(cuda, 24)
    x, har, s = (torch.from_numpy(inp[k]).pin_memory() for k in ("x", "har", "s"))
    f0 = torch.from_numpy(synth.f0_curve(24, 3)).pin_memory()

    def call(x):
        return gen.synthesize(x, har, s) if form == "har" else gen.synthesize_f0(x, f0, 5, s)

    want = call(x).clone()
    with pytest.raises(RuntimeError, match=r"reported status 0x10000 "):
        call(x * 1e9)
    assert torch.equal(call(x), want) and ops.conv_tc_status() == 0
