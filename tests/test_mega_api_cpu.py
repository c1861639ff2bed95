"""Host side of the fused MoE API without a GPU: the input loader of ``SymmBuffer`` (ue8m0 codes from power-of-two fp32
block scales), the argument rules of ``fp8_fp4_mega_moe`` in the order the reference states them
(``experiments/megamoe/python/deep_ep_experimental/megamoe/api.py:520-567``), shared-expert weight joining and the
statistics update.  The buffer object is assembled by hand around a recording engine; no kernel runs.
"""
import contextlib
import types

import pytest
import torch

from deepep_b200.models import mega_moe as MM
from deepep_b200.oracle import megamoe as O
from deepep_b200.utils.math import per_token_cast_to_fp8

H, I, K, E, M = 256, 128, 2, 4, 16


class RecordingEngine:
    def __init__(self):
        self.calls, self.sm_count = [], 4
        self.scratch = [dict(expert_rows=torch.tensor([3, 0, 5, 1, 9], dtype=torch.int32))]
        self.checked = 0

    def forward(self, ys, tokens, l1, l2, fused=True, x_bf16=None, timer=None):
        self.calls.append(dict(ys=ys, tokens=tokens, l1=l1, l2=l2, fused=fused, x_bf16=x_bf16, timer=timer))

    def check(self):
        self.checked += 1


def make_buffer(shared=0, mma_type="fp8xfp4", world=1):
    sym = object.__new__(MM.SymmBuffer)
    sym.hidden, sym.intermediate_hidden, sym.num_topk, sym.num_experts = H, I, K, E
    sym.num_max_tokens_per_rank, sym.num_shared_experts, sym.mma_type, sym.world_size = M, shared, mma_type, world
    sym.device = torch.device("cpu")
    sym.x = torch.zeros((M, H), dtype=torch.float8_e4m3fn)
    sym.x_sf = torch.zeros((M, H // 32), dtype=torch.uint8)
    sym.topk_idx = torch.full((M, K), -1, dtype=torch.int32)
    sym.topk_weights = torch.zeros((M, K), dtype=torch.float32)
    sym.engine, sym._joined, sym.batch_size = RecordingEngine(), {}, 0
    return sym


def weights(experts=E, seed=0):
    return MM.transform_weights_for_mega_moe(*O.make_weights(experts, H, I, seed))


def test_load_inputs_converts_power_of_two_block_scales():
    sym = make_buffer()
    x = torch.randn((5, H), generator=torch.Generator().manual_seed(2)) * 4
    q, scale = per_token_cast_to_fp8(x, use_ue8m0=True)                       # fp32 [5, H / 128], powers of two
    idx = torch.tensor([[0, 1], [2, 3], [1, -1], [0, 3], [2, 1]])
    w = torch.rand((5, K))
    assert sym.load_inputs(q, scale, idx, w) is sym and sym.batch_size == 5
    # every 128-block scale serves its four 32-value blocks; decoding the codes gives the input scales back exactly
    decoded = torch.exp2(sym.x_sf[:5].float() - 127)
    assert torch.equal(decoded, scale.repeat_interleave(4, dim=1))
    assert torch.equal(sym.x[:5].view(torch.uint8), q.view(torch.uint8))
    assert sym.topk_idx[:5].tolist() == idx.tolist() and torch.equal(sym.topk_weights[:5], w)
    assert torch.equal(O.dequantize_mxfp8(sym.x[:5], sym.x_sf[:5]), (q.float().view(5, -1, 128) * scale.unsqueeze(2)).view(5, H))
    # ue8m0 codes are taken as they are
    codes, sf = O.quantize_mxfp8(x)
    sym.load_inputs(codes, sf, idx, w)
    assert torch.equal(sym.x_sf[:5], sf)
    # scales that ue8m0 cannot carry exactly are refused, as are wrong shapes and oversized batches
    with pytest.raises(ValueError, match="powers of two"):
        sym.load_inputs(q, scale * 1.5, idx, w)
    with pytest.raises(ValueError, match="x_sf must be"):
        sym.load_inputs(q, scale[:, :1], idx, w)
    with pytest.raises(ValueError, match="e4m3"):
        sym.load_inputs(q.float(), scale, idx, w)
    big = torch.zeros((M + 1, H), dtype=torch.float8_e4m3fn)
    with pytest.raises(ValueError, match="batch"):
        sym.load_inputs(big, torch.ones((M + 1, H // 128)), idx, w)
    with pytest.raises(ValueError, match="batch size"):
        sym.prepare(M + 1)
    sym.validate_inputs(5, x=torch.zeros((5, H), dtype=torch.bfloat16))
    with pytest.raises(ValueError, match="x override"):
        sym.validate_inputs(5, x=torch.zeros((5, H)))
    with pytest.raises(ValueError, match="batch size"):
        sym.validate_inputs(0)
    sym.topk_idx[0, 0] = E
    with pytest.raises(ValueError, match="outside"):
        sym.validate_inputs(5)
    sym.topk_idx[0, 0] = 0
    sym.topk_weights[1, 1] = float("nan")
    with pytest.raises(ValueError, match="finite"):
        sym.validate_inputs(5)


def test_inputs_are_copied_on_the_buffers_device(monkeypatch):
    """The copy kernel is launched with the buffer's device current, whichever device the caller works on."""
    log, current = [], [0]

    @contextlib.contextmanager
    def device(index):
        before, current[0] = current[0], index
        yield
        current[0] = before

    monkeypatch.setattr(torch.cuda, "current_device", lambda: current[0])
    monkeypatch.setattr(torch.cuda, "device", device)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda d: types.SimpleNamespace(cuda_stream=100 + getattr(d, "index", d)))

    def tensor(dtype, *shape):
        return types.SimpleNamespace(dtype=dtype, shape=shape, device=torch.device("cuda", 1), data_ptr=lambda: 4096, is_contiguous=lambda: True)

    sym = object.__new__(MM.SymmBuffer)
    sym.engine = object.__new__(MM.MegaEngine)
    sym.engine.C = types.SimpleNamespace(mega_load=lambda *args: log.append((current[0], args[-1])))
    sym.num_max_tokens_per_rank, sym.hidden, sym.num_topk, sym.device = 8, 256, 2, torch.device("cuda", 1)
    sym.x, sym.x_sf = tensor(torch.float8_e4m3fn, 8, 256), tensor(torch.uint8, 8, 8)
    sym.topk_idx, sym.topk_weights = tensor(torch.int32, 8, 2), tensor(torch.float32, 8, 2)
    given = tensor(torch.float8_e4m3fn, 3, 256), tensor(torch.uint8, 3, 8), tensor(torch.int64, 3, 2), tensor(torch.float32, 3, 2)
    for here in (0, 1):
        current[0] = here
        sym._copy_inputs(*given)
        assert current[0] == here
    assert log == [(1, 101), (1, 101)]


def test_an_engine_is_ready_for_any_stream(monkeypatch):
    """The counters that calls find zero are zeroed on the stream on which the engine is made; it is waited for before a call on
    another stream can read them."""
    log = []
    zeros = torch.zeros
    monkeypatch.setattr(torch, "zeros", lambda *a, **k: (log.append("zeros"), zeros(*a, **k))[1])
    monkeypatch.setattr(MM, "require_native", lambda name: types.SimpleNamespace(mega_input_offsets=lambda *a: [0] * 6))
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda device: types.SimpleNamespace(multi_processor_count=148))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device: types.SimpleNamespace(synchronize=lambda: log.append("synchronize")))
    layout = types.SimpleNamespace(world=1, max_tokens=4, hidden=256, topk=2, mega=0)
    engine = MM.MegaEngine([None], layout, torch.device("cpu"), 4, 128)
    assert "clean" in engine.scratch[0] and log.count("synchronize") == 1 and log[-1] == "synchronize"


@pytest.mark.parametrize("world,experts,hidden,inter,topk,tokens,swapped", [
    (1, 8, 1024, 512, 2, 96, True), (1, 8, 1024, 512, 2, 100, False), (1, 8, 1024, 512, 2, 128, False),      # 24, 25 and 32 rows per expert
    (1, 32, 2048, 768, 4, 192, True), (1, 32, 2048, 768, 4, 256, False),                                      # 75 MB of weights
    (1, 64, 2048, 768, 8, 256, True), (1, 32, 7168, 2048, 8, 128, True), (1, 32, 7168, 2048, 8, 129, False),  # more than the L2 holds
    (4, 16, 4096, 1024, 2, 48, True), (4, 16, 4096, 1024, 2, 64, False), (2, 32, 4096, 1536, 4, 128, True)])
def test_when_operands_are_swapped(world, experts, hidden, inter, topk, tokens, swapped):
    """Both sides of the line, which depends on the weights that one rank holds."""
    engine = object.__new__(MM.MegaEngine)
    engine.world, engine.E, engine.L, engine.H, engine.I, engine.K = world, experts, experts // world, hidden, inter, topk
    assert engine.use_swap([tokens] * world) is swapped


@pytest.mark.parametrize("experts,topk,shared,tokens,alone", [(32, 8, 0, 64, True), (32, 8, 0, 65, False), (128, 7, 1, 64, True), (8, 1, 0, 513, False),
                                                               (129, 8, 0, 32, True), (129, 8, 1, 32, False), (1024, 8, 0, 64, False)])
def test_when_every_block_derives_the_layout(experts, topk, shared, tokens, alone):
    """Both sides of the line: 512 slots, 256 with more than 128 experts."""
    engine = object.__new__(MM.MegaEngine)
    engine.C, engine.E, engine.K, engine.S = types.SimpleNamespace(mega_alone_slots=512), experts, topk, shared
    assert engine.use_alone([tokens]) is alone


def test_forward_argument_rules_and_what_reaches_the_engine():
    sym, (l1, l2) = make_buffer(), weights()
    y = torch.zeros((6, H), dtype=torch.bfloat16)
    stats = torch.tensor([10, 10, 10, 10], dtype=torch.int32)
    assert MM.fp8_fp4_mega_moe(y, l1, l2, sym, cumulative_local_expert_recv_stats=stats) is None
    call = sym.engine.calls[-1]
    assert call["ys"][0] is y and call["tokens"] == [6] and call["l1"][0] is l1 and call["l2"][0] is l2
    assert call["fused"] is True and call["x_bf16"] is None and call["timer"] is None
    assert stats.tolist() == [13, 10, 15, 11]                                  # the routed experts' rows, not the fifth entry
    xb = torch.zeros((6, H), dtype=torch.bfloat16)
    MM.fp8_fp4_mega_moe(y, l1, l2, sym, x=xb, fused=False)
    assert sym.engine.calls[-1]["x_bf16"][0] is xb and sym.engine.calls[-1]["fused"] is False and sym.engine.checked == 0
    for kwargs, kind, message in (
            (dict(recipe=(1, 1, 128)), NotImplementedError, "recipe"),
            (dict(activation="gelu"), NotImplementedError, "SwiGLU"),
            (dict(activation_clamp=7.0), NotImplementedError, "SwiGLU"),
            (dict(fast_math=False), NotImplementedError, "SwiGLU"),
            (dict(shared_l1_weights=l1), ValueError, "both shared"),
            (dict(shared_l1_weights=l1, shared_l2_weights=l2), ValueError, "num_shared_experts"),
            (dict(x=xb.float()), ValueError, "x override"),
            (dict(cumulative_local_expert_recv_stats=stats.long()), ValueError, "int32"),
            (dict(timer=torch.zeros((4, 8), dtype=torch.int32)), ValueError, "allocate_timer"),
            (dict(timer=torch.zeros((4, 8), dtype=torch.int64), fused=False), ValueError, "fused")):
        with pytest.raises(kind, match=message):
            MM.fp8_fp4_mega_moe(y, l1, l2, sym, **kwargs)
    with pytest.raises(TypeError, match="SymmBuffer"):
        MM.fp8_fp4_mega_moe(y, l1, l2, object())
    with pytest.raises(TypeError, match="transform_weights"):
        MM.fp8_fp4_mega_moe(y, (None, None), l2, sym)
    with pytest.raises(ValueError, match="bf16"):
        MM.fp8_fp4_mega_moe(y.float(), l1, l2, sym)
    with pytest.raises(ValueError, match="non-empty"):
        MM.fp8_fp4_mega_moe(y[:0], l1, l2, sym)
    with pytest.raises(ValueError, match="experts"):
        MM.fp8_fp4_mega_moe(y, *weights(experts=2), sym)
    with pytest.raises(ValueError, match="other kind"):
        MM.fp8_fp4_mega_moe(y, l1, l2, make_buffer(mma_type="fp8xfp8"))


def test_shared_experts_are_joined_once_per_weight_set():
    sym, (l1, l2), (s1, s2) = make_buffer(shared=1), weights(), weights(experts=1, seed=9)
    y = torch.zeros((4, H), dtype=torch.bfloat16)
    MM.fp8_fp4_mega_moe(y, l1, l2, sym, s1, s2)
    first = sym.engine.calls[-1]
    j1, j2 = first["l1"][0], first["l2"][0]
    assert j1.experts == E + 1 and j2.experts == E + 1 and (j1.n, j1.k, j2.n, j2.k) == (2 * I, H, H, I)
    assert torch.equal(j1.packed[:l1.packed.shape[0]], l1.packed) and torch.equal(j1.packed[l1.packed.shape[0]:], s1.packed)
    assert torch.equal(j2.sf_chunks, torch.cat([l2.sf_chunks, s2.sf_chunks]))
    MM.fp8_fp4_mega_moe(y, l1, l2, sym, s1, s2)
    assert sym.engine.calls[-1]["l1"][0] is j1 and sym.engine.calls[-1]["l2"][0] is j2      # joined once, reused
    f1, f2 = MM.transform_weights_for_mega_moe(*O.make_fp8_weights(1, H, I, 3))
    with pytest.raises(ValueError, match="weight type"):
        sym.joined_weights(l1, f1)
    with pytest.raises(ValueError, match="num_shared_experts"):
        MM.fp8_fp4_mega_moe(y, l1, l2, sym)


def test_joined_weights_are_never_stale():
    """The kernel gets the addresses of the tensors that hold the weights now: after a change in place (through ``.data`` too), after
    a field was given another tensor, and for another set of weights."""
    sym, (l1, _), (s1, _) = make_buffer(shared=1), weights(), weights(experts=1, seed=9)
    first = sym.joined_weights(l1, s1)
    l1.packed.add_(1)
    s1.sf_chunks.data.add_(1)
    j = sym.joined_weights(l1, s1)
    assert torch.equal(j.packed, torch.cat([l1.packed, s1.packed])) and torch.equal(j.sf_chunks, torch.cat([l1.sf_chunks, s1.sf_chunks]))
    l1.packed = l1.packed.clone()
    hold = []
    args = MM._weight_args(sym.joined_weights(l1, s1), hold)
    assert (args["b"], args["sfb"], args["b_rows"]) == (l1.packed.data_ptr(), l1.sf_chunks.data_ptr(), E * 2 * I)
    assert (args["b2"], args["sfb2"], args["b2_rows"]) == (s1.packed.data_ptr(), s1.sf_chunks.data_ptr(), 2 * I)
    assert "b2" not in MM._weight_args(l1, hold) and MM._weight_args(l1, hold)["b"] == l1.packed.data_ptr()
    # shared weights at an odd address, or strided, are copied for the launch as the copy engine cannot read them there
    odd = MM.MegaWeights(torch.zeros(s1.packed.numel() + 8, dtype=torch.uint8)[8:].view_as(s1.packed).copy_(s1.packed), s1.sf_chunks, 1, s1.n, s1.k)
    strided = MM.MegaWeights(s1.packed, torch.stack([s1.sf_chunks, s1.sf_chunks], 1)[:, 0], 1, s1.n, s1.k)
    for w in (odd, strided):
        args = MM._weight_args(sym.joined_weights(l1, w), hold)
        assert "b2" not in args and (args["b"], args["sfb"], args["b_rows"]) == (hold[-2].data_ptr(), hold[-1].data_ptr(), (E + 1) * 2 * I)
        assert torch.equal(hold[-2], torch.cat([l1.packed, s1.packed])) and torch.equal(hold[-1], torch.cat([l1.sf_chunks, s1.sf_chunks]))
    other, _ = weights(experts=1, seed=10)
    other.packed.set_(s1.packed)                                    # another set of weights at the same address
    k = sym.joined_weights(l1, other)
    assert k is not first and torch.equal(k.sf_chunks[-other.sf_chunks.numel():], other.sf_chunks)


def test_weight_transform_shapes_and_rules():
    (w1, w1_sf), (w2, w2_sf) = O.make_weights(E, H, I, 0)
    l1, l2 = MM.transform_weights_for_mega_moe((w1, w1_sf), (w2, w2_sf))
    assert (l1.experts, l1.n, l1.k, l1.fp8) == (E, 2 * I, H, False) and (l2.experts, l2.n, l2.k) == (E, H, I)
    assert l1.packed.dtype == torch.uint8 and l1.packed.numel() == w1.numel() and l2.packed.numel() == w2.numel()
    assert l1.sf_chunks.numel() >= w1_sf.numel() and l1.sf_chunks.numel() % 512 == 0
    (f1, f1_sf), (f2, f2_sf) = O.make_fp8_weights(E, H, I, 1)
    g1, g2 = MM.transform_weights_for_mega_moe((f1, f1_sf), (f2, f2_sf))
    assert g1.fp8 and g2.fp8 and g1.packed.numel() == f1.numel() and (g1.k, g2.k) == (H, I)
    with pytest.raises(ValueError, match="same kind"):
        MM.transform_weights_for_mega_moe((f1, f1_sf), (w2, w2_sf))
    # the reference documents the scales as [L, N, K / 64, 2]: the same bytes, accepted as they are
    r1, r2 = MM.transform_weights_for_mega_moe((w1, w1_sf.view(E, 2 * I, H // 64, 2)), (w2, w2_sf.view(E, H, I // 64, 2)), shared=True)
    assert torch.equal(r1.sf_chunks, l1.sf_chunks) and torch.equal(r2.sf_chunks, l2.sf_chunks) and torch.equal(r1.packed, l1.packed)
    with pytest.raises(NotImplementedError, match="SwiGLU"):
        MM.transform_weights_for_mega_moe((w1, w1_sf), (w2, w2_sf), "gelu")


def test_kernel_failure_report_names_the_wait():
    """``MegaEngine.check`` turns the kernel's error word (which wait ran out) into a message; zero means no failure."""
    eng = object.__new__(MM.MegaEngine)
    eng.scratch = [dict(err=torch.zeros(1, dtype=torch.int32)), dict(err=torch.zeros(1, dtype=torch.int32))]
    eng.check()
    eng.scratch[1]["err"][0] = 8
    with pytest.raises(RuntimeError, match="local rank 1: it was waiting for operands arriving in a stage"):
        eng.check()
    eng.scratch[1]["err"][0] = 77
    with pytest.raises(RuntimeError, match="site 77"):
        eng.check()
    assert set(MM.MegaEngine.WAIT_SITES) == set(range(1, 11))
