"""Sizes at which the work split of the kernels changes: tile edges, remainders, smallest and largest of a range, against the
oracle (bit for bit: moved rows, and sums whose order and roundings the contract fixes)."""
import pytest
import torch

from deepep_b200.oracle import reference as R
from helpers import bits_equal, make_routes, make_weights
from test_ht_virtual_gpu import run_case
from test_ll_gpu import _case as ll_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("world,tokens,hidden,experts,topk,mode", [
    (1, [1], 7168, 256, 8, 2),              # one token: its row is cut into as many pieces as it has groups of 128 values
    (1, [256], 136, 8, 3, 0),               # the last group of a row is short
    (1, [33], 128, 1, 1, 1),                # a single group, a single expert
    (1, [250], 8192, 1000, 9, 2),           # several pieces of a row per warp, more experts than layout threads
    (2, [1, 256], 384, 1024, 8, 2),         # the most experts; own rows next to rows of a peer
    (4, [255, 0, 1, 32], 640, 8, 6, 0),
    (8, [9, 64, 65, 1, 31, 33, 2, 128], 1152, 64, 8, 1),
])
def test_low_latency_splits(world, tokens, hidden, experts, topk, mode):
    ll_case(world, tokens, hidden, experts, topk, mode, routes="invalid", repeats=3)


# one rank: mask words (32 tokens), batches of the table (2048 slots), one and two experts per thread, short last pieces
@pytest.mark.parametrize("tokens,hidden,experts,topk,mode", [
    (1, 8, 1, 1, 0), (1, 7168, 384, 8, 2), (31, 264, 513, 7, 0), (32, 256, 512, 16, 1), (33, 1032, 1024, 16, 0),
    (129, 128, 511, 16, 2), (256, 640, 1024, 16, 0), (255, 8192, 9, 9, 2), (256, 1280, 40, 3, 1)])
def test_low_latency_on_one_rank(monkeypatch, tokens, hidden, experts, topk, mode):
    """Repeated and out-of-range ids among the slots; rows, scales, weights, counts and the combine against the oracle, for which
    the later ones of repeated ids are empty slots."""
    from types import SimpleNamespace

    import test_ll_gpu

    def routes(kind, t, E, K, world, seed):
        g = torch.Generator().manual_seed(seed)
        idx = torch.randint(-1, E + 1, (t, K), generator=g)
        idx[::3, K // 2:] = idx[::3, :K - K // 2].clone()      # the second half repeats the first
        idx[1::4] = idx[1::4, :1].clone()                       # one expert in every slot
        return idx

    def first_only(idx):
        earlier = (idx.unsqueeze(2) == idx.unsqueeze(1)).tril(-1).any(2)
        return torch.where(earlier, torch.full_like(idx, -1), idx)

    monkeypatch.setattr(test_ll_gpu, "make_routes", routes)
    monkeypatch.setattr(test_ll_gpu, "R", SimpleNamespace(
        dispatch=lambda xs, idx, *args, **kw: R.dispatch(xs, [first_only(i) for i in idx], *args, **kw),
        low_latency_combine=R.low_latency_combine))
    test_ll_gpu._case(1, [tokens], hidden, experts, topk, mode)


@pytest.mark.parametrize("world,tokens,hidden,experts,topk,kw", [
    (1, [1], 7168, 256, 8, dict(dmode=2)),             # one token, many pieces
    (1, [65], 8, 16, 9, {}),                           # rows of one 16-byte piece; two groups of operands per token
    (1, [129], 520, 32, 16, dict(with_bias=True)),     # a short last span, sixteen operands
    (1, [2300], 1032, 8, 2, {}),                       # more tokens than warps
    (1, [640], 7168, 64, 6, dict(dmode=1, alignment=16)),
    (2, [64, 63], 1544, 32, 16, dict(with_bias=True)), # partials and more than eight local rows
    (4, [192, 1, 0, 65], 2048, 64, 12, dict(expand=False)),
    (8, [40] * 8, 1024, 64, 16, dict(dmode=2, alignment=128)),
])
def test_high_throughput_splits(world, tokens, hidden, experts, topk, kw):
    run_case(world, tokens, hidden, experts, topk, "invalid", repeats=2, **kw)


# one rank: tiles of 64 tokens, 16 ranges of them, one to four shares of a range, one thread per expert and none left for the hits
@pytest.mark.parametrize("tokens,experts,topk,expand,alignment", [
    (1, 1, 1, True, 1), (64, 5, 3, True, 16), (65, 1024, 16, True, 128), (1024, 1023, 8, True, 1), (1025, 64, 8, False, 1),
    (2049, 1024, 8, False, 1), (3000, 300, 11, True, 128), (16384, 1024, 16, True, 1), (16321, 40, 1, True, 16)])
def test_routing_plan_of_one_rank(tokens, experts, topk, expand, alignment):
    """Every field of the plan against its definition, with empty, out-of-range and repeated slots; one expert gets most tokens."""
    from deepep_b200.parallel.virtual import VirtualWorld

    g = torch.Generator().manual_seed(tokens + experts)
    idx = torch.randint(-1, experts + 1, (tokens, topk), generator=g)
    idx[torch.rand((tokens, topk), generator=g) < 0.2] = 0
    idx[5::9] = -1
    w = torch.rand((tokens, topk), generator=g)
    dev = torch.device("cuda")
    with VirtualWorld(1, tokens, 8, topk, timeout=10.0) as vw:
        plan = vw.engine.notify([idx.to(dev)], [w.to(dev)], experts, expand=expand, alignment=alignment, rank_matrix=True)[0]
        torch.cuda.synchronize()

    earlier = (idx.unsqueeze(2) == idx.unsqueeze(1)).tril(-1).any(2)
    valid = (idx >= 0) & (idx < experts) & ~earlier
    hit = valid.any(1)
    staged = torch.where(hit, hit.cumsum(0) - 1, torch.full((tokens,), -1))
    assert torch.equal(plan.send_slot[:, 0].cpu().long(), staged)
    starts = torch.cat((torch.zeros(1, dtype=torch.long), hit.long().cumsum(0)))
    tiles = -(-tokens // 64)
    assert torch.equal(plan.chunk_start[0].cpu().long(), starts[torch.arange(tiles + 1).mul(64).clamp(max=tokens)])
    assert torch.equal(plan.send_chunk_prefix[0].cpu().long(), starts[torch.arange(tiles) * 64])
    assert plan.rank_rows.tolist() == [0, int(hit.sum())] and plan.rank_tokens.tolist() == [tokens]
    assert plan.rank_matrix.tolist() == plan.rank_prefix.tolist() == [[int(hit.sum())]] and plan.num_staged_rows == int(hit.sum())
    t, k = valid.nonzero(as_tuple=True)
    counts = torch.bincount(idx[t, k], minlength=experts)
    assert plan.expert_counts.cpu().tolist() == counts.tolist() == plan.expert_counts_list
    blocks = (counts + alignment - 1) // alignment * alignment if expand else counts
    offsets = torch.cat((torch.zeros(1, dtype=torch.long), blocks.cumsum(0)))
    assert torch.equal(plan.expert_offsets.cpu().long(), offsets)
    meta, slot_row = plan.stage_meta.cpu().long(), torch.full((tokens, topk), -1)
    src, row_w = plan.recv_row_src.cpu().long(), plan.recv_w.cpu()
    mask = (valid.long() << torch.arange(topk)).sum(1)
    if expand:
        order = torch.argsort(idx[t, k], stable=True)
        t, k = t[order], k[order]
        e = idx[t, k]
        row = offsets[e] + torch.arange(len(e)) - (counts.cumsum(0) - counts)[e]
        slot_row[t, k] = row
        want, want_w = torch.full((int(offsets[-1]),), -1), torch.zeros((int(offsets[-1]),))
        want[row], want_w[row] = t * topk + k, w[t, k]
        assert plan.num_rows == len(want) and torch.equal(src[:len(want)], want) and torch.equal(row_w[:len(want)], want_w)
        at = valid.long().cumsum(1)[t, k] + 1
        assert torch.equal(meta[staged[t], at], row | k << 27) and torch.equal(meta[staged[hit], 1], valid.sum(1)[hit])
    else:
        assert plan.num_rows == int(hit.sum()) and torch.equal(src[:plan.num_rows], hit.nonzero()[:, 0] * topk)
        assert torch.equal(plan.recv_src_idx[:plan.num_rows].cpu().long(), hit.nonzero()[:, 0])
        assert torch.equal(row_w[:plan.num_rows], torch.where(valid, w, torch.zeros(()))[hit])
        assert torch.equal(plan.recv_idx[:plan.num_rows].cpu(), torch.where(valid, idx, torch.full_like(idx, -1))[hit])
        assert torch.equal(meta[staged[hit], 2], staged[hit]) and torch.equal(meta[staged[hit], 3], mask[hit])
    assert torch.equal(plan.slot_row.cpu().long(), slot_row) and torch.equal(meta[staged[hit], 0], hit.nonzero()[:, 0])


def test_v1_tables_of_several_ranks():
    """What the V1 handle is made of, with ranks of unequal size and one without tokens."""
    from deepep_b200.parallel.virtual import VirtualWorld

    world, tokens, experts, topk, dev = 4, [130, 0, 64, 201], 16, 3, torch.device("cuda")
    idx = [make_routes("empty", t, experts, topk, world, r) for r, t in enumerate(tokens)]
    with VirtualWorld(world, max(tokens), 64, topk, timeout=10.0) as vw:
        plans = vw.engine.notify([i.to(dev) for i in idx], [make_weights(t, topk, 1).to(dev) for t in tokens], experts, expand=False,
                                 rank_matrix=True)
        torch.cuda.synchronize()
        vw.engine.check_status()
    hits = [torch.stack([((i >= 0) & (i // (experts // world) == d)).any(1) for d in range(world)], 1).long() for i in idx]   # [T, P]
    matrix = torch.stack([h.sum(0) for h in hits])
    for r, plan in enumerate(plans):
        assert torch.equal(plan.rank_matrix.cpu().long(), matrix) and torch.equal(plan.rank_prefix.cpu().long(), matrix.cumsum(0))
        starts = torch.cat((torch.zeros((1, world), dtype=torch.long), hits[r].cumsum(0)))
        tiles = torch.arange(max(1, -(-tokens[r] // 64))) * 64
        assert torch.equal(plan.send_chunk_prefix.cpu().long(), starts[tiles].t())
        sources = torch.cat([h[:, r].nonzero()[:, 0] for h in hits])
        assert torch.equal(plan.recv_src_idx[:plan.num_rows].cpu().long(), sources)


@pytest.mark.parametrize("tokens,experts,topk,world", [(0, 8, 2, 2), (1, 1024, 16, 8), (40000, 24, 5, 1), (16385, 1000, 8, 4), (0, 1024, 16, 8),
                                                       (1, 512, 16, 8), (511, 64, 6, 1), (2048, 512, 3, 2), (2049, 512, 3, 2), (2048, 513, 8, 1)])
def test_v1_layout(tokens, experts, topk, world):
    from deepep_b200.ops import load_native

    dev = torch.device("cuda")
    idx = torch.randint(-2, experts + 2, (tokens, topk), generator=torch.Generator().manual_seed(tokens)).to(dev)
    per_rank, per_expert = (torch.full((n,), 77, dtype=torch.int32, device=dev) for n in (world, experts))
    in_rank = torch.ones((tokens, world), dtype=torch.bool, device=dev)
    load_native().layout(idx.data_ptr(), tokens, topk, experts, world, per_rank.data_ptr(), per_expert.data_ptr(), in_rank.data_ptr(),
                         torch.cuda.current_stream().cuda_stream)
    ok = (idx >= 0) & (idx < experts)
    want = torch.stack([(ok & (idx // (experts // world) == r)).any(1) for r in range(world)], 1)
    assert torch.equal(in_rank, want) and torch.equal(per_rank.long(), want.sum(0))
    assert torch.equal(per_expert.long(), torch.bincount(idx[ok], minlength=experts))


@pytest.mark.parametrize("dmode", [0, 1, 2])
@pytest.mark.parametrize("tokens,hidden,experts,topk,expand,alignment", [
    (1, 128, 4, 1, True, 1), (9, 1152, 16, 2, True, 16), (70, 1024, 7, 7, True, 128), (33, 8192, 64, 16, True, 1),
    (257, 2176, 48, 3, True, 1), (65, 4224, 32, 8, False, 1), (1, 128, 3, 3, False, 1)])
def test_one_rank_with_and_without_a_budget_of_blocks(filled_outputs, tokens, hidden, experts, topk, expand, alignment, dmode):
    """The kernels of one piece per warp (no budget) and those of a few persistent blocks give the same bits, rows, scales, zeroed
    padding, sums, biases and values alike; empty and out-of-range slots among them."""
    from deepep_b200.parallel.virtual import VirtualWorld
    from deepep_b200.utils.math import per_token_cast_to_fp8

    dev = torch.device("cuda")
    x = torch.randn((tokens, hidden), generator=torch.Generator().manual_seed(3)).bfloat16()
    idx = make_routes("empty" if tokens > 1 else "random", tokens, experts, topk, 1, 5)
    idx[1::7] = experts + 3
    w = make_weights(tokens, topk, 8).to(dev)
    src = tuple(t.to(dev) for t in per_token_cast_to_fp8(x)) if dmode == 1 else x.to(dev)
    bias = tuple(torch.randn((tokens, hidden), generator=torch.Generator().manual_seed(r)).bfloat16().to(dev) for r in (1, 2))
    with VirtualWorld(1, tokens, hidden, topk, timeout=10.0) as vw:
        eng = vw.engine
        plan = eng.notify([idx.to(dev)], [w], experts, expand=expand, alignment=alignment)
        got = [eng.dispatch([src], plan, dmode, blocks=blocks)[0] for blocks in (0, 5, 0)]
        rows = torch.randn((plan[0].num_rows, hidden), generator=torch.Generator().manual_seed(4)).bfloat16().to(dev)
        sums = []
        for blocks in (0, 5, 0):
            for b in (None, bias[0], bias):
                sums += eng.combine([rows], plan, [plan[0].recv_w], bias=None if b is None else [b], blocks=blocks)
            sums += eng.combine([rows], plan, [None], blocks=blocks)
        torch.cuda.synchronize()
        eng.check_status()
    for out, sf in got[1:]:
        assert bits_equal(out, got[0][0]) and (sf is None or bits_equal(sf, got[0][1]))
    for i, (out, out_w) in enumerate(sums):
        assert bits_equal(out, sums[i % 4][0]) and (out_w is None or bits_equal(out_w, sums[i % 4][1]))


def _torch_activation(gate_up, grad):
    x = gate_up.detach().requires_grad_()
    gate, up = x.chunk(2, dim=-1)
    h = torch.nn.functional.silu(gate) * up
    h.backward(grad)
    return h.detach(), x.grad


def _same_values(a, b):
    """Equal bit for bit, or both NaN."""
    return bool(((a.view(torch.int16) == b.view(torch.int16)) | (a.isnan() & b.isnan())).all())


@pytest.mark.parametrize("rows,inter", [(1, 8), (33, 264), (4, 1536), (2400, 520)])
def test_expert_activation(rows, inter):
    """silu(gate) * up and its gradient are those of the separate bf16 operations, bit for bit."""
    from deepep_b200.models.moe_layer import _activate

    gen = torch.Generator().manual_seed(rows + inter)
    gu = (3 * torch.randn((rows, 2 * inter), generator=gen)).bfloat16().cuda()
    dh = torch.randn((rows, inter), generator=gen).bfloat16().cuda()
    x = gu.clone().requires_grad_()
    h = _activate(x)
    h.backward(dh)
    want, grad = _torch_activation(gu, dh)
    assert _same_values(h.detach(), want) and _same_values(x.grad, grad)


def test_expert_activation_of_every_gate_value():
    """All 65536 bf16 gates (subnormals, infinities and NaN included) against ups and gradients of every size, special ones too."""
    from deepep_b200.models.moe_layer import _activate

    gen = torch.Generator().manual_seed(5)
    gate = torch.arange(-32768, 32768, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    cols = 256
    anything = lambda: torch.randint(-32768, 32768, (65536, cols), generator=gen, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    usual = lambda: torch.randn((65536, cols), generator=gen).bfloat16()
    for up, dh in ((usual(), usual()), (anything(), usual()), (anything(), anything())):
        gu = torch.cat([gate.unsqueeze(1).expand(-1, cols), up], dim=1).contiguous().cuda()
        x = gu.clone().requires_grad_()
        h = _activate(x)
        h.backward(dh.cuda())
        want, grad = _torch_activation(gu, dh.cuda())
        assert _same_values(h.detach(), want) and _same_values(x.grad, grad)


def test_expert_activation_under_autograd_modes():
    """Second derivatives, forward mode, batched gradients, vmap and tracing see the separate operations."""
    from torch.autograd import forward_ad
    from torch.fx.experimental.proxy_tensor import make_fx

    from deepep_b200.models.moe_layer import _activate, _separate_operations

    gen = torch.Generator().manual_seed(9)
    gu, dh, v = (torch.randn(s, generator=gen).bfloat16().cuda() for s in ((17, 48), (17, 24), (17, 48)))
    results = {}
    for fn in (_activate, _separate_operations):
        x, g = gu.clone().requires_grad_(), dh.clone().requires_grad_()
        first, = torch.autograd.grad(fn(x), x, g, create_graph=True)
        second = torch.autograd.grad(first, (x, g), v)
        with forward_ad.dual_level():
            tangent = forward_ad.unpack_dual(fn(forward_ad.make_dual(gu, v))).tangent.clone()
        batched, = torch.autograd.grad(fn(x), x, torch.stack([dh, 2 * dh, -dh]), is_grads_batched=True)
        mapped = torch.func.vmap(fn)(torch.stack([gu, v]))
        results[fn] = [first.detach(), *second, tangent, batched, mapped]
    for a, b in zip(*results.values()):
        assert _same_values(a, b)
    assert _same_values(torch.compile(_activate, backend="eager", fullgraph=True)(gu), _activate(gu))
    traced = make_fx(_activate)(gu)
    assert any("silu" in str(n.target) for n in traced.graph.nodes) and _same_values(traced(v), _activate(v))


@pytest.mark.parametrize("rows,width", [(1, 8), (33, 1032), (1500, 4096), (7, 264)])
def test_weighted_rows(rows, width):
    """The product of rows with their weights and both gradients, against the separate operations bit for bit (values of every
    size, infinities and NaN included), and their second derivatives."""
    from deepep_b200.models.moe_layer import _weigh

    gen = torch.Generator().manual_seed(rows)
    anything = torch.randint(-32768, 32768, (rows, width), generator=gen, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    usual, dh = (torch.randn((rows, width), generator=gen).bfloat16() for _ in range(2))
    w = torch.rand((rows,), generator=gen)
    w[0] = float("inf") if rows > 1 else 1.5
    for src, need in ((usual, (True, True)), (anything, (True, True)), (usual, (True, False)), (usual, (False, True))):
        results = []
        for fn in (lambda r, f: _weigh(r, f, torch.bfloat16), lambda r, f: r * f.unsqueeze(1).to(torch.bfloat16)):
            r, f = src.cuda().requires_grad_(need[0]), w.cuda().requires_grad_(need[1])
            out, wanted = fn(r, f), [t for t in (r, f) if t.requires_grad]
            grads = torch.autograd.grad(out, wanted, dh.cuda(), retain_graph=True)
            again = torch.autograd.grad(out, wanted, dh.cuda(), create_graph=True)
            results.append([out.detach(), *grads, *[t.detach() for t in again]])
        for a, b in zip(*results):
            if a.dtype == torch.float32:               # the weights' gradients are bf16 sums handed back as fp32
                assert bool(((a == b) | (a.isnan() & b.isnan())).all())
            else:
                assert _same_values(a, b)


@pytest.mark.parametrize("tokens,hidden,experts,topk", [(1, 8, 2, 1), (33, 264, 9, 3), (130, 2056, 40, 7), (64, 4096, 64, 6),
                                                        (17, 8192, 32, 16), (300, 1024, 8, 1)])
def test_weighed_combine(filled_outputs, tokens, hidden, experts, topk):
    """Sums and row gradients as from the separate kernels bit for bit.  The weights' gradients are sums of the same bf16 terms in
    another order, rounded to bf16: fp32 sums of n terms differ by at most 2 n 2^-24 of the sum of their magnitudes, and the rounding
    adds half a step of 2^-8 on either side."""
    from deepep_b200 import ElasticBuffer
    from deepep_b200.models import moe_layer as M

    dev = torch.device("cuda")
    g = torch.Generator().manual_seed(tokens)
    idx, w = make_routes("empty" if tokens > 1 else "random", tokens, experts, topk, 1, 3).to(dev), make_weights(tokens, topk, 4).to(dev)
    buf = ElasticBuffer(None, num_max_tokens_per_rank=max(tokens, 300), hidden=hidden, num_topk=topk, explicitly_destroy=True)
    x = torch.zeros((tokens, hidden), dtype=torch.bfloat16, device=dev)
    _, _, recv_w, handle, _ = buf.dispatch(x, topk_idx=idx, topk_weights=w, num_experts=experts, do_expand=True)
    rows = torch.randn((handle._plan.num_rows, hidden), generator=g).bfloat16().to(dev)
    grad = torch.randn((tokens, hidden), generator=g).bfloat16().to(dev)

    def fused(a, b):
        out = M._weigh_and_combine(buf, a, b, handle, torch.bfloat16)
        assert type(out.grad_fn).__name__ == "_WeighAndCombineBackward"
        return out

    def separate(a, b):
        return M._Combine.apply(buf, M._weigh(a, b, torch.bfloat16), handle)

    for which in ((True, True), (True, False), (False, True)):
        for again in (False, True):
            got = []
            for f in (fused, separate):
                a, b = rows.clone().requires_grad_(which[0]), recv_w.clone().requires_grad_(which[1])
                out = f(a, b)
                got.append((out, *torch.autograd.grad(out, [t for t in (a, b) if t.requires_grad], grad, create_graph=again)))
            for name, p, q in zip(["out"] + [n for n, need in zip(("rows", "weights"), which) if need], *got):
                if name == "weights":
                    token = handle._plan.recv_row_src[:rows.shape[0]].long() // topk
                    size = (rows.float() * grad.float()[token]).abs().sum(1)
                    assert bool(((p - q).abs() <= q.abs() * 2.0 ** -8 + size * hidden * 2.0 ** -23).all())
                else:
                    assert bits_equal(p, q), (name, which, again)
    buf.destroy()


@pytest.fixture
def filled_outputs(monkeypatch):
    """Whatever the engine allocates holds 0x55 in every byte before a kernel sees it."""
    empty = torch.empty

    def filled(*args, **kwargs):
        t = empty(*args, **kwargs)
        if t.is_cuda:
            t.view(torch.uint8).fill_(0x55)
            torch.cuda.synchronize()              # the kernels may run on another stream
        return t

    monkeypatch.setattr(torch, "empty", filled)


def _untouched(t):
    return bool((t.view(torch.uint8) == 0x55).all())


@pytest.mark.parametrize("payload", ["bf16", "fp8", "fp8_fused"])
@pytest.mark.parametrize("alignment,experts", [(128, 24), (16, 700)])
def test_padding_rows_are_zero(filled_outputs, payload, alignment, experts):
    """Rows that no token fills, and their scales, are zero whatever the memory held, rows of tokens are not touched, fresh and
    cached, with the exact and with the worst-case row count."""
    from deepep_b200 import ElasticBuffer
    from deepep_b200.utils.math import per_token_cast_to_fp8

    dev, T, H, K = torch.device("cuda"), 300, 896, 5
    x = torch.randn((T, H), generator=torch.Generator().manual_seed(4)).bfloat16()
    idx, w = make_routes("invalid", T, experts, K, 1, 6), make_weights(T, K, 2)
    src = per_token_cast_to_fp8(x) if payload == "fp8" else x
    ref, lays = R.dispatch([src], [idx], [w], experts, do_expand=True, expert_alignment=alignment, quantize_fp8=payload == "fp8_fused")
    want = ref[0][0] if isinstance(ref[0][0], tuple) else (ref[0][0],)
    used = torch.zeros((lays[0].num_rows,), dtype=torch.bool)
    used[lays[0].row_index] = True
    buf = ElasticBuffer(None, num_max_tokens_per_rank=T, hidden=H, num_topk=K, use_fp8_dispatch=payload == "fp8_fused",
                        explicitly_destroy=True)
    on_gpu = tuple(t.to(dev) for t in src) if payload == "fp8" else src.to(dev)
    handle = None
    for exact in (True, True, False):
        fresh = dict(topk_idx=idx.to(dev), topk_weights=w.to(dev), num_experts=experts, expert_alignment=alignment, do_expand=True,
                     do_cpu_sync=exact)
        got, _, _, h, _ = buf.dispatch(on_gpu, **(fresh if handle is None or not exact else dict(handle=handle)))
        handle = handle or h
        got = got if isinstance(got, tuple) else (got,)
        for g, e in zip(got, want):
            rows = e.shape[0]
            assert bits_equal(g[:rows][used.to(dev)], e[used]), "a token's row differs"
            assert not bool(g.view(torch.uint8)[:rows][~used.to(dev)].any()) and not bool(g.view(torch.uint8)[rows:].any())
    buf.destroy()


@pytest.mark.parametrize("hidden,expand,alignment", [(7168, True, 1), (7168, True, 128), (4096, False, 1), (64, True, 16)])
def test_device_profile_counts_every_row_once(hidden, expand, alignment):
    """On one rank, however many pieces and spans a row is cut into: the dispatch's records add up to the rows written, those of
    the combine to the rows read."""
    from deepep_b200.parallel.virtual import VirtualWorld

    T, E, K = 333, 16, 4
    x = torch.randn((T, hidden), generator=torch.Generator().manual_seed(1)).bfloat16()
    idx, w = make_routes("invalid", T, E, K, 1, 2), make_weights(T, K, 3)
    _, lays = R.dispatch([x], [idx], [w], E, do_expand=expand, expert_alignment=alignment)
    with VirtualWorld(1, T, hidden, K, timeout=10.0) as vw:
        eng = vw.engine
        plans = eng.notify([idx.cuda()], [w.cuda()], E, expand=expand, alignment=alignment)
        eng.enable_device_profile(True)
        (rows, _), = eng.dispatch([x.cuda()], plans, 0)
        eng.combine([rows], plans, [None])
        prof = eng.pop_device_profile()
        eng.check_status()
    for op in ("dispatch", "combine"):
        assert sum(b["rows"] for b in prof[op, 0]) == lays[0].row_index.numel(), op


def test_counts_of_an_awaited_call_and_tables_made_on_demand():
    """The host reads the counts of the call it waits for, also behind calls that it does not wait for, whose counts differ; the
    tables of a handle appear when asked for, and changing one in place through its view is noticed."""
    from deepep_b200 import ElasticBuffer

    dev, T, E, K = torch.device("cuda"), 200, 24, 3
    x = torch.randn((T, 256), generator=torch.Generator().manual_seed(1)).bfloat16().to(dev)
    buf = ElasticBuffer(None, num_max_tokens_per_rank=256, hidden=256, num_topk=K, explicitly_destroy=True)
    for low_latency in (False, True):
        for seed in range(12):
            idx = make_routes("empty", T, E, K, 1, seed).to(dev)
            args = dict(topk_weights=make_weights(T, K, seed).to(dev), num_experts=E, do_expand=not low_latency)
            if seed % 3:
                buf.dispatch(x, topk_idx=make_routes("random", T, E, K, 1, 100 + seed).to(dev), do_cpu_sync=False, **args)
            handle = buf.dispatch(x, topk_idx=idx, **args)[3]
            assert handle.is_low_latency == low_latency
            assert handle.num_recv_tokens_per_expert_list == torch.bincount(idx[idx >= 0], minlength=E).tolist()
            psum = handle.psum_num_recv_tokens_per_expert
            assert psum is handle.psum_num_recv_tokens_per_expert
            assert psum.tolist() == torch.tensor(handle.num_recv_tokens_per_expert_list).cumsum(0).tolist()
        rows = torch.zeros((handle.num_expanded_tokens, 256), dtype=torch.bfloat16, device=dev)
        buf.combine(rows, handle)
        handle.recv_src_metadata.add_(1)
        with pytest.raises(RuntimeError, match="modified in place"):
            buf.combine(rows, handle)
    buf.destroy()


@pytest.mark.parametrize("counts,k,n", [
    ([1], 64, 64),                                   # one row, one step, a quarter of a tile
    ([128, 0, 129, 256, 257, 0, 127], 192, 320),     # both sides of a half tile and of a tile, empty experts, a short last tile
    ([0, 0, 0], 128, 64),
    ([3] * 300 + [700], 64, 576),                    # more experts than one scan step, many tiles per block
])
def test_grouped_gemm_on_one_rank(counts, k, n):
    """Both operators on a single rank against float32 (bf16 results: 2^-8 relative, sums of k products: 1e-5 of their size), with
    the gathered rows handed out; an output that overlaps x takes the general kernels and gives the same bits."""
    from deepep_b200.ops import ep_gmm_fused as G
    from deepep_b200.ops import load_native

    C, dev, rows, E = load_native(), torch.device("cuda"), sum(counts), len(counts)
    layout = C.make_mega_layout(1, 1, 128, 1, G.GmmEngine.region_bytes(C, max(rows, 1), max(k, n), max(k, n)))
    s = C.Session(0, 1, layout.total, 20.0)
    s.attach_peers([s.workspace])
    try:
        eng = G.GmmEngine([s], layout, dev, max(rows, 1), max(k, n), max(k, n))
        gen = torch.Generator().manual_seed(rows + k)
        x = torch.randn((rows, k), generator=gen).bfloat16()
        w = torch.randn((E, k, n), generator=gen).bfloat16()
        want, size, at = torch.zeros((rows, n)), torch.zeros((rows, n)), 0
        for e, c in enumerate(counts):
            want[at:at + c] = x[at:at + c].float() @ w[e].float()
            size[at:at + c] = x[at:at + c].float().abs() @ w[e].float().abs()
            at += c
        dx, dw, dc = x.to(dev), w.to(dev), torch.tensor(counts, dtype=torch.int32, device=dev)
        gathered, outs = torch.full_like(dx, 7.0), []
        for _ in range(2):
            out, back = (torch.full((rows, n), 5.0, dtype=torch.bfloat16, device=dev) for _ in range(2))
            eng.a2av_gmm([dx], [dw], [dc], [out], [gathered], num_experts=E)
            eng.gmm_a2av([dx], [dw], [dc], [back], num_experts=E)
            outs += [out, back]
        out = torch.full((rows, n), 5.0, dtype=torch.bfloat16, device=dev)
        assert bits_equal(eng.a2av_gmm([dx], [dw], [dc], [out], num_experts=E)[0], x)      # the gathered rows, without a buffer
        outs.append(out)
        assert eng.scratch[0]["gathered"] is None
        memory = torch.zeros((rows * max(k, n),), dtype=torch.bfloat16, device=dev)       # x and the output start at one address
        shared_x, shared_out = memory[:rows * k].view(rows, k), memory[:rows * n].view(rows, n)
        for op in (eng.a2av_gmm, eng.gmm_a2av):
            shared_x.copy_(dx)
            used = op([shared_x], [dw], [dc], [shared_out], num_experts=E)
            assert used is None or bits_equal(used[0], x)
            outs.append(shared_out.clone())
        eng.check()
        assert bits_equal(gathered, x)
        assert torch.all((outs[0].cpu().float() - want).abs() <= want.abs() * 2 ** -8 + 1e-5 * size)
        for other in outs[1:]:
            assert torch.equal(other, outs[0])
        if rows:                                         # more rows than x holds: reported, and nothing is written
            out = torch.full((rows, n), 5.0, dtype=torch.bfloat16, device=dev)
            eng.gmm_a2av([dx], [dw], [dc + rows], [out], num_experts=E)
            with pytest.raises(RuntimeError, match="row counts"):
                eng.check()
            assert bool((out == 5.0).all())
    finally:
        torch.cuda.synchronize()
        s.close()


@pytest.mark.parametrize("alignment", [1, 16])
def test_high_throughput_calls_after_an_abort_touch_nothing(filled_outputs, alignment):
    """Once a wait of the rank ran out, calls queued behind it neither read the plan nor write their outputs."""
    from deepep_b200.parallel.virtual import VirtualWorld

    dev, T, H, E, K = torch.device("cuda"), 70, 256, 8, 3
    x = torch.randn((T, H), generator=torch.Generator().manual_seed(4)).bfloat16().to(dev)
    idx, w = make_routes("invalid", T, E, K, 1, 6).to(dev), make_weights(T, K, 2).to(dev)
    with VirtualWorld(1, T, H, K, timeout=0.05) as vw:
        eng = vw.engine
        eng.local_direct = False                           # through the staging area and the partials, as with peers
        plans = eng.notify([idx], [w], E, alignment=alignment)
        (rows, _), = eng.dispatch([x], plans, 0)
        vw.sessions[0].wait_probe(torch.cuda.current_stream().cuda_stream)
        (later, _), = eng.dispatch([x], plans, 0)
        (out, out_w), = eng.combine([rows], plans, [plans[0].recv_w[:plans[0].num_rows].contiguous()])
        torch.cuda.synchronize()
        assert vw.sessions[0].status()["where"] == 99
        assert not _untouched(rows) and _untouched(later) and _untouched(out) and _untouched(out_w)


def test_routing_pass_that_gives_up_leaves_an_empty_plan(filled_outputs):
    """One of two ranks runs alone: its wait for the peer's table runs out, the plan says 'no rows', and the calls queued behind
    it without a look at the host touch nothing."""
    from deepep_b200.ops import load_native
    from deepep_b200.parallel.engine_cuda import CudaEngine

    C, dev, T, H, E, K = load_native(), torch.device("cuda", torch.cuda.current_device()), 300, 256, 8, 3
    layout = C.make_layout(2, T, H, K)
    ranks = [C.Session(r, 2, layout.total, 0.05) for r in range(2)]
    try:
        for s in ranks:
            s.attach_peers([r.workspace for r in ranks])
        eng = CudaEngine(ranks[:1], layout, dev)
        x = torch.randn((T, H), generator=torch.Generator().manual_seed(4)).bfloat16().to(dev)
        idx, w = make_routes("invalid", T, E, K, 2, 6).to(dev), make_weights(T, K, 2).to(dev)
        plans = eng.notify([idx], [w], E, alignment=16, cpu_sync=False)
        (rows, _), = eng.dispatch([x], plans, 0)
        (out, _), = eng.combine([rows], plans, [None])
        torch.cuda.synchronize()
        st = ranks[0].status()
        assert st["code"] == 1 and st["op"] == 1 and st["where"] == 1 and st["peer"] == 1
        plan = plans[0]
        assert not bool(plan.rank_rows.any()) and not bool(plan.expert_counts.any()) and not bool(plan.expert_offsets.any())
        assert _untouched(rows) and _untouched(out) and all(r.guard_intact() for r in ranks)
    finally:
        torch.cuda.synchronize()
        for s in ranks:
            s.close()
