"""Low-latency dispatch/combine kernels: virtual ranks on one GPU against the oracle, and CUDA-graph replay."""
import pytest
import torch

from deepep_b200.oracle import reference as R
from deepep_b200.utils.math import per_token_cast_to_fp8
from helpers import bits_equal, make_routes, make_weights

pytestmark = pytest.mark.gpu


def _case(world, tokens, H, E, K, mode, routes="random", repeats=2):
    from deepep_b200.parallel.virtual import VirtualWorld
    from deepep_b200.ops import load_native

    C = load_native()
    dev = torch.device("cuda")
    M = max(max(tokens), 1)
    with VirtualWorld(world, M, H, K, timeout=10.0, ll_bytes=C.ll_region_bytes(world, M, K, H)) as vw:
        eng = vw.engine
        for rep in range(repeats):
            xs = [torch.randn((t, H), generator=torch.Generator().manual_seed(rep * 100 + r)).bfloat16() for r, t in enumerate(tokens)]
            idx = [make_routes(routes, t, E, K, world, rep * 10 + r) for r, t in enumerate(tokens)]
            ws = [make_weights(t, K, rep + r) for r, t in enumerate(tokens)]
            if mode == 1:
                q = [per_token_cast_to_fp8(x) for x in xs]
                dx, rx_in = [(a.to(dev), b.to(dev)) for a, b in q], q
            else:
                dx, rx_in = [x.to(dev) for x in xs], xs
            res = eng.ll_dispatch(dx, [i.to(dev) for i in idx], [w.to(dev) for w in ws], E, mode)
            ref, lays = R.dispatch(rx_in, idx, ws, E, do_expand=True, quantize_fp8=(mode == 2))
            for r in range(world):
                plan, rx, rsf = res[r]
                assert plan.num_rows == lays[r].num_rows
                assert plan.expert_counts_list == lays[r].expert_counts.tolist()
                if mode == 0:
                    assert bits_equal(rx, ref[r][0])
                else:
                    assert bits_equal(rx, ref[r][0][0]) and bits_equal(rsf, ref[r][0][1])
                assert torch.equal(plan.recv_w[:plan.num_rows].cpu(), ref[r][2])
            eouts = [torch.randn((lays[r].num_rows, H), generator=torch.Generator().manual_seed(7 + r)).bfloat16() for r in range(world)]
            outs = eng.ll_combine([e.to(dev) for e in eouts], [res[r][0] for r in range(world)])
            cref = R.low_latency_combine(eouts, lays, ws, tokens)
            torch.cuda.synchronize()
            eng.check_status()
            for r in range(world):
                assert bits_equal(outs[r], cref[r]), f"rank {r} combined output differs"


@pytest.mark.parametrize("world", [1, 2, 4, 8])
def test_ll_bf16(world):
    _case(world, [100 + 7 * r for r in range(world)], 1024, 16 * world, 4, 0, repeats=3)


def test_ll_invalid_and_empty():
    _case(4, [128, 0, 5, 256], 512, 32, 8, 0, routes="empty")


def test_ll_fp8():
    _case(2, [128, 77], 2048, 32, 8, 1)
    _case(2, [128, 77], 2048, 32, 8, 2)


def test_ll_decode_shape():
    _case(8, [128] * 8, 7168, 384, 8, 2, repeats=1)


def test_ll_graph_replay_public_api():
    """dispatch + combine through ElasticBuffer inside one captured CUDA graph, replayed with new inputs."""
    from deepep_b200 import ElasticBuffer

    dev = torch.device("cuda")
    T, H, E, K = 64, 1024, 16, 4
    buf = ElasticBuffer(None, num_max_tokens_per_rank=128, hidden=H, num_topk=K, explicitly_destroy=True)
    x = torch.zeros((T, H), dtype=torch.bfloat16, device=dev)
    idx = torch.zeros((T, K), dtype=torch.int64, device=dev)
    w = torch.zeros((T, K), dtype=torch.float32, device=dev)

    def fill(seed):
        x.copy_(torch.randn((T, H), generator=torch.Generator().manual_seed(seed)).bfloat16())
        idx.copy_(make_routes("random", T, E, K, 1, seed))
        w.copy_(make_weights(T, K, seed))

    def step():
        rx, _, rw, handle, _ = buf.dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E, do_cpu_sync=False)
        assert handle.is_low_latency
        out, _, _ = buf.combine(rx, handle)
        return out

    fill(0)
    for _ in range(2):
        step()           # warm up outside the graph
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    for seed in (1, 2, 3):
        fill(seed)
        graph.replay()
        torch.cuda.synchronize()
        ok = make_routes("random", T, E, K, 1, seed) >= 0
        expect = x.float().cpu() * (make_weights(T, K, seed) * ok).sum(1, keepdim=True)
        assert torch.allclose(out.float().cpu(), expect, rtol=0.02, atol=0.05)
    buf.destroy()


def test_ll_empty_batch_takes_the_same_path():
    """The path is chosen from the buffer and the options, never from a rank's own token count: an empty batch on a
    decode buffer runs the low-latency kernels too (with peers, a rank that chose differently would never be answered)."""
    from deepep_b200 import ElasticBuffer

    dev = torch.device("cuda")
    H, E, K = 512, 16, 4
    buf = ElasticBuffer(None, num_max_tokens_per_rank=64, hidden=H, num_topk=K, explicitly_destroy=True)
    x = torch.zeros((0, H), dtype=torch.bfloat16, device=dev)
    idx = torch.zeros((0, K), dtype=torch.int64, device=dev)
    w = torch.zeros((0, K), dtype=torch.float32, device=dev)
    rx, _, rw, handle, _ = buf.dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E)
    assert handle.is_low_latency and rx.shape == (0, H) and handle.num_recv_tokens_per_expert_list == [0] * E
    out, _, _ = buf.combine(rx, handle)
    torch.cuda.synchronize()
    assert out.shape == (0, H)
    buf.destroy()


def test_ll_cached_dispatch_asynchronous():
    """A cached low-latency dispatch that the caller waits for through its event gives the rows of the original, also when memory
    is taken and given back on the current stream meanwhile."""
    from deepep_b200 import ElasticBuffer

    dev = torch.device("cuda")
    T, H, E, K = 96, 2048, 32, 4
    buf = ElasticBuffer(None, num_max_tokens_per_rank=128, hidden=H, num_topk=K, explicitly_destroy=True)
    x = torch.randn((T, H), generator=torch.Generator().manual_seed(3)).bfloat16().to(dev)
    idx, w = make_routes("invalid", T, E, K, 1, 4).to(dev), make_weights(T, K, 5).to(dev)
    rx, _, _, handle, _ = buf.dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E)
    assert handle.is_low_latency
    first, _, _ = buf.combine(rx, handle)
    for _ in range(4):
        again, _, _, _, event = buf.dispatch(x, handle=handle, async_with_compute_stream=True)
        fills = [torch.full((n,), -1, dtype=torch.int32, device=dev) for n in (1, E, E + 1, 128 * K, T * K, rx.shape[0])]
        with event:
            pass
        assert bits_equal(again, rx)
        out, _, done = buf.combine(again, handle, async_with_compute_stream=True)
        done.current_stream_wait()
        assert bits_equal(out, first)
        del fills
    buf.destroy()


@pytest.mark.parametrize("mode,tensors", [(0, 6), (2, 7)])
def test_ll_dispatch_allocates_its_outputs_only(mode, tensors):
    """An eager dispatch is bound by the host: rows, scales, weights, sources, counts, offsets and the row count are all the
    tensors it makes (the rows of the rank's own slots lie behind the row count)."""
    from deepep_b200.ops import load_native
    from deepep_b200.parallel.virtual import VirtualWorld

    T, H, E, K = 20, 256, 16, 4
    with VirtualWorld(1, T, H, K, timeout=10.0, ll_bytes=load_native().ll_region_bytes(1, T, K, H)) as vw:
        x = torch.randn((T, H), generator=torch.Generator().manual_seed(1)).bfloat16().cuda()
        idx, w = make_routes("random", T, E, K, 1, 2).cuda(), make_weights(T, K, 3).cuda()
        counted = lambda: torch.cuda.memory_stats()["allocation.all.allocated"]
        before = counted()
        (plan, rx, _), = vw.engine.ll_dispatch([x], [idx], [w], E, mode, cpu_sync=False)
        assert counted() - before == tensors
        torch.cuda.synchronize()
        assert int(plan.num_rows_dev[0]) == T * K and sorted(plan.num_rows_dev[1:].tolist()) == list(range(T * K))
        if mode == 0:
            assert bits_equal(rx[plan.num_rows_dev[1:].long()], x.repeat_interleave(K, 0))


def _one_rank(T, H, E, K):
    from deepep_b200.ops import load_native
    from deepep_b200.parallel.virtual import VirtualWorld

    x = torch.randn((T, H), generator=torch.Generator().manual_seed(1)).bfloat16()
    idx, w = make_routes("random", T, E, K, 1, 2), make_weights(T, K, 3)
    return VirtualWorld(1, T, H, K, timeout=0.05, ll_bytes=load_native().ll_region_bytes(1, T, K, H)), x, idx, w


def test_ll_combine_after_an_abort_touches_nothing():
    """Once a wait of the rank ran out, a queued combine neither reads the handle's tables nor writes the output; with the status
    cleared the same handle works again."""
    world, x, idx, w = _one_rank(24, 512, 16, 4)
    with world as vw:
        (plan, rx, _), = vw.engine.ll_dispatch([x.cuda()], [idx.cuda()], [w.cuda()], 16, 0)
        vw.sessions[0].wait_probe(torch.cuda.current_stream().cuda_stream)
        out = torch.full((24, 512), 7.0, dtype=torch.bfloat16, device="cuda")
        vw.engine.ll_combine([rx], [plan], outs=[out])
        torch.cuda.synchronize()
        assert vw.sessions[0].status()["where"] == 99 and bool((out == 7.0).all())
        vw.sessions[0].clear_status()
        vw.engine.ll_combine([rx], [plan], outs=[out])
        torch.cuda.synchronize()
        vw.engine.check_status()
        ref, lays = R.dispatch([x], [idx], [w], 16, do_expand=True)
        assert bits_equal(out, R.low_latency_combine([ref[0][0]], lays, [w], [24])[0])


def test_ll_combine_reports_rows_that_x_does_not_have():
    """A table that names rows behind the expert outputs is reported and the rows are not used (the memory behind is there)."""
    from deepep_b200.parallel.engine_cuda import CommunicationError

    world, x, idx, w = _one_rank(24, 512, 16, 4)
    with world as vw:
        (plan, rx, _), = vw.engine.ll_dispatch([x.cuda()], [idx.cuda()], [w.cuda()], 16, 0)
        rows = rx.shape[0]
        both = torch.cat([rx, rx])
        plan.num_rows_dev[1:] += rows
        out = torch.full((24, 512), 7.0, dtype=torch.bfloat16, device="cuda")
        vw.engine.ll_combine([both[:rows]], [plan], outs=[out])
        torch.cuda.synchronize()
        assert bool((out == 7.0).all())
        with pytest.raises(CommunicationError, match="bad argument .*rows that the expert outputs do not have"):
            vw.engine.check_status()


def test_ll_dispatch_that_gives_up_leaves_no_rows_behind():
    """One of two ranks runs alone: its wait for the peer's routing table runs out, the handle's tables say 'no rows', and a
    combine that was queued behind the dispatch without a look at the host writes nothing."""
    from deepep_b200.ops import load_native
    from deepep_b200.parallel.engine_cuda import CudaEngine

    C, T, H, E, K = load_native(), 24, 512, 16, 4
    layout = C.make_layout(2, T, H, K, C.ll_region_bytes(2, T, K, H), 0, 0)
    ranks = [C.Session(r, 2, layout.total, 0.05) for r in range(2)]
    try:
        for s in ranks:
            s.attach_peers([r.workspace for r in ranks])
        eng = CudaEngine(ranks[:1], layout, torch.device("cuda", torch.cuda.current_device()))
        x = torch.randn((T, H), generator=torch.Generator().manual_seed(1)).bfloat16().cuda()
        idx, w = make_routes("random", T, E, K, 2, 2).cuda(), make_weights(T, K, 3).cuda()
        (plan, rx, _), = eng.ll_dispatch([x], [idx], [w], E, 0, cpu_sync=False)
        out = torch.full((T, H), 7.0, dtype=torch.bfloat16, device="cuda")
        eng.ll_combine([rx], [plan], outs=[out])
        torch.cuda.synchronize()
        st = ranks[0].status()
        assert st["code"] == 1 and st["op"] == 4 and st["where"] == 1 and st["peer"] == 1
        assert int(plan.num_rows_dev[0]) == 0 and bool((plan.num_rows_dev[1:] == -1).all()) and bool((out == 7.0).all())
    finally:
        torch.cuda.synchronize()
        for s in ranks:
            s.close()


@pytest.mark.parametrize("limit", [0.002, 0.05])
def test_ll_dispatch_reports_rows_that_never_came(limit):
    """One of two ranks runs alone and finds the peer's routing table, but none of the rows that it announces: the dispatch that
    reads its counts back raises itself, whether its kernel gives up while the host still polls or later."""
    from deepep_b200.models.mega_moe import _view
    from deepep_b200.ops import load_native
    from deepep_b200.parallel.engine_cuda import CommunicationError, CudaEngine

    C, T, H, E, K, P = load_native(), 24, 512, 16, 4, 2
    region = C.ll_region_bytes(P, T, K, H)
    layout = C.make_layout(P, T, H, K, region, 0, 0)
    ranks = [C.Session(r, P, layout.total, limit) for r in range(P)]
    try:
        for s in ranks:
            s.attach_peers([r.workspace for r in ranks])
        # what the peer would have written for the first call: header, table, weights and flag, in this order and 1024-byte aligned
        sizes = dict(hdr=P * 16, idx=P * T * K * 4, w=P * T * K * 4, flag=P * 8)
        at, dev = ranks[0].workspace + layout.ll + region // 2, torch.device("cuda", torch.cuda.current_device())
        part = {}
        for name, nbytes in sizes.items():
            part[name] = _view(at, nbytes, dev)
            at += -(-nbytes // 1024) * 1024
        part["hdr"].view(torch.int32).view(P, 4)[1, 0] = 5
        part["idx"].view(torch.int32).view(P, T, K)[1, :5] = torch.arange(K, dtype=torch.int32, device=dev)
        part["w"].view(torch.float32).view(P, T, K)[1, :5] = 0.25
        part["flag"].view(torch.int64)[1] = 1
        torch.cuda.synchronize()
        eng = CudaEngine(ranks[:1], layout, dev)
        x = torch.randn((T, H), generator=torch.Generator().manual_seed(1)).bfloat16().cuda()
        idx, w = make_routes("random", T, E, K, P, 2).cuda(), make_weights(T, K, 3).cuda()
        with pytest.raises(CommunicationError, match=r"ll_dispatch timeout at wait site 2 \(a part of a row from a source rank\) on peer 1"):
            eng.ll_dispatch([x], [idx], [w], E, 0)
    finally:
        torch.cuda.synchronize()
        for s in ranks:
            s.close()
