"""alltoallv_gmm / gmm_alltoallv kernels (virtual ranks in one cooperative launch) against a plain fp32 restatement."""
import pytest
import torch

from deepep_b200.ops import ep_gmm_fused as G

pytestmark = pytest.mark.gpu


def _counts(world, E, max_rows, seed, empty_expert=None):
    g = torch.Generator().manual_seed(seed)
    out = []
    for s in range(world):
        c = torch.randint(0, 2 * max_rows // E + 1, (E,), generator=g)
        if empty_expert is not None:
            c[empty_expert] = 0
        while int(c.sum()) > max_rows:
            c = c // 2
        out.append(c.tolist())
    return out


def _close(actual, expected, what):
    a, e = actual.float().cpu(), expected.float()
    assert a.shape == e.shape, (what, a.shape, e.shape)
    if a.numel() == 0:
        return
    err = (a - e).abs().max().item()
    scale = e.abs().max().item() + 1e-6
    assert err <= 2e-2 * scale, f"{what}: max abs error {err} against magnitude {scale}"


def _world(world, E, K, N, max_rows, seed=0, empty_expert=None, reps=2, zero_copy=False):
    from deepep_b200.ops import load_native

    C = load_native()
    dev = torch.device("cuda")
    L = E // world
    counts = _counts(world, E, max_rows, seed, empty_expert)
    gen = torch.Generator().manual_seed(seed + 1)
    xs = [torch.randn((sum(c), K), generator=gen).to(torch.bfloat16) for c in counts]
    ws = [(torch.randn((L, K, N), generator=gen) / K ** 0.5).to(torch.bfloat16) for _ in range(world)]
    ref_out, ref_gathered = G.reference_alltoallv_gmm(xs, ws, counts, E)
    # second op: the expert ranks multiply what they gathered by a second weight and send it back
    ws2 = [(torch.randn((L, K, N), generator=gen) / K ** 0.5).to(torch.bfloat16) for _ in range(world)]
    ref_back = G.reference_gmm_alltoallv(ref_gathered, ws2, counts, E)

    layout = C.make_mega_layout(world, 1, 128, 1, G.GmmEngine.region_bytes(C, max_rows, K, N))
    sessions = [C.Session(r, world, layout.total, 20.0) for r in range(world)]
    for s in sessions:
        s.attach_peers([q.workspace for q in sessions])
    try:
        eng = G.GmmEngine(sessions, layout, dev, max_rows, K, N)
        d_x = [x.to(dev) for x in xs]
        if zero_copy:    # inputs written into the stage area are read by the peers in place
            d_x = [eng.symmetric_input(r, x.shape[0], K) for r, x in enumerate(xs)]
            for v, x in zip(d_x, xs):
                v.copy_(x)
        d_w, d_w2 = [w.to(dev) for w in ws], [w.to(dev) for w in ws2]
        d_c = [torch.tensor(c, dtype=torch.int32, device=dev) for c in counts]
        for rep in range(reps):
            outs = [torch.full((r.shape[0], N), float("nan"), dtype=torch.bfloat16, device=dev) for r in ref_out]
            gath = [torch.full((r.shape[0], K), float("nan"), dtype=torch.bfloat16, device=dev) for r in ref_gathered]
            eng.a2av_gmm(d_x, d_w, d_c, outs, gath, num_experts=E)
            back = [torch.full((x.shape[0], N), float("nan"), dtype=torch.bfloat16, device=dev) for x in xs]
            if zero_copy:
                back = [eng.symmetric_output(r, x.shape[0], N) for r, x in enumerate(xs)]
            eng.gmm_a2av(gath, d_w2, d_c, back, num_experts=E)
            torch.cuda.synchronize()
            eng.check()
            for s in sessions:
                assert s.status()["code"] == 0, s.status()
            for r in range(world):
                assert torch.equal(gath[r].cpu(), ref_gathered[r]), f"rank {r}: gathered rows differ (rep {rep})"
                _close(outs[r], ref_out[r], f"a2av_gmm rank {r} rep {rep}")
                _close(back[r], ref_back[r], f"gmm_a2av rank {r} rep {rep}")
    finally:
        torch.cuda.synchronize()
        for s in sessions:
            s.close()


def test_single_rank_grouped_gemm():
    _world(1, 4, 256, 256, 600)


@pytest.mark.parametrize("counts, K, N", [
    ([1], 64, 64), ([1, 383], 128, 192), ([256, 257, 0, 128, 511, 512, 513, 129], 320, 320), ([4097, 3], 576, 448),
    ([700], 1024, 7168), ([0, 2000, 1, 130, 0, 260], 192, 7168), ([256, 257, 0, 128, 511, 512, 513, 129], 320, 1984), ([300], 640, 1024)])
def test_tile_edges_on_a_single_rank(counts, K, N):
    """Edges of the 256-row tiles (one half, both, a row more), empty experts, column blocks past the last one, K loops shorter
    and longer than the pipeline, fewer tiles than blocks (narrow tiles) and many more."""
    from deepep_b200.ops import load_native

    C, dev, E, rows = load_native(), torch.device("cuda"), len(counts), sum(counts)
    gen = torch.Generator().manual_seed(rows + K)
    x = torch.randn((rows, K), generator=gen).to(torch.bfloat16)
    w = (torch.randn((E, K, N), generator=gen) / K ** 0.5).to(torch.bfloat16)
    ref = torch.cat([a.float() @ b.float() for a, b in zip(x.split(counts), w)])
    layout = C.make_mega_layout(1, 1, 128, 1, G.GmmEngine.region_bytes(C, rows, K, N))
    session = C.Session(0, 1, layout.total, 20.0)
    session.attach_peers([session.workspace])
    try:
        eng = G.GmmEngine([session], layout, dev, rows, K, N)
        c = torch.tensor(counts, dtype=torch.int32, device=dev)
        d_x, d_w = x.to(dev), w.to(dev)
        for out_rows in (rows, rows + 3):
            out = torch.full((out_rows, N), float("nan"), dtype=torch.bfloat16, device=dev)
            gathered = torch.full((rows, K), float("nan"), dtype=torch.bfloat16, device=dev)
            eng.a2av_gmm([d_x], [d_w], [c], [out], [gathered], num_experts=E)
            back = torch.full((rows, N), float("nan"), dtype=torch.bfloat16, device=dev)
            eng.gmm_a2av([d_x], [d_w], [c], [back], num_experts=E)
            torch.cuda.synchronize()
            eng.check()
            assert torch.equal(gathered.cpu(), x)
            # one rounding to bf16 (2^-9 of the value) behind fp32 sums of K products
            assert torch.allclose(out[:rows].float().cpu(), ref, rtol=2.0 ** -8, atol=1e-4) and bool(out[rows:].isnan().all())
            assert torch.equal(out[:rows], back)
    finally:
        torch.cuda.synchronize()
        session.close()


@pytest.mark.parametrize("world", [1, 2])
def test_counts_of_either_integer_type(world):
    """Counts in 64 bits are read where they lie and give the bits of counts in 32 bits; negative ones count as none, and a count
    beyond any buffer is reported."""
    from deepep_b200.ops import load_native

    C, dev, E, K, N = load_native(), torch.device("cuda"), 6, 128, 192
    counts = _counts(world, E, 400, 9)
    xs = [torch.randn((sum(c), K), generator=torch.Generator().manual_seed(r)).bfloat16().to(dev) for r, c in enumerate(counts)]
    ws = [torch.randn((E // world, K, N), generator=torch.Generator().manual_seed(7 + r)).bfloat16().to(dev) for r in range(world)]
    received = [sum(c[e] for c in counts for e in range(r * E // world, (r + 1) * E // world)) for r in range(world)]
    layout = C.make_mega_layout(world, 1, 128, 1, G.GmmEngine.region_bytes(C, 800, K, N))
    sessions = [C.Session(r, world, layout.total, 20.0) for r in range(world)]
    for s in sessions:
        s.attach_peers([q.workspace for q in sessions])
    try:
        eng, results = G.GmmEngine(sessions, layout, dev, 800, K, N), []
        for dtype in (torch.int32, torch.int64):
            c = [torch.tensor(v, dtype=dtype, device=dev) for v in counts]
            outs = [torch.zeros((r, N), dtype=torch.bfloat16, device=dev) for r in received]
            gathered = [torch.zeros((r, K), dtype=torch.bfloat16, device=dev) for r in received]
            eng.a2av_gmm(xs, ws, c, outs, gathered, num_experts=E)
            back = [torch.zeros((x.shape[0], N), dtype=torch.bfloat16, device=dev) for x in xs]
            eng.gmm_a2av(gathered, ws, c, back, num_experts=E)
            torch.cuda.synchronize()
            eng.check()
            results.append(outs + gathered + back)
        assert all(torch.equal(a, b) for a, b in zip(*results)) and all(bool(t.any()) for t in results[0] if t.numel())
        if world == 1:
            few = torch.tensor([3, -5, 0, 0, 0, -(1 << 40)], device=dev)
            out = torch.zeros((3, N), dtype=torch.bfloat16, device=dev)
            eng.a2av_gmm([xs[0][:3].contiguous()], ws, [few], [out], num_experts=E)
            eng.check()
            # one rounding to bf16 behind an fp32 sum of 128 products of size one
            assert torch.allclose(out.float(), xs[0][:3].float() @ ws[0][0].float(), rtol=2.0 ** -8, atol=1e-3)
            eng.a2av_gmm(xs, ws, [torch.tensor([1 << 40] * E, device=dev)], [torch.empty((received[0], N), dtype=torch.bfloat16, device=dev)],
                         num_experts=E)
            with pytest.raises(RuntimeError, match="row counts"):
                eng.check()
    finally:
        torch.cuda.synchronize()
        for s in sessions:
            s.close()


@pytest.mark.parametrize("op", ["a2av_gmm", "gmm_a2av"])
@pytest.mark.parametrize("dtype,most", [(torch.int32, 2 ** 31 - 1), (torch.int64, 1 << 40)])
@pytest.mark.parametrize("oversized", [(0, 3), (2, 3), (0, 5), (4, 5), tuple(range(6))])
def test_counts_whose_sum_fits_no_int_are_reported_by_every_owner(op, dtype, most, oversized):
    """Two ranks of three experts each, both of which name more rows than an int holds: the owners of those experts, and of any
    behind the first of them, report it (a sum that wrapped round would look like one that fits)."""
    from deepep_b200.ops import load_native

    C, dev, world, E, K, N = load_native(), torch.device("cuda"), 2, 6, 64, 64
    layout = C.make_mega_layout(world, 1, 128, 1, G.GmmEngine.region_bytes(C, 64, K, N))
    sessions = [C.Session(r, world, layout.total, 20.0) for r in range(world)]
    for s in sessions:
        s.attach_peers([q.workspace for q in sessions])
    try:
        eng = G.GmmEngine(sessions, layout, dev, 64, K, N)
        counts = [most if e in oversized else 2 for e in range(E)]
        rows = [torch.ones((16, K), dtype=torch.bfloat16, device=dev) for _ in range(world)]
        weights = [torch.ones((E // world, K, N), dtype=torch.bfloat16, device=dev) for _ in range(world)]
        outs = [torch.zeros((16, N), dtype=torch.bfloat16, device=dev) for _ in range(world)]
        getattr(eng, op)(rows, weights, [torch.tensor(counts, dtype=dtype, device=dev) for _ in range(world)], outs, num_experts=E)
        torch.cuda.synchronize()
        codes = [int(sc["err"].item()) for sc in eng.scratch]
        first = min(oversized)
        assert codes == [2 if first < 3 else 0, 2] and all(s.status()["code"] == 0 for s in sessions)
        if first >= 3:                      # the first rank's experts are served as ever: two rows from, or back to, either rank
            done, rows = (outs[:1], 12) if op == "a2av_gmm" else (outs, 6)
            assert all(bool((out[:rows] == K).all()) for out in done)
    finally:
        torch.cuda.synchronize()
        for s in sessions:
            s.close()


def test_both_tile_widths_give_the_same_rows():
    """Nine narrow tiles (one and two halves high): on nine blocks all at once, on eight and six the short ones of the last row block
    are second tiles, behind 13 K steps in a pipeline of four; on five and two blocks the wide ones take their place."""
    from deepep_b200.ops import load_native

    C, dev, counts, K, N = load_native(), torch.device("cuda"), [200, 0, 256, 100], 832, 384
    rows, gen = sum(counts), torch.Generator().manual_seed(4)
    x = torch.randn((rows, K), generator=gen).to(torch.bfloat16)
    w = (torch.randn((4, K, N), generator=gen) / K ** 0.5).to(torch.bfloat16)
    ref = torch.cat([a.float() @ b.float() for a, b in zip(x.split(counts), w)])
    layout = C.make_mega_layout(1, 1, 128, 1, G.GmmEngine.region_bytes(C, rows, K, N))
    session = C.Session(0, 1, layout.total, 20.0)
    session.attach_peers([session.workspace])
    try:
        d_x, d_w, d_c = x.to(dev), w.to(dev), torch.tensor(counts, dtype=torch.int32, device=dev)
        outs = []
        for blocks in (9, 8, 6, 5, 2):
            assert C.gmm_narrow_tiles(3, counts[-1], rows, K, N, blocks) is (blocks >= 6)
            eng = G.GmmEngine([session], layout, dev, rows, K, N, num_sms=blocks)
            outs.append(torch.full((rows, N), float("nan"), dtype=torch.bfloat16, device=dev))
            eng.a2av_gmm([d_x], [d_w], [d_c], [outs[-1]], num_experts=4)
            torch.cuda.synchronize()
            eng.check()
        # one rounding to bf16 (2^-9 of the value) behind fp32 sums of K products
        assert torch.allclose(outs[0].float().cpu(), ref, rtol=2.0 ** -8, atol=1e-4)
        assert all(torch.equal(outs[0], o) for o in outs[1:])
    finally:
        torch.cuda.synchronize()
        session.close()


def test_two_ranks_odd_sizes():
    _world(2, 6, 192, 320, 500, seed=3, empty_expert=2)


def test_zero_copy_views():
    _world(2, 4, 128, 128, 400, seed=9, zero_copy=True)


def test_four_ranks():
    _world(4, 8, 512, 512, 700, seed=5)


def test_eight_ranks_many_experts():
    _world(8, 32, 128, 256, 300, seed=7, empty_expert=9)


def test_row_counts_that_do_not_fit_are_reported():
    from deepep_b200.ops import load_native

    C = load_native()
    dev = torch.device("cuda")
    E, K, N, max_rows = 2, 64, 64, 256
    layout = C.make_mega_layout(1, 1, 128, 1, G.GmmEngine.region_bytes(C, max_rows, K, N))
    s = C.Session(0, 1, layout.total, 20.0)
    s.attach_peers([s.workspace])
    try:
        eng = G.GmmEngine([s], layout, dev, max_rows, K, N)
        x = torch.zeros((100, K), dtype=torch.bfloat16, device=dev)
        w = torch.zeros((E, K, N), dtype=torch.bfloat16, device=dev)
        counts = torch.tensor([90, 90], dtype=torch.int32, device=dev)     # 180 rows claimed, 100 staged
        out = torch.zeros((180, N), dtype=torch.bfloat16, device=dev)
        eng.a2av_gmm([x], [w], [counts], [out], num_experts=E)
        torch.cuda.synchronize()
        with pytest.raises(RuntimeError, match="row counts"):
            eng.check()
    finally:
        s.close()


def _real_worker(rank, world, port, results):
    import os

    import torch.distributed as dist

    os.environ.update(MASTER_ADDR="127.0.0.1", MASTER_PORT=str(port), NCCL_NVLS_ENABLE="0")
    torch.cuda.set_device(rank)
    dev = torch.device("cuda", rank)
    dist.init_process_group("nccl", rank=rank, world_size=world, device_id=dev)
    try:
        E, K, N, max_rows = 8, 256, 320, 600
        L = E // world
        counts = _counts(world, E, max_rows, 21, empty_expert=3)
        gen = torch.Generator().manual_seed(22)
        xs = [torch.randn((sum(c), K), generator=gen).to(torch.bfloat16) for c in counts]
        ws = [(torch.randn((L, K, N), generator=gen) / K ** 0.5).to(torch.bfloat16) for _ in range(world)]
        ws2 = [(torch.randn((L, K, N), generator=gen) / K ** 0.5).to(torch.bfloat16) for _ in range(world)]
        ref_out, ref_g = G.reference_alltoallv_gmm(xs, ws, counts, E)
        ref_back = G.reference_gmm_alltoallv(ref_g, ws2, counts, E)
        G.init_group(dist.group.WORLD, max_rows=max_rows, max_k=K, max_n=N, timeout=30.0)
        glob = [counts[s][rank * L + l] for s in range(world) for l in range(L)]
        for rep in range(2):
            out, gathered = G.alltoallv_gmm(xs[rank].to(dev), ws[rank].to(dev), counts[rank], torch.tensor(glob, device=dev),
                                            ep_size=world, expert_num=E, output_all_to_allv=True)
            back = G.gmm_alltoallv(gathered, ws2[rank].to(dev), torch.tensor(counts[rank], device=dev), glob, ep_size=world, expert_num=E)
            torch.cuda.synchronize()
            assert torch.equal(gathered.cpu(), ref_g[rank])
            _close(out, ref_out[rank], f"a2av_gmm rank {rank} rep {rep}")
            _close(back, ref_back[rank], f"gmm_a2av rank {rank} rep {rep}")
        results[rank] = True
    except Exception as exc:  # surfaced by the parent
        results[rank] = repr(exc)
    finally:
        G.destroy_group()
        dist.destroy_process_group()


@pytest.mark.parametrize("world", [2, 4])
def test_real_ranks_public_api(world):
    import socket

    import torch.multiprocessing as mp

    if torch.cuda.device_count() < world:
        pytest.skip(f"needs {world} GPUs")
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        port = s.getsockname()[1]
    results = mp.Manager().dict()
    mp.spawn(_real_worker, args=(world, port, results), nprocs=world, join=True)
    assert dict(results) == {r: True for r in range(world)}
