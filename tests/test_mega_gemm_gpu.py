"""Block-scaled tcgen05 grouped GEMM (e4m3 x e2m1, ue8m0 per 32) against an fp32 PyTorch reference."""
import pytest
import torch

from deepep_b200.oracle import megamoe as O

pytestmark = pytest.mark.gpu


def _run(rows_per_expert, n_total, k, seed=0, b_tx=None, pair=False, stages=0, commit_every=0, blocks=148, swap=False):
    from deepep_b200.ops import load_native

    C = load_native()
    dev = torch.device("cuda")
    g = torch.Generator().manual_seed(seed)
    experts = len(rows_per_expert)
    tiles = [-(-r // 256) * 2 if pair else -(-r // 128) for r in rows_per_expert]   # CTA pairs: whole pairs of tiles per expert
    rows_pad = 128 * sum(tiles)
    x = torch.randn((rows_pad, k), generator=g)
    a_codes, a_sf = O.quantize_mxfp8(x)
    packed = torch.randint(0, 256, (experts * n_total, k // 2), generator=g, dtype=torch.uint8)
    b_sf = torch.randint(118, 123, (experts * n_total, k // 32), generator=g, dtype=torch.uint8)
    mtile_expert = torch.tensor([e for e, t in enumerate(tiles) for _ in range(t)], dtype=torch.int32)
    ref = torch.empty((rows_pad, n_total))
    a_f, b_f = O.dequantize_mxfp8(a_codes, a_sf), O.unpack_fp4(packed, b_sf)
    short = torch.zeros((rows_pad,), dtype=torch.bool)              # rows behind the end of a tile that is told its rows
    told = mtile_expert.clone()
    if swap:
        rows = [min(128, r - 128 * t) for r, n in zip(rows_per_expert, tiles) for t in range(n)]
        told |= torch.tensor(rows, dtype=torch.int32) << C.mega_tile_rows_shift
        for mt, r in enumerate(rows):
            short[mt * 128 + r:(mt + 1) * 128] = True
    for mt, e in enumerate(mtile_expert.tolist()):
        ref[mt * 128:(mt + 1) * 128] = a_f[mt * 128:(mt + 1) * 128] @ b_f[e * n_total:(e + 1) * n_total].t()
    d = dict(a=a_codes.view(torch.uint8).to(dev), b=O.tile_fp4_rows(packed).to(dev), sfa=O.to_sf_chunks(a_sf).to(dev), sfb=O.to_sf_chunks(b_sf).to(dev),
             mt=told.to(dev), n=torch.tensor([len(mtile_expert)], dtype=torch.int32, device=dev),
             c=torch.zeros((rows_pad, n_total), dtype=torch.float32, device=dev), err=torch.zeros(1, dtype=torch.int32, device=dev))
    args = dict(a=d["a"].data_ptr(), b=d["b"].data_ptr(), sfa=d["sfa"].data_ptr(), sfb=d["sfb"].data_ptr(),
                mtile_expert=d["mt"].data_ptr(), num_mtiles=d["n"].data_ptr(), rows_pad=rows_pad, k=k, b_rows=experts * n_total,
                n_total=n_total, epi=0, c=d["c"].data_ptr(), ldc=n_total, error_flag=d["err"].data_ptr())
    if b_tx is not None:
        args["b_tx_bytes"] = b_tx
    if pair:
        args["pair"] = 1
    if swap:
        args["swap"] = 1
    if stages:
        args["stages"] = stages
    if commit_every:
        args["commit_every"] = commit_every
    C.mega_gemm(args, None, blocks, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert d["err"].item() == 0, "a pipeline wait ran out inside the GEMM kernel"
    out = d["c"].cpu()
    ref[short], out[short] = 0.0, 0.0
    err = (out - ref).abs().max().item()
    scale = ref.abs().max().item()
    assert err <= 2e-3 * scale + 1e-3, f"max abs error {err} (reference scale {scale})"


def test_single_tile():
    _run([128], 256, 128)


def test_k_loop_and_tiles():
    _run([128, 256], 256, 1024)


def test_grouped_shapes():
    _run([100, 1, 300, 128], 512, 2048, seed=3)


@pytest.mark.parametrize("rows", [[1], [16], [17, 32, 33, 128], [31, 5, 150, 48, 300], [32] * 40])
def test_swapped_operands(rows):
    """Tiles of few rows multiply the weights by the rows: next to tiles that do not, short and whole scale groups, one and several
    tiles a block."""
    _run(rows, 256, 128, seed=1, swap=True)
    _run(rows, 512, 896, seed=2, swap=True, blocks=3)


def test_cta_pairs_single_pair():
    """One pair of row blocks, one N tile: the smallest case of the cta_group::2 path (two CTAs, M = 256)."""
    _run([256], 256, 128, pair=True)


def test_cta_pairs_grouped_shapes():
    """Several experts (odd tile counts are padded to whole pairs), a K loop longer than the pipeline, several N tiles."""
    _run([100, 1, 300, 256], 512, 2048, seed=3, pair=True)


def test_pipeline_depth_and_commit_grouping():
    """The operand pipeline with other depths and with two stages released per commit gives the same numbers (K loop of
    16 steps, longer than any of the pipelines; plain and CTA-pair kernels)."""
    _run([128, 256], 256, 2048, seed=5, stages=2)
    _run([128, 256], 256, 2048, seed=5, stages=4, commit_every=2)
    _run([256, 512], 512, 2048, seed=6, pair=True, stages=6, commit_every=2)
    _run([256], 256, 2048, seed=7, pair=True, stages=3)


@pytest.mark.parametrize("k", [128, 256, 640, 896, 1152])
@pytest.mark.parametrize("pair, stages", [(False, 2), (False, 4), (True, 4), (True, 6)])
def test_short_scale_groups(k, pair, stages):
    """Tiles whose last group of scales holds one to four of its K steps, several tiles per CTA in a row: with four stages or more
    the two slots of the scales are filled again while younger steps than the oldest stage are still being multiplied (two stages:
    the wait for the stage always covers the slot)."""
    _run([256, 100, 130], 512, k, seed=k + stages, pair=pair, stages=stages, blocks=2)


@pytest.mark.parametrize("k", [128, 640, 1152])
@pytest.mark.parametrize("pair, stages", [(False, 4), (True, 6)])
def test_short_scale_groups_with_two_stages_per_commit(k, pair, stages):
    """The last step of a group of scales may be the first of the two that share a commit: the slot waits for the second one too."""
    _run([256, 100, 130], 512, k, seed=k, pair=pair, stages=stages, commit_every=2, blocks=2)


def _exact_operands(tiles, n_total, k, exponent, seed):
    """Operands whose products and sums are exact in fp32 in any order: codes -2..2, e2m1 weights, one scale of 2^exponent."""
    g = torch.Generator().manual_seed(seed)
    rows, experts = 128 * len(tiles), max(tiles) + 1
    a = torch.randint(-2, 3, (rows, k), generator=g).float().to(torch.float8_e4m3fn)
    packed = torch.randint(0, 256, (experts * n_total, k // 2), generator=g, dtype=torch.uint8)
    a_sf = torch.full((rows, k // 32), 127, dtype=torch.uint8)
    b_sf = torch.full((experts * n_total, k // 32), 127 + exponent, dtype=torch.uint8)
    b = O.unpack_fp4(packed, b_sf).view(experts, n_total, k)
    product = torch.cat([a[128 * i:128 * i + 128].float() @ b[e].t() for i, e in enumerate(tiles)])
    dev = torch.device("cuda")
    d = dict(a=a.view(torch.uint8).to(dev), b=O.tile_fp4_rows(packed).to(dev), sfa=O.to_sf_chunks(a_sf).to(dev),
             sfb=O.to_sf_chunks(b_sf).to(dev), mtile_expert=torch.tensor(tiles, dtype=torch.int32, device=dev),
             num_mtiles=torch.tensor([len(tiles)], dtype=torch.int32, device=dev), error_flag=torch.zeros(1, dtype=torch.int32, device=dev))
    args = dict({name: t.data_ptr() for name, t in d.items()}, rows_pad=rows, k=k, b_rows=experts * n_total, n_total=n_total)
    return product, d, args


@pytest.mark.parametrize("k, pair", [(128, False), (640, False), (640, True), (1152, False)])
def test_combine_epilogue_writes_exact_rows(k, pair):
    """Rows of several tiles per CTA, turned in registers, land in the slots that ``row_src`` names and nowhere else, each the
    product rounded once to bf16."""
    from deepep_b200.models.mega_moe import _view
    from deepep_b200.ops import load_native

    C, dev, tiles, hidden, topk = load_native(), torch.device("cuda"), [0, 0, 1, 1, 2, 2], 512, 3
    product, d, args = _exact_operands(tiles, hidden, k, 0, seed=k)
    rows, M = product.shape[0], 300
    layout = C.make_mega_layout(1, M, 128, topk, M * topk * hidden * 2 + 1024)
    session = C.Session(0, 1, layout.total, 20.0)
    session.attach_peers([session.workspace])
    try:
        g = torch.Generator().manual_seed(k + 1)
        slot = torch.randperm(M * topk, generator=g)[:rows].to(torch.int32)
        slot[torch.rand(rows, generator=g) < 0.2] = -1             # padding rows
        comb = _view(session.workspace + layout.mega, M * topk * hidden * 2, dev).view(torch.bfloat16).view(M * topk, hidden)
        comb.fill_(-7.0)
        row_src = slot.to(dev)
        C.mega_gemm(dict(args, epi=2, row_src=row_src.data_ptr(), comb_off=layout.mega, max_tokens=M, topk=topk, hidden=hidden,
                         pair=int(pair)), session, 4, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert d["error_flag"].item() == 0
        want = torch.full((M * topk, hidden), -7.0, dtype=torch.bfloat16)
        want[slot[slot >= 0].long()] = product[slot >= 0].bfloat16()
        assert torch.equal(comb.cpu(), want)
    finally:
        torch.cuda.synchronize()
        session.close()


@pytest.mark.parametrize("k, pair", [(128, False), (640, False), (640, True), (1152, False)])
def test_swiglu_epilogue_of_exact_products(k, pair):
    """The drained halves of several tiles per CTA: the activation of each bf16 product, requantised.  The fast exponential and
    division may move a value over a rounding line: one e4m3 step (2^-3 of the value, the block's smallest step below that)."""
    from deepep_b200.ops import load_native

    C, tiles, inter = load_native(), [0, 0, 1, 1, 2, 2], 256
    product, d, args = _exact_operands(tiles, 2 * inter, k, -7, seed=k + 2)
    rows = product.shape[0]
    a2 = torch.zeros((rows, inter), dtype=torch.uint8, device="cuda")
    a2_sf = torch.zeros((rows // 128 * (inter // 128) * 512,), dtype=torch.uint8, device="cuda")
    C.mega_gemm(dict(args, epi=1, a2=a2.data_ptr(), a2_sf=a2_sf.data_ptr(), inter=inter, pair=int(pair)), None, 4,
                torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert d["error_flag"].item() == 0
    first = O.bf16(product).view(rows, inter // 128, 2, 128)        # every 256 columns: 128 of the gate, 128 of up
    gate, up = first[:, :, 0].reshape(rows, inter), first[:, :, 1].reshape(rows, inter)
    codes, sf = O.quantize_mxfp8(gate / (1 + torch.exp(torch.clamp(-gate, -80, 80))) * up)
    want, chunks = O.dequantize_mxfp8(codes, sf), O.to_sf_chunks(sf)
    assert (a2_sf.cpu() != chunks).float().mean() < 1e-3
    got_sf = torch.empty_like(sf)
    r, b = torch.meshgrid(torch.arange(rows), torch.arange(inter // 32), indexing="ij")
    got_sf[r, b] = a2_sf.cpu()[((r // 128) * (inter // 128) + b // 4) * 512 + r % 32 * 16 + r % 128 // 32 * 4 + b % 4]
    got = O.dequantize_mxfp8(a2.cpu().view(torch.float8_e4m3fn), got_sf)
    step = want.abs() / 8 + want.view(rows, -1, 32).abs().amax(-1).repeat_interleave(32, dim=1) * 2.0 ** -16
    assert bool(((got - want).abs() <= step).all()) and (got != want).float().mean() < 1e-3
