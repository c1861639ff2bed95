"""Host-side logic of the CUDA engine with a recording stand-in for the native module (no GPU): how blocks are divided
between the NVLink side and the local side, worst-case row capacities, and the passes of a combine whose workspace
holds the partials of a token window only.  Parity: the reference tests its host ops against a fake native module
(``tests/runtime/test_runtime.py``)."""
import types

import pytest
import torch

from deepep_b200.parallel import engine_cuda as EC


def make_engine(world=4, n=1, sm_count=148, max_tokens=1024, partial_tokens=1024, topk=8, hidden=256, local_direct=True):
    calls = []

    class Native:
        def combine(self, lay, sessions, args, send, recv, stream, local_direct, profile, begin, end):
            calls.append(dict(send=send, recv=recv, begin=begin, end=end, ranks=len(args), local_direct=local_direct))

    eng = object.__new__(EC.CudaEngine)
    eng.C, eng.sessions, eng.n, eng.world, eng.sm_count = Native(), [object()] * n, n, world, sm_count
    eng.device = torch.device("cpu")
    eng.layout = types.SimpleNamespace(world=world, max_tokens=max_tokens, partial_tokens=partial_tokens, topk=topk, hidden=hidden)
    eng.default_blocks = eng.combine_blocks = eng.dispatch_blocks = max(2, min(sm_count // n, sm_count - 4))
    eng.combine_send_fraction = EC.COMBINE_SEND_FRACTION.get(world, 0.6)
    eng.dispatch_send_fraction = EC.DISPATCH_SEND_FRACTION.get(world, 0.35)
    eng.local_direct, eng._profile, eng._device_profile, eng._prof, eng._timings = local_direct, False, False, {}, []
    eng._stream = lambda stream=None: 0
    return eng, calls


def plan_for(tokens, rows, topk=8):
    z = torch.zeros(4, dtype=torch.int32)
    return types.SimpleNamespace(num_tokens=tokens, stage_meta=z, rank_rows=z, rank_tokens=z, send_slot=z,
                                 topk_idx=torch.zeros(4, dtype=torch.int64), meta_stride=10, num_experts=16, expand=True, num_rows=rows)


def test_block_division():
    eng, _ = make_engine(world=8)
    assert eng.split_blocks(0, 0.35) == (50, 94)                       # default budget: all but four SMs
    assert eng.split_blocks(64, 0.5) == (32, 32) and eng.split_blocks(3, 0.99) == (2, 1) and eng.split_blocks(2, 0.0) == (1, 1)
    assert eng.split_blocks(10_000, 0.6) == (89, 59)                   # a request above the device is cut to it
    one, _ = make_engine(world=1)
    assert one.split_blocks(100, 1.0) == (100, 0) and one.split_blocks(100, 0.0) == (0, 100)     # one rank, direct local rows
    staged, _ = make_engine(world=1, local_direct=False)
    assert staged.split_blocks(100, 1.0) == (99, 1)                    # rows go through the staging area: both sides needed


def test_worst_case_row_capacity():
    eng, _ = make_engine(world=4, max_tokens=1000, topk=8)
    assert eng.row_capacity(16, 1, True) == 4 * 1000 * 4               # four local experts bound the copies of a token
    assert eng.row_capacity(256, 1, True) == 4 * 1000 * 8
    assert eng.row_capacity(256, 128, True) == 4 * 1000 * 8 + 64 * 127  # every local expert may need a full pad
    assert eng.row_capacity(256, 1, False) == 4 * 1000                 # rank layout: one row per (source, token)


def test_combine_runs_one_pass_per_token_window():
    # real ranks cannot see each other's batch sizes: every rank runs every pass of the capped workspace
    eng, calls = make_engine(world=4, n=1, max_tokens=1024, partial_tokens=256)
    x = torch.zeros((8, 256), dtype=torch.bfloat16)
    out = eng.combine([x], [plan_for(300, 8)], [None])
    assert [(c["begin"], c["end"]) for c in calls] == [(0, 256), (256, 512), (512, 768), (768, 1024)]
    assert out[0][0].shape == (300, 256) and out[0][1] is None and all(c["send"] + c["recv"] == 144 for c in calls)
    # virtual ranks share one launch and know all batch sizes: passes stop at the largest batch
    eng, calls = make_engine(world=2, n=2, max_tokens=1024, partial_tokens=256)
    eng.combine([x, x], [plan_for(300, 8), plan_for(10, 8)], [None, None])
    assert [(c["begin"], c["end"]) for c in calls] == [(0, 256), (256, 512)] and calls[0]["ranks"] == 2
    # a workspace that holds all partials: one pass
    eng, calls = make_engine(world=4, n=1, max_tokens=1024, partial_tokens=1024)
    w = torch.zeros((8,), dtype=torch.float32)
    out = eng.combine([x], [plan_for(0, 8)], [w], split=(40, 24))
    assert [(c["begin"], c["end"], c["send"], c["recv"]) for c in calls] == [(0, 1024, 40, 24)] and out[0][1].shape == (0, 8)
    with pytest.raises(ValueError, match="must not exceed 148"):
        eng.combine([x], [plan_for(4, 8)], [None], split=(100, 60))


def test_a_handle_watches_the_tables_that_kernels_read_again():
    """The V1 handle's prefix tables and source tokens lie beside the routing tables, but changing them in place is the caller's
    business, as it is with a tensor of its own; a changed routing table is refused."""
    from deepep_b200.parallel.elastic import EPHandle

    ints, views = EC._slab_layout(5, 1, 2, 64, 4, 1, 8, 10, 1)
    slab = torch.zeros((ints,), dtype=torch.int32)
    for name, write in [(n, lambda t: t.add_(1)) for n in views] + [("recv_src_idx", lambda t: t[:3].fill_(7))]:
        plan = EC.RoutingPlan(num_tokens=5, num_experts=8, num_topk=2, expand=False, alignment=1, meta_stride=4, num_rows=10,
                              num_staged_rows=10, expert_counts_list=[0] * 8, topk_idx=torch.zeros((5, 2), dtype=torch.int64), recv_w=None,
                              recv_idx=None, slab=slab, slab_ptr=slab.data_ptr(), views=views)
        handle = EPHandle(False, 8, 1, 64, 0, plan.topk_idx, 10, 10, [0] * 8, *[None] * 7)
        handle._plan = plan
        handle._snapshot()
        table = getattr(plan, name)
        assert table.shape == torch.Size(views[name][1]) and table.data_ptr() == slab.data_ptr() + 4 * views[name][0]
        write(table)
        if name in ("rank_matrix", "rank_prefix", "send_chunk_prefix", "recv_src_idx"):
            handle._check_unchanged()
        else:
            with pytest.raises(RuntimeError, match="modified in place"):
                handle._check_unchanged()


def test_rows_off_their_boundary_are_refused(monkeypatch):
    """The kernels read and write rows in pieces of 16 bytes: a tensor that starts between two of them (a slice of a longer one) is
    refused by every launch, before anything is queued.  Sessions on host-memory doubles of the CUDA entry points."""
    from deepep_b200.models.mega_moe import MegaEngine, MegaWeights
    from deepep_b200.ops import ep_gmm_fused as G, load_native

    C = load_native(build_if_missing=True)
    C.testing_install_fake_cuda(True)
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda device: types.SimpleNamespace(multi_processor_count=148))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: types.SimpleNamespace(cuda_stream=0, synchronize=lambda: None))
    cpu, T, H, K, E = torch.device("cpu"), 4, 128, 2, 4
    rows = lambda n, shift=1, dtype=torch.bfloat16, width=H: torch.zeros((n * width + 8,), dtype=dtype)[shift:shift + n * width].view(n, width)
    assert rows(T).is_contiguous() and rows(T).data_ptr() % 16 and rows(T, 0).data_ptr() % 16 == 0
    sessions = []

    def session(layout):
        sessions.append(C.Session(0, 1, layout.total, 5.0, "ipc"))
        sessions[-1].attach_peers([sessions[-1].workspace])
        return [sessions[-1]]

    try:
        layout = C.make_layout(1, T, H, K, C.ll_region_bytes(1, T, K, H), 0, 0)
        eng = EC.CudaEngine(session(layout), layout, cpu)
        idx, w = torch.zeros((T, K), dtype=torch.int64), torch.ones((T, K))
        ints, views = EC._slab_layout(T, 1, K, T, 4, 1, E, T * K, 0)
        slab = torch.zeros((ints,), dtype=torch.int32)
        plan = EC.RoutingPlan(num_tokens=T, num_experts=E, num_topk=K, expand=True, alignment=1, meta_stride=4, num_rows=T * K,
                              num_staged_rows=T, expert_counts_list=[T * K, 0, 0, 0], topk_idx=idx, recv_w=None, recv_idx=None, slab=slab,
                              slab_ptr=slab.data_ptr(), views=views)
        low = EC.RoutingPlan(num_tokens=T, num_experts=E, num_topk=K, expand=True, alignment=1, meta_stride=0, num_rows=T, num_staged_rows=0,
                             expert_counts_list=None, topk_idx=idx, recv_w=None, recv_idx=None, topk_w=w, local_row_ptr=slab.data_ptr())
        low.recv_row_src = low.num_rows_dev = slab
        calls = [lambda: eng.dispatch([rows(T)], [plan], 0), lambda: eng.dispatch([(rows(T, 1, torch.float8_e4m3fn), torch.ones((T, 1)))], [plan], 1),
                 lambda: eng.combine([rows(T * K)], [plan], [None]),
                 lambda: eng.combine([rows(T * K, 0)], [plan], [None], bias=[(rows(T, 0), rows(T))]),
                 lambda: eng.ll_dispatch([rows(T)], [idx], [w], E, 0, cpu_sync=False), lambda: eng.ll_combine([rows(T)], [low])]
        glayout = C.make_mega_layout(1, 1, H, 1, G.GmmEngine.region_bytes(C, 8, H, H))
        gmm = G.GmmEngine(session(glayout), glayout, cpu, 8, H, H)
        weight, counts = torch.zeros((2, H, H), dtype=torch.bfloat16), torch.tensor([2, 2], dtype=torch.int32)
        calls += [lambda: gmm.a2av_gmm([rows(T)], [weight], [counts], [rows(T, 0)], num_experts=2),
                  lambda: gmm.a2av_gmm([rows(T, 0)], [weight], [counts], [rows(T, 0)], [rows(T)], num_experts=2),
                  lambda: gmm.gmm_a2av([rows(T, 0)], [weight], [counts], [rows(T)], num_experts=2)]
        mlayout = C.make_mega_layout(1, T, 256, K, MegaEngine.mega_bytes(C, T, 256, K))
        mega = MegaEngine(session(mlayout), mlayout, cpu, E, 128)
        one = [MegaWeights(torch.zeros((64, 64), dtype=torch.uint8), torch.zeros((512,), dtype=torch.uint8), E, 256, 256)]
        wide = lambda shift: rows(T, shift, width=256)
        stream = types.SimpleNamespace(cuda_stream=0)
        calls += [lambda: mega.forward([wide(1)], [T], one, one, stream), lambda: mega.forward([wide(0)], [T], one, one, stream, x_bf16=[wide(1)])]
        table = dict(mapping=slab.data_ptr(), rows=T, topk=K, expanded_rows=T)
        fixed = dict(table, out_sf=None, out_w=None, x_sf=None, topk_idx=None, topk_w=None, expert_offsets=slab.data_ptr(),
                     actual_counts=slab.data_ptr(), tile_counts=None, err=None, caps=None, experts=E, row_bytes=2 * H, num_sf=0, cached=1)
        good, bad = rows(T, 0), rows(T)
        for x, out in ((bad, good), (good, bad)):
            calls += [lambda x=x, out=out: C.expand(dict(fixed, x=x.data_ptr(), out=out.data_ptr()), 1, 0),
                      lambda x=x, out=out: C.aggregate(dict(table, x=x.data_ptr(), out=out.data_ptr(), row_w=None, values=None, out_values=None,
                                                            hidden=H, is_half=0), 0)]
        for call in calls:
            with pytest.raises(ValueError, match="16-byte boundary"):
                call()
    finally:
        for s in sessions:
            s.close()
        C.testing_restore_cuda()
        C.testing_clear()


def test_status_block_becomes_a_readable_error():
    class Session:
        def __init__(self, **status):
            self._status = dict(code=0, op=0, rank=0, peer=0, where=0, expected=0, seen=0, **status) if not status else status

        def status(self):
            return self._status

    eng = object.__new__(EC.CudaEngine)
    eng.sessions = [Session()]
    eng.check_status()                                                     # code 0: nothing to report
    eng.sessions = [Session(), Session(code=1, op=3, rank=5, peer=2, where=1, expected=7, seen=6)]
    with pytest.raises(EC.CommunicationError, match=r"rank 5: combine timeout at wait site 1 \(the partial sums of an expert rank\) on "
                                                     r"peer 2 \(expected 7, saw 6\); restart"):
        eng.check_status()
    eng.sessions = [Session(code=2, op=2, rank=0, peer=-1, where=103, expected=10, seen=12)]
    with pytest.raises(EC.CommunicationError, match=r"dispatch bad argument at wait site 103 on peer -1"):
        eng.check_status()
    assert all(op in EC.OP_NAMES for op, _ in EC.WAIT_SITES)


def test_argument_keys_agree_between_python_and_the_bindings():
    """The engine hands every kernel its arguments as a dict; the bindings read the keys they know and treat a missing one
    as null / zero.  A misspelt key would therefore go unnoticed until a kernel dereferences the null: the two key sets
    must be equal for every operation."""
    import ast
    import os
    import re

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

    def cpp_keys(path, func):
        src = open(os.path.join(root, "deepep_b200", "csrc", path)).read()
        start = src.index("{", src.index(func + "("))
        depth, at = 0, start
        while True:
            depth += {"{": 1, "}": -1}.get(src[at], 0)
            if depth == 0:
                break
            at += 1
        body = src[start:at]
        return set(re.findall(r'\(d, "([A-Za-z0-9_]+)"', body)) | set(re.findall(r'd\["([A-Za-z0-9_]+)"\]', body))

    tree = ast.parse(open(os.path.join(root, "deepep_b200", "parallel", "engine_cuda.py")).read())
    methods = {f.name: f for n in ast.walk(tree) if isinstance(n, ast.ClassDef) and n.name == "CudaEngine"
               for f in n.body if isinstance(f, ast.FunctionDef)}

    def py_keys(method):
        keys = set()
        for call in ast.walk(methods[method]):
            if isinstance(call, ast.Call) and getattr(call.func, "attr", None) == "append" and call.args \
                    and isinstance(call.args[0], ast.Call) and getattr(call.args[0].func, "id", None) == "dict":
                keys |= {k.arg for k in call.args[0].keywords}
        return keys

    for func, path, method in (("op_notify", "bindings.cpp", "notify"), ("op_dispatch", "bindings.cpp", "dispatch"),
                               ("op_combine", "bindings.cpp", "combine"), ("op_ll_dispatch", "ll_bindings.cpp", "ll_dispatch"),
                               ("op_ll_combine", "ll_bindings.cpp", "ll_combine")):
        native, python = cpp_keys(path, func), py_keys(method)
        assert python and native == python, (func, sorted(python - native), sorted(native - python))


@pytest.mark.parametrize("world", [1, 2])
def test_scratch_of_the_routing_pass(monkeypatch, world):
    """Several ranks' counts pass through memory that the engine owns; a single rank's stay on the chip, and nothing is allocated."""
    monkeypatch.setattr(EC, "require_native", lambda name: types.SimpleNamespace(chunk_tokens=64, max_experts=1024))
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda device: types.SimpleNamespace(multi_processor_count=148))
    eng = EC.CudaEngine([None], types.SimpleNamespace(world=world, max_tokens=100, partial_tokens=100, topk=2, hidden=64), torch.device("cpu"))
    shapes = {name: tuple(t.shape) for name, t in eng._scratch[0].items()}
    assert shapes == ({} if world == 1 else dict(hist=(4 * 1024,), hits=(4,), own_hits=(4,), cnt=(2 * 1024,)))
    calls = []
    eng.C.notify = lambda lay, sessions, args, *rest: calls.append(args[0])
    eng._stream = lambda stream=None: 0
    eng.notify([torch.zeros((100, 2), dtype=torch.int64)], [None], 4, cpu_sync=False)
    assert all((calls[0][name] is None) == (world == 1) for name in ("hist", "hits", "own_hits", "cnt"))
