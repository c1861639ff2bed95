"""What an asynchronous call keeps alive: every tensor whose address a kernel got is either owned by the buffer or held by the
returned event, so that nothing goes back to the allocator while the communication stream still uses it.  The CUDA engine runs
on CPU tensors with a recording stand-in for the native module (no GPU)."""
import contextlib
import types

import pytest
import torch

import deepep_b200 as deep_ep
from deepep_b200.parallel import engine_cuda as EC
from helpers import make_routes, make_weights

T, H, E, K, M = 40, 256, 8, 3, 64


class Native:
    """Records the address arguments of the calls."""
    chunk_tokens, max_experts = 64, 1024

    def __init__(self):
        self.addresses = []

    def __getattr__(self, op):
        def call(lay, sessions, args, *rest):
            for d in args:
                self.addresses += [(op, key, v) for key, v in d.items() if isinstance(v, int) and v > 1 << 24]
        return call


class FakeStream:
    cuda_stream = 0

    def wait_event(self, event): ...
    def wait_stream(self, other): ...
    def synchronize(self): ...


@pytest.fixture
def buf(monkeypatch):
    if torch.cuda.is_available():
        pytest.skip("the stand-ins replace the streams; test without a GPU")
    made = deep_ep.ElasticBuffer(None, num_max_tokens_per_rank=M, hidden=H, num_topk=K, explicitly_destroy=True, device="cpu")
    stream = FakeStream()
    made.runtime = types.SimpleNamespace(stream=stream, failed=False, ensure_alive=lambda: None, close=lambda: None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: stream)
    monkeypatch.setattr(made, "_on", lambda comm: contextlib.nullcontext())
    eng = object.__new__(EC.CudaEngine)
    eng.C, eng.sessions, eng.n, eng.world, eng.sm_count = Native(), [object()], 1, 1, 148
    eng.device = torch.device("cpu")
    eng.layout = types.SimpleNamespace(world=1, max_tokens=M, partial_tokens=M, topk=K, hidden=H)
    eng.default_blocks = eng.combine_blocks = eng.dispatch_blocks = 144
    eng.dispatch_send_fraction, eng.combine_send_fraction = 1.0, 0.0
    eng.local_direct, eng._profile, eng._device_profile, eng._prof, eng._timings, eng._nt = True, False, False, {}, [], 1
    eng._scratch = [{name: torch.empty((4096,), dtype=torch.int32) for name in ("hist", "hits", "own_hits", "cnt")}]
    made.engine = eng
    yield made
    made.runtime = None


def _spans(item):
    if isinstance(item, torch.Tensor):
        store = item.untyped_storage()
        yield store.data_ptr(), store.data_ptr() + store.nbytes()
    elif isinstance(item, (list, tuple)):
        for inner in item:
            yield from _spans(inner)


def _check(buf, event):
    assert event.event is not None and buf.engine.C.addresses
    held = list(_spans(event._retained_objects)) + list(_spans([list(s.values()) for s in buf.engine._scratch]))
    for op, key, address in buf.engine.C.addresses:
        assert any(lo <= address < hi for lo, hi in held), f"{op}: {key} is not kept alive"
    buf.engine.C.addresses.clear()


def _inputs():
    x = torch.randn(T, H).bfloat16()
    return x, make_routes("random", T, E, K, 1, 5), make_weights(T, K, 2)


def test_low_latency_calls(buf):
    x, idx, w = _inputs()
    rx, _, _, handle, event = buf.dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E, do_cpu_sync=False,
                                           async_with_compute_stream=True)
    assert handle.is_low_latency
    _check(buf, event)
    event = buf.dispatch(x, handle=handle, async_with_compute_stream=True)[4]
    _check(buf, event)
    event = buf.dispatch(x, handle=handle, async_with_compute_stream=True, allocate_on_comm_stream=True)[4]
    _check(buf, event)
    out, _, event = buf.combine(rx, handle, async_with_compute_stream=True)
    _check(buf, event)


@pytest.mark.parametrize("expand,alignment", [(True, 1), (True, 16), (False, 1)])
def test_high_throughput_calls(buf, expand, alignment):
    x, idx, w = _inputs()
    rx, _, rw, handle, event = buf.dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E, do_expand=expand, do_cpu_sync=False,
                                            expert_alignment=alignment, num_max_tokens_per_rank=512, async_with_compute_stream=True)
    assert not handle.is_low_latency
    _check(buf, event)
    event = buf.dispatch(x, handle=handle, async_with_compute_stream=True)[4]
    _check(buf, event)
    event = buf.combine(rx, handle, topk_weights=rw, bias=(x, x.clone()), async_with_compute_stream=True)[2]
    _check(buf, event)


def test_combine_operands_that_are_not_rows_behind_rows(buf, monkeypatch):
    """A bias that is one row for all tokens, or strided, and strided weights are copied, on the communication stream: what the kernel
    gets lies row behind row, and the event holds it and what it was copied from."""
    x, idx, w = _inputs()
    rx, _, rw, handle, event = buf.dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E, do_expand=True, do_cpu_sync=False,
                                            num_max_tokens_per_rank=512, async_with_compute_stream=True)
    _check(buf, event)
    where = []
    monkeypatch.setattr(buf, "_on", lambda comm: (where.append(comm), contextlib.nullcontext())[1])
    seen = []
    launch = buf.engine.combine
    monkeypatch.setattr(buf.engine, "combine", lambda xs, plans, ws, bias=None, **k: (seen.append((ws[0], *bias[0])), launch(xs, plans, ws, bias=bias, **k))[1])
    one, wide = torch.randn(H).bfloat16(), torch.randn(T, 2 * H).bfloat16()
    for weights, bias in ((rw, (one.expand(T, H), None)), (rw, (wide[:, ::2], x)), (torch.stack([rw, rw], 1)[:, 0], (x, one.expand(T, H)))):
        event = buf.combine(rx, handle, topk_weights=weights, bias=bias, async_with_compute_stream=True)[2]
        for got, want in zip(seen.pop(), (weights, *bias)):
            assert (got is None) == (want is None)
            assert got is None or got.is_contiguous() and torch.equal(got.nan_to_num(), want.nan_to_num()) and (got is want) == want.is_contiguous()
        held = [t for t in event._retained_objects if isinstance(t, torch.Tensor)]
        assert all(any(t is h for h in held) for t in (weights, *bias) if t is not None) and where[0] is buf.runtime.stream
        _check(buf, event)
        where.clear()
    with pytest.raises(ValueError, match="buffer's device"):
        monkeypatch.setattr(buf, "on_cuda", True)
        buf.combine(rx, handle)


def test_v1_rank_matrix(buf):
    """The per-rank counts of the V1 handle are added up on the communication stream: kept alive by the event, and not cleared by
    torch on the current stream, which nothing would order before the additions (the launcher clears them)."""
    from torch.utils._python_dispatch import TorchDispatchMode

    cleared = []

    class Watch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            if "zero" in str(func) or "fill" in str(func):
                cleared.append(str(func))
            return func(*args, **(kwargs or {}))

    x, idx, w = _inputs()
    with Watch():
        event = buf.dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E, do_expand=False, do_cpu_sync=False,
                             num_max_tokens_per_rank=512, async_with_compute_stream=True, _rank_matrix=True)[4]
    assert not cleared
    assert any(key == "rank_matrix" for _, key, _ in buf.engine.C.addresses)
    _check(buf, event)
