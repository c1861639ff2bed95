"""Expert-parallel MoE layer for training: autograd through dispatch/combine by handle reversal.

The reference documents the rule (``README.md:168-219``, ``docs/elastic.md:7-17``) but ships no autograd
``Function``: the backward of ``combine`` is a cached ``dispatch`` of the gradient, the backward of
``dispatch`` is a ``combine`` of the row gradients, with the fp32 weight gradients riding the value channel.
"""
from __future__ import annotations

from functools import lru_cache

import torch
from torch.autograd import forward_ad

from ..ops import require_native
from ..parallel.elastic import ElasticBuffer


class _Dispatch(torch.autograd.Function):
    @staticmethod
    def forward(ctx, buffer: ElasticBuffer, x, topk_idx, topk_weights, num_experts, holder):
        recv_x, _, recv_w, handle, _ = buffer.dispatch(x, topk_idx=topk_idx, topk_weights=topk_weights, num_experts=num_experts,
                                                       do_expand=True)
        ctx.buffer, ctx.handle = buffer, handle
        holder["handle"] = handle
        ctx.mark_non_differentiable(handle.psum_num_recv_tokens_per_expert)
        return recv_x, recv_w, handle.psum_num_recv_tokens_per_expert

    @staticmethod
    def backward(ctx, grad_recv_x, grad_recv_w, _):
        gw = None if grad_recv_w is None else grad_recv_w.float().contiguous()
        if gw is None:
            gw = torch.zeros(grad_recv_x.shape[0], dtype=torch.float32, device=grad_recv_x.device)
        grad_x, grad_w, _ = ctx.buffer.combine(grad_recv_x.to(torch.bfloat16).contiguous(), ctx.handle, topk_weights=gw)
        return None, grad_x, None, grad_w, None, None


class _Combine(torch.autograd.Function):
    @staticmethod
    def forward(ctx, buffer: ElasticBuffer, expert_out, handle):
        out, _, _ = buffer.combine(expert_out, handle)
        ctx.buffer, ctx.handle = buffer, handle
        return out

    @staticmethod
    def backward(ctx, grad_out):
        grad_rows, _, _, _, _ = ctx.buffer.dispatch(grad_out.to(torch.bfloat16).contiguous(), handle=ctx.handle)
        return None, grad_rows, None


class _Swiglu(torch.autograd.Function):
    """``silu(gate) * up`` of bf16 rows ``[gate | up]``, one kernel each way."""

    @staticmethod
    def forward(ctx, gate_up):
        rows, width = gate_up.shape
        h = gate_up.new_empty((rows, width // 2))
        ctx.save_for_backward(gate_up)
        _launch("swiglu", gate_up, gate_up.data_ptr(), 0, h.data_ptr(), rows, width // 2, blocks=False)
        return h

    @staticmethod
    def backward(ctx, grad):
        gate_up, = ctx.saved_tensors
        again = torch.is_grad_enabled()                  # the gradient will be differentiated itself
        if again or not _ordinary(gate_up, grad):
            with torch.enable_grad():
                h = _separate_operations(gate_up)
            return torch.autograd.grad(h, gate_up, grad, create_graph=again)[0]
        grad, out = _readable(grad), torch.empty_like(gate_up)
        _launch("swiglu", gate_up, gate_up.data_ptr(), grad.data_ptr(), out.data_ptr(), gate_up.shape[0], gate_up.shape[1] // 2,
                blocks=False)
        return out


class _WeighRows(torch.autograd.Function):
    """bf16 rows times an fp32 weight each (rounded to bf16), one kernel each way; the weight's gradient is summed by torch."""

    @staticmethod
    def forward(ctx, rows, weights):
        out = torch.empty_like(rows)
        ctx.save_for_backward(rows, weights)
        _launch("row_scale", rows, rows.data_ptr(), weights.data_ptr(), out.data_ptr(), 0, 0, *rows.shape)
        return out

    @staticmethod
    def backward(ctx, grad):
        rows, weights = ctx.saved_tensors
        need = ctx.needs_input_grad
        again = torch.is_grad_enabled()
        if again or not _ordinary(rows, weights, grad):
            with torch.enable_grad():
                out = rows * weights.unsqueeze(1).to(rows.dtype)
            grads = iter(torch.autograd.grad(out, [t for t, n in zip((rows, weights), need) if n], grad, create_graph=again))
            return tuple(next(grads) if n else None for n in need)
        grad = _readable(grad)
        out = torch.empty_like(rows) if need[0] else None
        terms = torch.empty_like(rows) if need[1] else None
        _launch("row_scale", rows, grad.data_ptr(), weights.data_ptr(), 0 if out is None else out.data_ptr(),
                0 if terms is None else rows.data_ptr(), 0 if terms is None else terms.data_ptr(), *rows.shape)
        return out, None if terms is None else terms.sum(1, keepdim=True).to(weights.dtype).squeeze(1)


class _WeighAndCombine(torch.autograd.Function):
    """``_WeighRows`` and ``_Combine`` in one kernel each way, for a single rank: the products are never stored, and neither the rows
    of the gradient nor the terms of the weights' gradients are.  The products are rounded as there."""

    @staticmethod
    def forward(ctx, buffer: ElasticBuffer, rows, weights, handle):
        out, _, _ = buffer.combine(rows, handle, _row_weights=weights)
        ctx.buffer, ctx.handle = buffer, handle
        ctx.save_for_backward(rows, weights)
        return out

    @staticmethod
    def backward(ctx, grad):
        buffer, handle, (rows, weights) = ctx.buffer, ctx.handle, ctx.saved_tensors
        need = ctx.needs_input_grad[1:3]
        again = torch.is_grad_enabled()                  # the gradient will be differentiated itself
        if again or not (_weighable(rows, weights, torch.bfloat16) and _ordinary(grad)):
            grad_rows = buffer.dispatch(grad.to(torch.bfloat16).contiguous(), handle=handle)[0]
            with torch.enable_grad():
                out = rows * weights.unsqueeze(1).to(rows.dtype)
            grads = iter(torch.autograd.grad(out, [t for t, n in zip((rows, weights), need) if n], grad_rows, create_graph=again))
            return (None, *(next(grads) if n else None for n in need), None)
        plan = buffer._live_plan(handle)
        grad = _readable(grad.to(torch.bfloat16))
        out = torch.empty_like(rows) if need[0] else None
        grad_w = torch.empty_like(weights) if need[1] else None
        _launch("return_grad", rows, grad.data_ptr(), rows.data_ptr(), weights.data_ptr(), plan.slot_row.data_ptr(),
                0 if out is None else out.data_ptr(), 0 if grad_w is None else grad_w.data_ptr(), plan.num_tokens, plan.num_topk,
                *rows.shape, blocks=False)
        return None, out, grad_w, None


def _launch(op: str, like: torch.Tensor, *args, blocks: bool = True) -> None:
    """Launches a kernel on the current stream of the device of ``like``."""
    kernel, index = getattr(require_native("the training layer"), op), like.get_device()
    args += (_blocks(index),) if blocks else ()
    args += (torch._C._cuda_getCurrentRawStream(index),)
    if index == torch.cuda.current_device():
        kernel(*args)
    else:
        with torch.cuda.device(index):
            kernel(*args)


@lru_cache(maxsize=None)
def _blocks(index: int) -> int:
    return torch.cuda.get_device_properties(index).multi_processor_count * 8


def _readable(grad: torch.Tensor) -> torch.Tensor:
    """Contiguous and on a 16-byte boundary, as the kernels read it."""
    grad = grad.contiguous()
    return grad.clone() if grad.data_ptr() % 16 else grad


def _ordinary(*tensors: torch.Tensor) -> bool:
    """Tensors whose memory a kernel can read, in a call that nobody traces, batches or differentiates forward: a kernel behind
    an address is invisible to all of these."""
    if torch.compiler.is_compiling():                    # first: a compiler follows the rest of this function no further
        return False
    if torch._C._len_torch_dispatch_stack() or torch._C._are_functorch_transforms_active() or torch.jit.is_tracing():
        return False
    for t in tensors:
        if type(t) not in (torch.Tensor, torch.nn.Parameter) or torch._C._functorch.is_legacy_batchedtensor(t):
            return False
        if forward_ad._current_level >= 0 and forward_ad.unpack_dual(t).tangent is not None:
            return False
    return True


def _separate_operations(gate_up: torch.Tensor) -> torch.Tensor:
    gate, up = gate_up.chunk(2, dim=-1)
    return torch.nn.functional.silu(gate) * up


def _activate(gate_up: torch.Tensor) -> torch.Tensor:
    """``silu(gate) * up``.  The kernel takes bf16 rows that are contiguous, 16-byte aligned and a multiple of 8 values wide;
    anything else goes through torch, with the same results."""
    inter = gate_up.shape[1] // 2
    if (_ordinary(gate_up) and gate_up.is_cuda and gate_up.dtype == torch.bfloat16 and gate_up.is_contiguous() and inter % 8 == 0
            and inter > 0 and gate_up.data_ptr() % 16 == 0):
        return _Swiglu.apply(gate_up)
    return _separate_operations(gate_up)


def _weighable(rows: torch.Tensor, weights: torch.Tensor, dtype: torch.dtype) -> bool:
    """Contiguous, 16-byte aligned bf16 rows of a multiple of 8 values and fp32 weights of the same number, in an ordinary call."""
    return (_ordinary(rows, weights) and rows.is_cuda and rows.device == weights.device and rows.dtype == dtype == torch.bfloat16
            and weights.dtype == torch.float32 and rows.dim() == 2 and weights.shape == rows.shape[:1] and rows.numel() > 0
            and rows.shape[1] % 8 == 0 and rows.is_contiguous() and weights.is_contiguous() and rows.data_ptr() % 16 == 0)


def _weigh(rows: torch.Tensor, weights: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    """``rows`` times their weights rounded to ``dtype``, by a kernel where it takes them, else through torch with the same results."""
    return _WeighRows.apply(rows, weights) if _weighable(rows, weights, dtype) else rows * weights.unsqueeze(1).to(dtype)


def _weigh_and_combine(buffer: ElasticBuffer, rows: torch.Tensor, weights: torch.Tensor, handle, dtype: torch.dtype) -> torch.Tensor:
    weighs = getattr(buffer.engine, "weighs_rows", None)
    if weighs is not None and _weighable(rows, weights, dtype) and weighs(handle._plan, buffer.num_sms):
        return _WeighAndCombine.apply(buffer, rows, weights, handle)
    return _Combine.apply(buffer, _weigh(rows, weights, dtype).contiguous(), handle)


class ExpertParallelMoE(torch.nn.Module):
    """SwiGLU experts sharded over the ranks of ``buffer``; forward = dispatch -> local experts -> combine.

    ``w1 [L, 2I, H]`` holds gate rows then up rows, ``w2 [L, H, I]``; both bf16, Kaiming-uniform.
    The routing weight multiplies each expert output row before combine (whose reduction is unweighted).
    """

    def __init__(self, buffer: ElasticBuffer, num_experts: int, hidden: int, intermediate: int, device=None):
        super().__init__()
        self.buffer, self.num_experts = buffer, num_experts
        self.local = num_experts // buffer.world_size
        w1 = torch.empty((self.local, 2 * intermediate, hidden), dtype=torch.bfloat16, device=device)
        w2 = torch.empty((self.local, hidden, intermediate), dtype=torch.bfloat16, device=device)
        for w in (w1, w2):
            for e in range(self.local):
                torch.nn.init.kaiming_uniform_(w[e], a=5 ** 0.5)
        self.w1, self.w2 = torch.nn.Parameter(w1), torch.nn.Parameter(w2)
        self.use_grouped_mm = None        # decided at the first GPU forward (set it to False to force the per-expert loop)

    def experts(self, rows: torch.Tensor, psum: torch.Tensor, counts=None) -> torch.Tensor:
        """SwiGLU experts on expert-major rows.  On a GPU with a usable library grouped GEMM both projections are one
        ``torch._grouped_mm`` each (row ranges from the handle's cumulative counts, which stay on the device);
        otherwise a loop over the experts with the host-side counts of the handle (no device synchronisation)."""
        if rows.is_cuda and self.use_grouped_mm is None:
            from ..utils.grouped_mm import grouped_mm_usable

            self.use_grouped_mm = grouped_mm_usable()
        if rows.is_cuda and self.use_grouped_mm and rows.shape[0] > 0:
            offs = psum.to(torch.int32)
            gate_up = torch._grouped_mm(rows, self.w1.transpose(1, 2), offs=offs)
            return torch._grouped_mm(_activate(gate_up), self.w2.transpose(1, 2), offs=offs)
        bounds = [0]
        for c in (counts if counts is not None else torch.diff(psum, prepend=psum.new_zeros(1)).tolist()):
            bounds.append(bounds[-1] + int(c))
        outs = []
        for e in range(self.local):
            seg = rows[bounds[e]:bounds[e + 1]]
            gate, up = (seg @ self.w1[e].t()).chunk(2, dim=-1)
            outs.append((torch.nn.functional.silu(gate) * up) @ self.w2[e].t())
        return torch.cat(outs, dim=0) if outs else rows.new_zeros((0, self.w2.shape[1]))

    def forward(self, x: torch.Tensor, topk_idx: torch.Tensor, topk_weights: torch.Tensor) -> torch.Tensor:
        holder = {}
        recv_x, recv_w, psum = _Dispatch.apply(self.buffer, x, topk_idx, topk_weights, self.num_experts, holder)
        y = self.experts(recv_x, psum, holder["handle"].num_recv_tokens_per_expert_list)
        return _weigh_and_combine(self.buffer, y, recv_w, holder["handle"], recv_x.dtype)


__all__ = ["ExpertParallelMoE"]
