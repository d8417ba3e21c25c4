"""Token embedding whose gradient is added to the owner's fp32 gradient buffer (csrc/elementwise.cu).

A parameter of the flat engine (one that has a unit and a `main_grad`) gets its embedding gradient there, row by row of the tokens
that occur, as the GEMM and norm epilogues do for theirs; everything else is `torch.nn.Embedding`: owners that wait for autograd's
accumulation hooks, weights with hooks, gradients that are asked for as results or differentiated again, transforms.  The dense gradient of 3003 tokens in a tied 32064 x 2048 matrix, its conversion and its addition
took 480 us, this 70.
"""
from __future__ import annotations

import torch

from . import _lib


def _takes(w: torch.Tensor) -> bool:
    g = getattr(w, "main_grad", None)
    return (g is not None and getattr(w, "_ts_unit", None) is not None and g.dtype == torch.float32 and w.is_cuda
            and w.dtype == torch.bfloat16 and g.is_cuda and g.is_contiguous() and g.shape == w.shape and w.shape[1] % 8 == 0
            and g.data_ptr() % 16 == 0 and not w._backward_hooks and not w._post_accumulate_grad_hooks)


def _accumulates(w: torch.Tensor) -> bool | None:
    """Whether the running backward pass accumulates the gradient of leaf `w`: None where it is asked for as a result
    (`torch.autograd.grad`), False where it is not asked for at all."""
    try:
        return torch._C._will_engine_execute_node(torch.autograd.graph.get_gradient_edge(w).node)
    except RuntimeError:
        return None


def add_rows(grad: torch.Tensor, ids: torch.Tensor, dy: torch.Tensor) -> None:
    """grad [V, H] fp32 += dy [T, H] bf16 at rows ids [T]; sums in the order of the tokens."""
    lib = _lib.load("elementwise")
    T, H = dy.shape
    values, order = ids.to(torch.int32).sort(stable=True)
    part = torch.empty(lib.ts_embedding_bwd_parts(T), H, dtype=torch.float32, device=dy.device)
    rc = lib.ts_embedding_bwd(_lib.ptr(dy), _lib.ptr(values), _lib.ptr(order), _lib.ptr(grad), _lib.ptr(part), T, H, _lib.stream_ptr())
    _lib.check(rc, "ts_embedding_bwd")


class _EmbeddingFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, ids, w):
        ctx.save_for_backward(ids)
        ctx.weight = w                       # whose values the gradient does not need: they may change before it is formed
        return torch.nn.functional.embedding(ids, w)

    @staticmethod
    def backward(ctx, dy):
        (ids,), w = ctx.saved_tensors, ctx.weight
        wanted = _accumulates(w)
        if wanted is False:
            return None, None
        flat, d2 = ids.reshape(-1), dy.reshape(-1, w.shape[1])
        # (with grad mode on, the gradient will be differentiated itself)
        if wanted is None or torch.is_grad_enabled() or not (_takes(w) and dy.dtype == torch.bfloat16 and d2.shape[0] > 0):
            return None, torch.ops.aten.embedding_dense_backward(dy, ids, w.shape[0], -1, False)
        d2 = d2 if d2.is_contiguous() and d2.data_ptr() % 16 == 0 else d2.clone(memory_format=torch.contiguous_format)
        grad = w.main_grad
        if not getattr(w, "grad_added", False):
            grad.zero_()
            w.grad_added = True
        add_rows(grad, flat, d2)
        return None, None


class TokenEmbedding(torch.nn.Embedding):
    def forward(self, ids: torch.Tensor) -> torch.Tensor:
        w = self.weight
        if (torch.is_grad_enabled() and w.requires_grad and _takes(w) and self.padding_idx is None and self.max_norm is None
                and not self.scale_grad_by_freq and not self.sparse and not ids.is_floating_point()
                and not torch._C._are_functorch_transforms_active() and torch.autograd.forward_ad._current_level < 0):
            return _EmbeddingFn.apply(ids, w)
        return super().forward(ids)
