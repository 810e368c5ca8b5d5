"""Embedding lookup whose gradient goes straight into the sharded engine's flat gradient buffer."""
from __future__ import annotations

import torch
import torch.nn.functional as F

from .. import _lib

MAX_POSITIONS = 8192  # of zc_embedding_grad


class _Embedding(torch.autograd.Function):
    """The table is kept by reference, as the linear layers keep their weights: under the sharded engines its storage is
    released after forward, and backward only writes ``weight.main_grad``."""

    @staticmethod
    def forward(ctx, ids, weight):
        ctx.save_for_backward(ids)
        ctx.weight = weight
        ctx.shape = tuple(weight.shape)
        return F.embedding(ids, weight)

    @staticmethod
    def backward(ctx, dout):
        (ids,) = ctx.saved_tensors
        w, (rows, dim) = ctx.weight, ctx.shape
        mg = getattr(w, "main_grad", None)
        n = ids.numel()
        if (mg is not None and mg.dtype == torch.bfloat16 and mg.is_contiguous() and tuple(mg.shape) == (rows, dim)
                and mg.data_ptr() % 16 == 0 and dout.dtype == torch.bfloat16 and dim % 8 == 0 and 0 < n <= MAX_POSITIONS
                and ids.dtype == torch.int64 and not w._backward_hooks
                and not getattr(w, "_post_accumulate_grad_hooks", None)):
            ids, dout = ids.reshape(-1).contiguous(), dout.reshape(n, dim).contiguous()
            if dout.data_ptr() % 16:
                dout = dout.clone()
            _lib.check(_lib.cuda().zc_embedding_grad(ids.data_ptr(), dout.data_ptr(), mg.data_ptr(), n, dim, rows,
                                                     int(bool(w.main_grad_written)), _lib.stream_ptr(dout.device)),
                       "zc_embedding_grad")
            w.main_grad_written = True
            return None, None
        return None, torch.ops.aten.embedding_dense_backward(dout, ids, rows, -1, False)


def embedding(ids: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    """``weight[ids]``; a table that a sharded engine manages (it has ``main_grad``) gets its gradient there."""
    if weight.is_cuda and weight.requires_grad and hasattr(weight, "main_grad") and torch.is_grad_enabled():
        return _Embedding.apply(ids, weight)
    return F.embedding(ids, weight)
