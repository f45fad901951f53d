"""Token embedding tied to the output projection, with a resident bf16 working copy.

A tied embedding matrix is read twice per step (row gather at the bottom of the network, the
vocabulary GEMM at the top) and receives two gradient contributions (the weight gradient of
that GEMM at the start of backward, a row scatter at its end).  Under plain autocast this costs
a cast + pad of the whole fp32 matrix every step, a dense zero matrix for the scatter and two
dense additions.  ``TiedEmbedding`` keeps a bf16 copy padded to a multiple of 128 rows (written
by the fused AdamW kernel together with the fp32 parameter, like ``MasterLinear``'s), gathers bf16
rows from it, and - when a gradient arena is attached (``weight._dq_grad_padded``, see
parallel/reducer.py) - lets the GEMM write the fp32 weight gradient straight into the arena and
the scatter add its rows on top, so no dense temporary is ever made.

The reference takes Hugging Face's tied embeddings as they are
(testbed_evaluation/train_llm_causal.py:490-497); the parameter seen by hooks, optimizer state and
checkpoints here is still the fp32 ``weight`` of shape [vocab, hidden].
"""
from __future__ import annotations

from typing import Optional

import torch
import torch.nn as nn
import torch.nn.functional as F

from . import require
from ..utils import counters

PAD_ROWS = 128


class _LookupFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, ids, weight, shadow):
        ctx.save_for_backward(ids)
        ctx.rows = weight.shape[0]
        ctx.direct = getattr(weight, "_dq_grad_padded", None)
        ctx.sparse = getattr(weight, "_dq_sparse", None)
        return F.embedding(ids, shadow)

    @staticmethod
    def backward(ctx, dy):
        (ids,) = ctx.saved_tensors
        if ctx.sparse is not None:
            # multi-rank runs: keep the token rows; the reducer exchanges them and adds every rank's rows
            # after the dense (output-projection) part of the gradient has been reduced
            ctx.sparse["ids"] = ids.reshape(-1)
            ctx.sparse["rows"] = dy.reshape(-1, dy.shape[-1]).contiguous()
            return None, None, None
        rows = dy.reshape(-1, dy.shape[-1]).float()
        if ctx.direct is not None:
            # the output projection's weight gradient was written earlier in this backward pass
            ctx.direct.index_add_(0, ids.reshape(-1), rows)
            return None, None, None
        dw = torch.zeros(ctx.rows, dy.shape[-1], dtype=torch.float32, device=dy.device)
        dw.index_add_(0, ids.reshape(-1), rows)
        return None, dw, None


class _HeadFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, h, weight, shadow):
        ctx.save_for_backward(h, shadow)
        ctx.rows = weight.shape[0]
        ctx.direct = getattr(weight, "_dq_grad_padded", None)
        return h.reshape(-1, h.shape[-1]) @ shadow.t()

    @staticmethod
    def backward(ctx, dy):
        h, shadow = ctx.saved_tensors
        h2 = h.reshape(-1, h.shape[-1])
        dh = (dy @ shadow).reshape(h.shape) if ctx.needs_input_grad[0] else None
        if ctx.direct is not None:
            torch.mm(dy.t(), h2, out_dtype=torch.float32, out=ctx.direct)  # overwrites: first contribution
            return dh, None, None
        dw = torch.mm(dy.t(), h2, out_dtype=torch.float32)[: ctx.rows]
        return dh, dw, None


class _EmbedFn(torch.autograd.Function):
    """bf16(token row + position row [+ type row 0]) in one kernel; see csrc/kernels/embedding_ops.cu."""

    @staticmethod
    def forward(ctx, ids, weight, shadow, pos, typ):
        ctx.save_for_backward(ids)
        ctx.shapes = (weight.shape, None if pos is None else pos.shape, None if typ is None else typ.shape)
        ctx.direct = getattr(weight, "_dq_grad_padded", None)
        ctx.sparse = getattr(weight, "_dq_sparse", None)
        counters.add("embed_fwd")
        return require().embed_fwd(ids, shadow, pos, typ)

    @staticmethod
    def backward(ctx, dx):
        (ids,) = ctx.saved_tensors
        tok, pos, typ = ctx.shapes
        dx = dx.contiguous()
        dw = None
        if ctx.sparse is not None:
            ctx.sparse["ids"], ctx.sparse["rows"] = ids.reshape(-1), dx.view(-1, dx.shape[-1])
            target = None
        elif ctx.direct is not None:
            target = ctx.direct  # holds the output projection's weight gradient, written earlier in this backward pass
        else:
            target = dw = torch.zeros(tok, dtype=torch.float32, device=dx.device)
        dpos = None if pos is None else torch.empty(pos, dtype=torch.float32, device=dx.device)
        if target is not None or dpos is not None:
            require().embed_bwd(dx, ids, target, dpos)
            counters.add("embed_bwd")
        dtyp = None
        if typ is not None:
            dtyp = torch.zeros(typ, dtype=torch.float32, device=dx.device)
            require().colsum(dx.view(-1, dx.shape[-1]), dtyp[0])
            counters.add("colsum", 2)
        return None, dw, None, dpos, dtyp


class _HeadLossFn(torch.autograd.Function):
    """Mean cross-entropy of h W^T (+ bias) with the gradient of the logits written over them in the same pass
    (csrc/kernels/loss_fused.cu): the logits exist only between this node's two halves."""

    @staticmethod
    def forward(ctx, h, weight, shadow, bias, low_bias, labels, vocab: int, ignore_index: int, shift: bool):
        h2 = h.reshape(-1, h.shape[-1])
        logits = F.linear(h2, shadow, low_bias)
        loss, sums = require().ce_fused(logits, labels.contiguous(), vocab, ignore_index, shift, bias is not None)
        counters.add("ce_fused", 3 if bias is None else 4)
        ctx.save_for_backward(h, shadow, logits, sums)
        ctx.rows, ctx.has_bias = weight.shape[0], bias is not None
        ctx.direct = getattr(weight, "_dq_grad_padded", None)
        return loss

    @staticmethod
    def backward(ctx, g):
        h, shadow, dlogits, sums = ctx.saved_tensors
        g = g.to(torch.float32).reshape(1)
        require().ce_rescale_(dlogits, g)
        counters.add("ce_rescale")
        h2 = h.reshape(-1, h.shape[-1])
        dh = (dlogits @ shadow).view(h.shape) if ctx.needs_input_grad[0] else None
        dw = None
        if ctx.direct is not None:
            torch.mm(dlogits.t(), h2, out_dtype=torch.float32, out=ctx.direct)  # overwrites: first contribution
        else:
            dw = torch.mm(dlogits.t(), h2, out_dtype=torch.float32)[: ctx.rows]
        db = sums[: ctx.rows] * g if ctx.has_bias else None
        return dh, dw, None, db, None, None, None, None, None


class TiedEmbedding(nn.Embedding):
    """``nn.Embedding`` whose weight also serves as the output projection.

    ``lookup(ids)`` returns rows (bf16 from the working copy when it exists, else the parameter's
    dtype); ``logits(h)`` returns ``h @ W^T`` as [N, Vp] with the vocabulary padded to a multiple of
    128 (columns >= ``num_embeddings`` are zero weights; pair with ``fused_cross_entropy``).
    """

    def __init__(self, num_embeddings: int, embedding_dim: int):
        super().__init__(num_embeddings, embedding_dim)
        self.padded_rows = (num_embeddings + PAD_ROWS - 1) // PAD_ROWS * PAD_ROWS
        self.shadow: Optional[torch.Tensor] = None
        # a gradient arena reserves this many elements so that the padded GEMM can write in place
        self.weight._dq_padded_shape = (self.padded_rows, embedding_dim)

    def enable_shadow(self) -> torch.Tensor:
        w = self.weight
        w._dq_padded_shape = (self.padded_rows, self.embedding_dim)
        if self.shadow is None or self.shadow.device != w.device:
            self.shadow = torch.zeros(self.padded_rows, self.embedding_dim, dtype=torch.bfloat16, device=w.device)
        with torch.no_grad():
            self.shadow[: self.num_embeddings].copy_(w)
        return self.shadow

    def _use_shadow(self, device_type: str) -> bool:
        return self.shadow is not None and device_type == "cuda" and torch.is_autocast_enabled("cuda") \
            and torch.get_autocast_dtype("cuda") == torch.bfloat16

    def lookup(self, ids: torch.Tensor) -> torch.Tensor:
        if self._use_shadow(ids.device.type):
            return _LookupFn.apply(ids, self.weight, self.shadow)
        return F.embedding(ids, self.weight)

    def forward(self, ids: torch.Tensor) -> torch.Tensor:
        return self.lookup(ids)

    def embed(self, ids: torch.Tensor, pos: Optional[torch.Tensor] = None, typ: Optional[torch.Tensor] = None
              ) -> Optional[torch.Tensor]:
        """bf16 rows of `ids` [B, S] plus the first S rows of `pos` plus row 0 of `typ`, or None where the fused kernel
        does not apply (no bf16 working copy in use)."""
        if not self._use_shadow(ids.device.type) or self.embedding_dim % 8 != 0 or ids.dim() != 2 or ids.dtype != torch.int64:
            return None
        return _EmbedFn.apply(ids.contiguous(), self.weight, self.shadow, pos, typ)

    def loss(self, h: torch.Tensor, labels: torch.Tensor, bias: Optional[torch.Tensor] = None, shift: bool = False,
             ignore_index: int = -100) -> torch.Tensor:
        """Mean cross-entropy of ``logits(h, bias)`` against `labels` [B, S]; `shift`: position t predicts t + 1."""
        from .layers import fused_cross_entropy, shift_labels

        fused = self._use_shadow(h.device.type) and h.dtype == torch.bfloat16 and torch.is_grad_enabled() \
            and h.requires_grad and labels.dtype == torch.int64 and require().ce_fused_fits(self.padded_rows)
        if not fused:
            if shift:
                labels = shift_labels(labels)
            return fused_cross_entropy(self.logits(h, bias), labels.reshape(-1), self.num_embeddings, ignore_index)
        low = None
        if bias is not None:
            low = torch.zeros(self.padded_rows, dtype=torch.bfloat16, device=h.device)
            low[: self.num_embeddings].copy_(bias.detach())
        return _HeadLossFn.apply(h, self.weight, self.shadow, bias, low, labels, self.num_embeddings, ignore_index, shift)

    def logits(self, h: torch.Tensor, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
        if self._use_shadow(h.device.type) and h.dtype == torch.bfloat16:
            out = _HeadFn.apply(h, self.weight, self.shadow)
            if bias is not None:
                out = out + F.pad(bias.to(out.dtype), (0, self.padded_rows - self.num_embeddings))
            return out
        from .layers import padded_vocab_logits

        return padded_vocab_logits(h, self.weight, bias, PAD_ROWS)
