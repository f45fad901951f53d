"""Sub-layers of a transformer block as single autograd nodes around the fused kernels.

What a block's GEMMs and attention leave between them - residual additions, biases and their gradients, activations,
rotary embedding, packing of the attention gradients - is memory traffic; here it rides in as few passes as the data
flow allows:

* :func:`add_norm` adds a sub-layer's output (and its bias) to the residual stream and normalises it; backward adds the
  stream's gradient and takes the bias gradient on the way (csrc/kernels/residual_norm.cu);
* :func:`mlp` and :func:`attention` leave the bias of their last linear layer to the ``add_norm`` that follows; the
  GELU kernels carry the first layer's bias (csrc/kernels/activation_ops.cu), the packing of dq / dk / dv the
  projection's (csrc/kernels/attention_ops.cu).

Used for bf16 activations on CUDA when the linear layers hold bf16 working copies (ops/linear.py); parameter gradients
go to the gradient arena when one is attached, as in that module.  The block modules (models/) fall back to the plain
composition everywhere else.
"""
from __future__ import annotations

from typing import Optional

import torch
import torch.nn.functional as F

from . import require
from ..utils import counters


def fusable(x: torch.Tensor, *linears) -> bool:
    """Whether the fused sub-layers take this input and these linear layers."""
    return (x.is_cuda and x.dtype == torch.bfloat16 and x.shape[-1] % 8 == 0 and x.shape[-1] <= 2048
            and all(m.shadow is not None and m.out_features % 8 == 0 for m in linears))


def _arena(p) -> Optional[torch.Tensor]:
    return getattr(p, "_dq_grad", None) if p is not None else None


def _weight_grad(dy2: torch.Tensor, x2: torch.Tensor, out: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    """dy^T x in fp32, into the arena view when there is one (autograd then sees None)."""
    if out is not None:
        torch.mm(dy2.t(), x2, out_dtype=torch.float32, out=out)
        return None
    return torch.mm(dy2.t(), x2, out_dtype=torch.float32)


class _AddNormFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, delta, bias, w, b, eps: float, rms: bool, post: bool):
        s, y, mean, rstd = require().add_norm_fwd(x.contiguous(), None if delta is None else delta.contiguous(), bias, w, b,
                                                  eps, rms)
        counters.add("add_norm_fwd")
        ctx.set_materialize_grads(False)
        ctx.save_for_backward(s, w, mean, rstd)
        ctx.rms, ctx.post, ctx.has_delta, ctx.has_bias = rms, post, delta is not None, bias is not None and delta is not None
        ctx.wg, ctx.bg, ctx.biasg = _arena(w), _arena(b), _arena(bias)
        return (y, y.view_as(y)) if post else (x.view_as(x) if delta is None else s, y)

    @staticmethod
    def backward(ctx, g0, g1):
        s, w, mean, rstd = ctx.saved_tensors
        dy, dy2, ds = (g0, g1, None) if ctx.post else (g1, None, g0)
        if dy is None:
            dy, dy2 = (dy2, None) if dy2 is not None else (torch.zeros_like(s), None)
        dx, dw, db, dbias = require().add_norm_bwd(
            dy.contiguous(), None if dy2 is None else dy2.contiguous(), None if ds is None else ds.contiguous(), s, w, mean, rstd,
            ctx.rms, ctx.has_bias, ctx.wg, ctx.bg, ctx.biasg)
        counters.add("add_norm_bwd", 2)
        return (dx, dx if ctx.has_delta else None, dbias if ctx.has_bias and ctx.biasg is None else None,
                dw if ctx.wg is None else None, db if not ctx.rms and ctx.bg is None else None, None, None, None)


def add_norm(norm, x: torch.Tensor, delta: Optional[torch.Tensor] = None, bias: Optional[torch.Tensor] = None,
             post: bool = False):
    """s = x + (delta + bias) and y = norm(s), for a LayerNorm / RMSNorm module.  Returns (s, y); with `post` (the sum
    has no other reader) y twice: give one to the next sub-layer and one to the next residual addition, so that
    backward gets their gradients apart and adds them in its own pass."""
    b = getattr(norm, "bias", None)
    return _AddNormFn.apply(x, delta, bias, norm.weight.float(), None if b is None else b.float(), norm.eps, b is None, post)


class _ResidualAddFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, delta, bias):
        counters.add("residual_add")
        ctx.has_bias, ctx.biasg = bias is not None, _arena(bias)
        return require().residual_add(x.contiguous(), delta.contiguous(), bias)

    @staticmethod
    def backward(ctx, ds):
        db = None
        if ctx.has_bias:
            db = require().colsum(ds.reshape(-1, ds.shape[-1]).contiguous(), ctx.biasg)
            counters.add("colsum", 2)
        return ds, ds, db if ctx.biasg is None else None


def residual_add(x: torch.Tensor, delta: torch.Tensor, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """x + (delta + bias): the sum of :func:`add_norm` where no norm follows in the same call."""
    return _ResidualAddFn.apply(x, delta, bias)


class _MlpFn(torch.autograd.Function):
    """act(x W1^T + b1) W2^T (+ b2), act = GELU."""

    @staticmethod
    def forward(ctx, x, w1, s1, b1, w2, s2, b2, b2_low, tanh_form: bool):
        pre = F.linear(x, s1)
        act = require().gelu_fwd(pre, b1, tanh_form)
        counters.add("gelu_fwd")
        ctx.save_for_backward(x, pre, act, s1, s2, b1)
        ctx.tanh, ctx.has_b2 = tanh_form, b2 is not None
        ctx.arena = (_arena(w1), _arena(b1), _arena(w2), _arena(b2))
        return F.linear(act, s2, b2_low)

    @staticmethod
    def backward(ctx, dy):
        x, pre, act, s1, s2, b1 = ctx.saved_tensors
        g1, gb1, g2, gb2 = ctx.arena
        dy2 = dy.reshape(-1, dy.shape[-1])
        dw2 = _weight_grad(dy2, act.reshape(-1, act.shape[-1]), g2)
        dact = (dy2 @ s2).view_as(pre)
        dpre, db1 = require().gelu_bwd(dact, pre, b1, ctx.tanh, gb1)
        counters.add("gelu_bwd", 1 if b1 is None else 2)
        dpre2 = dpre.view(-1, dpre.shape[-1])
        dw1 = _weight_grad(dpre2, x.reshape(-1, x.shape[-1]), g1)
        dx = (dpre2 @ s1).view_as(x) if ctx.needs_input_grad[0] else None
        db2 = None
        if ctx.has_b2:
            db2 = require().colsum(dy2.contiguous(), gb2)
            counters.add("colsum", 2)
        return (dx, dw1, None, db1 if b1 is not None and gb1 is None else None, dw2, None,
                db2 if gb2 is None else None, None, None)


def mlp(x: torch.Tensor, fc, proj, tanh_form: bool, with_bias: bool) -> torch.Tensor:
    """proj(gelu(fc(x))) for two MasterLinear layers; without `with_bias` the bias of `proj` is left to the caller."""
    use = with_bias and proj.bias is not None
    return _MlpFn.apply(x, fc.weight, fc.shadow, fc.bias, proj.weight, proj.shadow, proj.bias if use else None,
                        proj.low_bias() if use else None, tanh_form)


class _AttentionFn(torch.autograd.Function):
    """proj(attention(qkv(x))), the attention core being the library's; rotary embedding in place on the packed qkv."""

    @staticmethod
    def forward(ctx, x, w1, s1, b1, b1_low, w2, s2, b2, b2_low, cos, sin, nh: int, nkv: int, causal: bool, grad: bool):
        B, S, _ = x.shape
        D = s2.shape[1] // nh
        qkv = F.linear(x, s1, b1_low)
        if cos is not None:
            require().rope_qkv_(qkv, cos, sin, nh, nkv, D)
            counters.add("rope_qkv")
        heads = qkv.view(B, S, nh + 2 * nkv, D).transpose(1, 2)
        q, k, v = heads[:, :nh], heads[:, nh: nh + nkv], heads[:, nh + nkv:]
        with torch.set_grad_enabled(grad):
            if grad:
                q, k, v = (t.detach().requires_grad_() for t in (q, k, v))
            core = F.scaled_dot_product_attention(q, k, v, is_causal=causal, enable_gqa=nkv != nh)
        o = core.detach().transpose(1, 2).reshape(B, S, nh * D)
        ctx.save_for_backward(x, o, s1, s2, cos, sin)
        ctx.core, ctx.inputs = (core, (q, k, v)) if grad else (None, None)
        ctx.has_b1, ctx.has_b2 = b1 is not None, b2 is not None
        ctx.arena = (_arena(w1), _arena(b1), _arena(w2), _arena(b2))
        return F.linear(o, s2, b2_low)

    @staticmethod
    def backward(ctx, dy):
        x, o, s1, s2, cos, sin = ctx.saved_tensors
        g1, gb1, g2, gb2 = ctx.arena
        core, inputs = ctx.core, ctx.inputs
        ctx.core = ctx.inputs = None
        B, nh, S, D = core.shape
        dy2 = dy.reshape(-1, dy.shape[-1])
        dw2 = _weight_grad(dy2, o.view(-1, o.shape[-1]), g2)
        do = (dy2 @ s2).view(B, S, nh, D).transpose(1, 2)
        dq, dk, dv = (t if t.stride(-1) == 1 else t.contiguous() for t in torch.autograd.grad(core, inputs, do))
        del core, inputs
        dqkv, db1 = require().qkv_grad_pack(dq, dk, dv, cos, sin, ctx.has_b1, gb1)
        counters.add("qkv_grad_pack", 2 if ctx.has_b1 else 1)
        dqkv = dqkv.view(-1, dqkv.shape[-1])
        dw1 = _weight_grad(dqkv, x.reshape(-1, x.shape[-1]), g1)
        dx = (dqkv @ s1).view_as(x) if ctx.needs_input_grad[0] else None
        db2 = None
        if ctx.has_b2:
            db2 = require().colsum(dy2.contiguous(), gb2)
            counters.add("colsum", 2)
        return (dx, dw1, None, db1 if ctx.has_b1 and gb1 is None else None, None, dw2, None,
                db2 if gb2 is None else None, None, None, None, None, None, None, None)


def attention(x: torch.Tensor, qkv, proj, nh: int, nkv: int, causal: bool, cos, sin, with_bias: bool) -> torch.Tensor:
    """proj(attention(qkv(x))); without `with_bias` the bias of `proj` is left to the caller.  cos / sin: rotary tables
    (then `qkv` has no bias) or None."""
    use = with_bias and proj.bias is not None
    return _AttentionFn.apply(x, qkv.weight, qkv.shadow, qkv.bias, qkv.low_bias(), proj.weight, proj.shadow,
                              proj.bias if use else None, proj.low_bias() if use else None, cos, sin, nh, nkv, causal,
                              torch.is_grad_enabled())
