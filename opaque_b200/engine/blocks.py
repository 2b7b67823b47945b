"""Whole sub-layers of the standard decoder blocks as autograd nodes.

A block written as one node per operation spends 25 us of host time per launch (module calls, argument checks of every product, an
autograd node and its views), more than most launches of a short batch take.  Here a block is two nodes around the library's
attention, :class:`GPT2In` / :class:`GPT2Out` and :class:`LoRAIn` / :class:`LoRAOut`, and each node's launches are one call of the
compiled sequences (``ops/csrc/block_steps.cpp``).  The same kernels in the same order on the same operands as the single nodes, so the
same bits; which blocks may run this way is the models' decision (``models/gpt2.py``, ``models/llama.py``), and it needs
:func:`available`.

Measured on one B200, per pass, single nodes / these: GPT-2 small 11 x 333 tokens forward and backward 10.2 / 7.1 ms (its kernels take
5.5), 5 x 257 tokens forward 3.4 / 2.1 ms (1.0); Llama-1B with LoRA, step of 2 x 128 tokens, 15.3 / 9.2 ms (5.2).
"""
from __future__ import annotations

from torch.autograd import Function

from .. import ops
from ..ops.functional import _layer_norm_param_grads
from . import fused


def available() -> bool:
    """Whether the compiled sequences are there and the products choose their kernel by themselves."""
    return ops.PAIR_GEMM and ops.block_steps() is not None


def one_stream(x, residual) -> bool:
    """Whether the two parts of a split stream are of one kind; a node's kernels read both the same way."""
    return residual is None or (residual.dtype is x.dtype and residual.is_cuda and residual.is_same_size(x))


def _weight_grads(cap, weight, bias, x2d, g2d):
    """A trained linear's gradients: to the capture (returns ``(None, None)``), or summed where no capture is active."""
    if cap is None:
        return g2d.t() @ x2d, g2d.sum(0)
    cap.add_linear(weight, x2d, g2d)
    cap.sum_jobs.append((cap.pe_view(bias), g2d))
    return None, None


def _norm_sums(trainable, norm, rows):
    """Where the backward kernel of a trained LayerNorm adds its per-example gradients (weight, bias), or ``(None, None)`` where they are
    summed apart: no capture; few rows, whose sums share a launch with the other layers'; or fewer examples than one per 256 columns.

    The kernel has at most 16 blocks per example (each is one more rounding of the example's sum), which for few long examples is too few
    for the chip, the sooner the wider the rows (us, apart / by the kernel: 8192 rows of 768 as 1, 2 and 4 examples 55 / 84, 36 / 45 and
    27 / 25, of 1024 65 / 124, 45 / 66 and 35 / 36; of 512 as 1 and 2 51 / 58 and 32 / 32; of 256 as 1 45 / 41)."""
    cap = fused.current_capture() if trainable else None
    if cap is None or cap.sums_wait(rows, norm.weight.shape[0]) or rows % cap.batch_size or norm.weight.shape[0] > 256 * cap.batch_size:
        return None, None
    return cap.pe_view(norm.weight), cap.pe_view(norm.bias)


class GPT2In(Function):
    """``s = x + residual``, its LayerNorm and the query / key / value projection: ``(q, k, v, s)`` with heads ``[B, heads, T, hd]``.
    Without ``residual`` the last output is ``None``: the stream goes on from ``x``."""

    @staticmethod
    def forward(ctx, x, residual, ln_w, ln_b, w, b, eps, heads, norm):
        B, T, d = x.shape
        y, s, stats, qkv = ops.block_steps().gpt2_in(x, residual, ln_w, ln_b, w, b, eps)
        ctx.trainable, ctx.norm, ctx.linear, ctx.carried = w.requires_grad, norm, (w, b), residual is not None
        ctx.save_for_backward(s, stats, ln_w, w, *((y,) if ctx.trainable else ()))
        q, k, v = qkv.view(B, T, 3, heads, d // heads).permute(2, 0, 3, 1, 4).unbind(0)
        return q, k, v, None if residual is None else s.view(x.shape)

    @staticmethod
    def backward(ctx, dq, dk, dv, ds):
        s, stats, ln_w, w, *trained = ctx.saved_tensors
        sums = _norm_sums(ctx.trainable, ctx.norm, s.shape[0])
        g, dy, dx = ops.block_steps().gpt2_in_bwd(dq, dk, dv, w, s, ln_w, stats, ds if ctx.carried else None,
                                                  ctx.needs_input_grad[0] or ctx.needs_input_grad[1] or ctx.trainable, *sums)
        dln = dlb = dw = db = None
        if ctx.trainable:
            dw, db = _weight_grads(fused.current_capture(), *ctx.linear, *trained, g)
            if sums[0] is None:
                dln, dlb = _layer_norm_param_grads(dy, s, ln_w, stats, ctx.norm, True)
        if dx is not None:
            dx = dx.view(dq.shape[0], dq.shape[2], -1)
        return dx, (dx if ctx.carried else None), dln, dlb, dw, db, None, None, None


class GPT2Out(Function):
    """From the attention's output ``o [B, heads, T, hd]``: its projection, ``s = residual + that``, LayerNorm and the GELU MLP.
    Returns ``(mlp output, s)``; ``keep``: a backward pass may follow."""

    @staticmethod
    def forward(ctx, o, residual, wo, bo, ln_w, ln_b, w1, b1, w2, b2, eps, norm, keep):
        o2, y, s, stats, f, h, m = ops.block_steps().gpt2_out(o, residual, wo, bo, ln_w, ln_b, w1, b1, w2, b2, eps, keep)
        ctx.trainable, ctx.norm, ctx.linears, ctx.dims = w1.requires_grad, norm, ((wo, bo), (w1, b1), (w2, b2)), (o.shape[0], o.shape[2], o.shape[1], o.shape[3])
        if keep:
            ctx.save_for_backward(s, stats, f, ln_w, wo, w1, w2, *((o2, y, h) if ctx.trainable else ()))
        return m.view(residual.shape), s.view(residual.shape)

    @staticmethod
    def backward(ctx, dm, ds):
        s, stats, f, ln_w, wo, w1, w2, *trained = ctx.saved_tensors
        sums = _norm_sums(ctx.trainable, ctx.norm, s.shape[0])
        g2, g1, dy, dx, do = ops.block_steps().gpt2_out_bwd(dm, f, w2, w1, s, ln_w, stats, ds, wo, *sums)
        grads = (None,) * 8
        if ctx.trainable:
            o2, y, h = trained
            cap, (lo, l1, l2) = fused.current_capture(), ctx.linears
            d2 = _weight_grads(cap, *l2, h, g2)
            d1 = _weight_grads(cap, *l1, y, g1)
            dln = _layer_norm_param_grads(dy, s, ln_w, stats, ctx.norm, True) if sums[0] is None else (None, None)
            grads = (*_weight_grads(cap, *lo, o2, dx), *dln, *d1, *d2)
        return (do.view(ctx.dims).transpose(1, 2), dx.view(dm.shape), *grads, None, None, None)


class LoRAIn(Function):
    """``s = x + residual``, its RMSNorm (frozen weight), the grouped LoRA projections of query, key and value (:class:`fused._LoRAQKV`)
    and the rotary embedding: ``(q, k, v, s)`` with heads ``[B, heads, T, hd]``.  Without ``residual`` the last output is ``None``."""

    @staticmethod
    def forward(ctx, x, residual, norm_w, w_all, aq, bq, ak, bk, av, bv, cos, sin, scaling, norm, heads):
        B, T, d = x.shape
        nh, nkv, hd = heads
        y, s, rstd, a_cat, b_block, xa, q, k, qkv = ops.block_steps().lora_in(x, residual, norm_w, *norm, aq, bq, ak, bk, av, bv, scaling, w_all,
                                                                              cos, sin, nh, nkv, hd)
        ctx.save_for_backward(s, rstd, norm_w, y, xa, w_all, a_cat, b_block, aq, bq, ak, bk, av, bv, cos, sin)
        ctx.scaling, ctx.offset, ctx.carried, ctx.dims = scaling, norm[1], residual is not None, (B, T, d, nh, nkv, hd)
        ctx.factors = (aq, bq), (ak, bk), (av, bv)
        v = qkv.view(B, T, nh + 2 * nkv, hd).narrow(2, nh + nkv, nkv)
        return q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), None if residual is None else s.view(B, T, d)

    @staticmethod
    def backward(ctx, dq, dk, dv, ds):
        s, rstd, norm_w, y, xa, w_all, a_cat, b_block, aq, bq, ak, bk, av, bv, cos, sin = ctx.saved_tensors
        B, T, d, nh, nkv, hd = ctx.dims
        g, q_all, dx = ops.block_steps().lora_in_bwd(dq, dk, dv, cos, sin, b_block, ctx.scaling, w_all, a_cat, s, norm_w, rstd,
                                                     ds if ctx.carried else None, ctx.offset, ctx.needs_input_grad[0] or ctx.needs_input_grad[1])
        parts = g.split((nh * hd, nkv * hd, nkv * hd), 1)
        cap = fused.current_capture()
        grads = (None,) * 6
        if cap is not None:
            cap.add_lora_qkv(ctx.factors, y, xa, parts, q_all)
        else:
            r = aq.shape[0]
            grads = [t for j in range(3) for t in (q_all[:, j * r:(j + 1) * r].t() @ y, parts[j].t() @ xa[:, j * r:(j + 1) * r])]
        if dx is not None:
            dx = dx.view(B, T, d)
        return (dx, dx if ctx.carried else None, None, None, *grads, None, None, None, None, None)


class LoRAOut(Function):
    """From the attention's output ``o [B, heads, T, hd]``: its LoRA projection, ``s = residual + that``, RMSNorm and the gated MLP
    (both frozen).  Returns ``(mlp output, s)``; ``keep``: a backward pass may follow."""

    @staticmethod
    def forward(ctx, o, residual, wo, a, b, norm_w, w_gate, w_up, w_down, scaling, norm, act, keep):
        o2, xa, s, rstd, g, u, m = ops.block_steps().lora_out(o, a, scaling, wo, b, residual, norm_w, *norm, w_gate, w_up, ops._GLU_ACT[act],
                                                              w_down, keep)
        if keep:
            ctx.save_for_backward(s, rstd, norm_w, o2, xa, wo, a, b, g, u, w_gate, w_up, w_down)
            ctx.scaling, ctx.offset, ctx.act, ctx.dims = scaling, norm[1], act, (o.shape[0], o.shape[2], o.shape[1], o.shape[3])
            ctx.factors = a, b
        return m.view(residual.shape), s.view(residual.shape)

    @staticmethod
    def backward(ctx, dm, ds):
        s, rstd, norm_w, o2, xa, wo, a, b, g, u, w_gate, w_up, w_down = ctx.saved_tensors
        dx, q, do = ops.block_steps().lora_out_bwd(dm, w_down, g, u, ops._GLU_ACT[ctx.act], ops.pick_glu_bwd(*g.shape, ops.lib.sm_count()), w_gate,
                                                   w_up, s, norm_w, rstd, ds, ctx.offset, b, ctx.scaling, wo, a)
        cap = fused.current_capture()
        da = db = None
        if cap is not None:
            cap.add_lora(*ctx.factors, o2, xa, dx, q)
        else:
            da, db = q.t() @ o2, dx.t() @ xa
        return do.view(ctx.dims).transpose(1, 2), dx.view(dm.shape), None, da, db, None, None, None, None, None, None, None, None
