"""GPT-2 decoder (LayerNorm, learned positions, GELU MLP, tied input/output embedding).

Parameter names follow Hugging Face ``GPT2LMHeadModel``.  HF stores the projections as ``Conv1D``
(``[in, out]``); here they are ``[out, in]`` linears and :func:`from_hf_state_dict` transposes on load.
The vocabulary is padded to a multiple of 64 rows so that logits rows stay 16-byte aligned for TMA.

Reference counterpart: packages/opaque-patches/src/opaque/api/patches/transformers/models/gpt2.py
(the reference only batchifies and disables the KV cache for this family).
"""
from __future__ import annotations

import dataclasses

import torch
from torch import nn

from .. import ops
from ..engine import blocks, fused
from ..functional import functional_checkpoint
from .layers import _FORWARDS, Embedding, LayerNorm, Linear, linear_cross_entropy, passable, per_example_token_weights


@dataclasses.dataclass
class GPT2Config:
    vocab_size: int = 50257
    n_positions: int = 1024
    n_embd: int = 768
    n_layer: int = 12
    n_head: int = 12
    layer_norm_epsilon: float = 1e-5

    @property
    def padded_vocab(self) -> int:
        return (self.vocab_size + 63) // 64 * 64

    @staticmethod
    def small() -> "GPT2Config":
        return GPT2Config()

    @staticmethod
    def tiny() -> "GPT2Config":
        return GPT2Config(vocab_size=500, n_positions=256, n_embd=128, n_layer=2, n_head=4)


class _SplitHeads(torch.autograd.Function):
    """``[B, T, 3·d]`` → three ``[B, heads, T, d/heads]`` views; the backward writes the three gradients into ONE
    buffer (one gather kernel) instead of three zero-filled full-size tensors that are then added."""

    @staticmethod
    def forward(ctx, qkv, heads):
        B, T, d3 = qkv.shape
        v5 = qkv.view(B, T, 3, heads, d3 // (3 * heads))
        ctx.shape = (B, T, 3, heads, d3 // (3 * heads))
        return tuple(v5[:, :, i].transpose(1, 2) for i in range(3))

    @staticmethod
    def backward(ctx, gq, gk, gv):
        return ops.merge_heads3(gq, gk, gv), None


class GPT2Block(nn.Module):
    def __init__(self, cfg: GPT2Config, dtype, device):
        super().__init__()
        d = cfg.n_embd
        self.nh = cfg.n_head
        self.ln_1 = LayerNorm(d, cfg.layer_norm_epsilon, dtype=dtype, device=device)
        self.attn_c_attn = Linear(d, 3 * d, bias=True, dtype=dtype, device=device)
        self.attn_c_proj = Linear(d, d, bias=True, dtype=dtype, device=device)
        self.ln_2 = LayerNorm(d, cfg.layer_norm_epsilon, dtype=dtype, device=device)
        self.mlp_c_fc = Linear(d, 4 * d, bias=True, dtype=dtype, device=device)
        self.mlp_c_proj = Linear(4 * d, d, bias=True, dtype=dtype, device=device)

    def forward(self, h):
        h = h + self._attention(self.ln_1(h))
        return h + self._mlp(self.ln_2(h))

    def forward_carried(self, x, residual):
        """The block on a split stream ``h = x + residual`` (``residual`` may be ``None``): every residual addition happens inside
        the next LayerNorm's kernel, and the two gradient branches meet in that kernel's backward.  Returns the pair."""
        if blocks.one_stream(x, residual) and self._two_nodes(x):
            m, n1, n2 = self._modules, self.ln_1, self.ln_2
            wq, wo, w1, w2 = (m[k]._parameters for k in _PROJECTIONS)
            q, k, v, s = blocks.GPT2In.apply(x, residual, n1.weight, n1.bias, wq["weight"], wq["bias"], n1.eps, self.nh, n1)
            o = nn.functional.scaled_dot_product_attention(q, k, v, is_causal=True)
            return blocks.GPT2Out.apply(o, x if s is None else s, wo["weight"], wo["bias"], n2.weight, n2.bias, w1["weight"], w1["bias"],
                                        w2["weight"], w2["bias"], n2.eps, n2, torch.is_grad_enabled())
        y, s = (self.ln_1(x), x) if residual is None else self.ln_1.add(x, residual)
        y, s = self.ln_2.add(self._attention(y), s)
        return self._mlp(y), s

    def _two_nodes(self, x) -> bool:
        """Whether the block may run as two autograd nodes around the attention (``engine/blocks.py``): plain projections with biases on
        the library's products, and its parameters all frozen, or all trained under a capture."""
        if type(self)._attention is not _BLOCK_PARTS[0] or type(self)._mlp is not _BLOCK_PARTS[1] or "_attention" in self.__dict__ \
                or "_mlp" in self.__dict__ or not blocks.available():
            return False
        m = self._modules
        linears = [m[k] for k in _PROJECTIONS]
        if not passable(*linears, m["ln_1"], m["ln_2"]):
            return False
        trained = linears[0].weight.requires_grad
        if trained and fused.current_capture() is None:
            return False
        for lin in linears:
            w, b = lin._parameters.get("weight"), lin._parameters.get("bias")          # None: no parameter of the module
            if lin.lora_A is not None or w is None or b is None or w.requires_grad != trained or b.requires_grad != trained \
                    or not fused._own_gemm_ok(x, w, b):
                return False
        for norm in (m["ln_1"], m["ln_2"]):
            w, b = norm._parameters.get("weight"), norm._parameters.get("bias")
            if w is None or b is None or w.requires_grad != trained or b.requires_grad != trained or w.dtype != torch.bfloat16 or b.dtype != torch.bfloat16:
                return False
        return x.shape[-1] % 8 == 0 and x.shape[-1] <= 1024

    def _mlp(self, y):
        return self.mlp_c_proj(ops.activation(self.mlp_c_fc(y), "gelu_tanh"))

    def _attention(self, y):
        B, T, d = y.shape
        qkv = self.attn_c_attn(y)
        if qkv.is_cuda and ops.functional.kernels_enabled():
            q, k, v = _SplitHeads.apply(qkv, self.nh)
        else:                                    # plain views (also what runs under vmap in the reference engine)
            v5 = qkv.view(B, T, 3, self.nh, d // self.nh)
            q, k, v = (v5[:, :, i].transpose(1, 2) for i in range(3))
        o = nn.functional.scaled_dot_product_attention(q, k, v, is_causal=True)
        return self.attn_c_proj(o.transpose(1, 2).reshape(B, T, d))


_FORWARDS[GPT2Block] = GPT2Block.forward
_BLOCK_PARTS = GPT2Block._attention, GPT2Block._mlp
_PROJECTIONS = ("attn_c_attn", "attn_c_proj", "mlp_c_fc", "mlp_c_proj")


class GPT2LMHeadModel(nn.Module):
    def __init__(self, cfg: GPT2Config, *, dtype=torch.bfloat16, device=None):
        super().__init__()
        self.config = cfg
        self.wte = Embedding(cfg.padded_vocab, cfg.n_embd, dtype=dtype, device=device)
        self.wpe = Embedding(cfg.n_positions, cfg.n_embd, dtype=dtype, device=device)
        self.h = nn.ModuleList(GPT2Block(cfg, dtype, device) for _ in range(cfg.n_layer))
        self.ln_f = LayerNorm(cfg.n_embd, cfg.layer_norm_epsilon, dtype=dtype, device=device)
        self.activation_checkpointing = False      # set by the trainer's gradient_checkpointing

    def _carries(self) -> bool:
        """Whether the blocks may run on the split stream, which calls neither a block's nor most norms' ``forward``: blocks and norms of
        these very classes with their own ``forward`` (none assigned to an instance or patched into the class, none compiled), and no
        hooks, on them or on all modules, that expect to be called with the unsplit tensors."""
        return all(type(blk) is GPT2Block and type(blk.ln_1) is LayerNorm and type(blk.ln_2) is LayerNorm for blk in self.h) \
            and type(self.ln_f) is LayerNorm and passable(self.ln_f, *(m for blk in self.h for m in (blk, blk.ln_1, blk.ln_2)))

    def hidden_states(self, input_ids):
        B, T = input_ids.shape
        pos = torch.arange(T, device=input_ids.device).expand(B, T)
        h = self.wte(input_ids) + self.wpe(pos)
        if h.is_cuda and ops.functional.kernels_enabled() and not (getattr(self, "activation_checkpointing", False) and torch.is_grad_enabled()) \
                and self._carries():
            x, residual = h, None
            for blk in self.h:
                x, residual = blk.forward_carried(x, residual)
            return self.ln_f(x) if residual is None else self.ln_f.add(x, residual)[0]
        for blk in self.h:
            if getattr(self, "activation_checkpointing", False) and torch.is_grad_enabled():
                h = (torch.utils.checkpoint.checkpoint(blk, h, use_reentrant=False) if ops.functional.kernels_enabled()
                     else functional_checkpoint(blk, h))          # torch.func transforms need the functional form
            else:
                h = blk(h)
        return self.ln_f(h)

    def forward(self, input_ids):
        return self.hidden_states(input_ids) @ self.wte.weight.t()

    def token_nll(self, input_ids, labels):
        """Per-token negative log-likelihood ``[N, T]`` (0 where ignored)."""
        from .llama import _token_nll
        return _token_nll(self, self.wte.weight, input_ids, labels)

    def per_example_loss(self, input_ids, labels):
        B, T = input_ids.shape
        h = self.hidden_states(input_ids).reshape(B * T, -1)
        w = per_example_token_weights(labels).reshape(-1)
        rows = linear_cross_entropy(h, self.wte.weight, labels.reshape(-1), w)
        return rows.view(B, T).sum(1)


def from_hf_state_dict(sd: dict) -> dict:
    """Map a Hugging Face GPT-2 state dict onto this module's names (transposing ``Conv1D`` weights)."""
    out = {}
    for k, v in sd.items():
        k = k.removeprefix("transformer.")
        if k == "lm_head.weight":
            continue
        k = k.replace("attn.c_attn", "attn_c_attn").replace("attn.c_proj", "attn_c_proj")
        k = k.replace("mlp.c_fc", "mlp_c_fc").replace("mlp.c_proj", "mlp_c_proj")
        if k.endswith(".weight") and any(t in k for t in ("attn_c_attn", "attn_c_proj", "mlp_c_fc", "mlp_c_proj")):
            v = v.t().contiguous()
        out[k] = v
    return out
