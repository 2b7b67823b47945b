"""Decoder blocks as two autograd nodes (engine/blocks.py) against the same blocks with one node per operation."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(model, batch, mode, unsplit):
    """Losses, gradients and the number of nodes taken; ``unsplit``: a hook on one projection of every block forbids the two nodes."""
    from opaque_b200.engine import blocks
    from opaque_b200.engine.fused import FusedDPEngine
    from opaque_b200.random import key
    hooks = []
    if unsplit:
        layers = model.h if hasattr(model, "h") else model.model.layers
        hooks = [(blk.mlp_c_fc if hasattr(blk, "mlp_c_fc") else blk.mlp.down_proj).register_forward_hook(lambda *a: None) for blk in layers]
    taken, apply = [], {}
    for cls in (blocks.GPT2In, blocks.GPT2Out, blocks.LoRAIn, blocks.LoRAOut):
        apply[cls] = cls.forward
        cls.forward = staticmethod(lambda ctx, *a, f=cls.forward: (taken.append(1), f(ctx, *a))[1])
    try:
        if mode == "capture":
            eng = FusedDPEngine(model, clipping_norm=1.0, noise_multiplier=0.0, normalize_by=2.0, key=key(0), microbatch_size=batch["labels"].shape[0])
            res = eng.accumulate(model.per_example_loss, batch)
            out = [res.losses, res.norms, eng.space.grad.local.clone()]
        elif mode == "autograd":                       # without a capture: gradients of the adapters through torch's engine
            params = [p for p in model.parameters() if p.requires_grad]
            nll = model.token_nll(**batch)
            out = [nll.detach(), *torch.autograd.grad(nll.sum(), params)]
        else:
            with torch.no_grad():
                out = [model.token_nll(**batch)]
    finally:
        for cls, f in apply.items():
            cls.forward = staticmethod(f)
        for h in hooks:
            h.remove()
    return out, len(taken)


def _close(a, b):
    # the same kernels on the same operands; norms and gradients add fp32 values with atomics, and two runs of the library's attention
    # backward round single values differently (2^-8)
    for i, (x, y) in enumerate(zip(a, b)):
        assert torch.equal(x, y) if i == 0 else float((x.float() - y.float()).norm()) <= 2e-3 * float(y.float().norm()) + 1e-12


@pytest.mark.parametrize("B,T", [(1, 1), (2, 64), (3, 77), (17, 250)])          # the last: norm sums in the norms' backward
@pytest.mark.parametrize("mode", ["capture", "none"])
def test_gpt2(B, T, mode):
    from opaque_b200.models import GPT2Config, GPT2LMHeadModel, shift_labels
    torch.manual_seed(T)
    model = GPT2LMHeadModel(GPT2Config.tiny(), device="cuda").requires_grad_(mode == "capture")
    for n, p in model.named_parameters():
        if n.endswith("bias"):
            torch.nn.init.normal_(p, std=0.1)
    ids = torch.randint(0, 500, (B, T), device="cuda")
    batch = {"input_ids": ids, "labels": shift_labels(ids)}
    one, n1 = _run(model, batch, mode, False)
    two, n2 = _run(model, batch, mode, True)
    assert (n1, n2) == (4, 0)
    _close(one, two)


@pytest.mark.parametrize("B,T,r", [(1, 1, 8), (2, 64, 16), (3, 77, 8)])
@pytest.mark.parametrize("mode", ["capture", "autograd", "none"])
def test_llama_lora(B, T, r, mode):
    from opaque_b200.models import LlamaConfig, LlamaForCausalLM, shift_labels
    torch.manual_seed(T)
    model = LlamaForCausalLM(LlamaConfig.tiny(), device="cuda")
    model.add_lora(r, 2.0 * r)
    for n, p in model.named_parameters():
        if n.endswith("lora_B"):
            torch.nn.init.normal_(p, std=0.05)
    ids = torch.randint(0, 256, (B, T), device="cuda")
    batch = {"input_ids": ids, "labels": shift_labels(ids)}
    one, n1 = _run(model, batch, mode, False)
    two, n2 = _run(model, batch, mode, True)
    assert (n1, n2) == (4, 0)
    _close(one, two)


@pytest.mark.parametrize("B,T,Hq,Hk,D", [(1, 1, 1, 1, 16), (2, 77, 4, 2, 32), (3, 130, 8, 8, 64), (2, 300, 6, 3, 128)])
def test_rotary_gradients_into_one_buffer(B, T, Hq, Hk, D):
    """q, k rotated back and v copied, from [B, heads, T, D] and from [B, T, heads, D] storage: the bits of the rotation and a concatenation."""
    import ctypes
    from opaque_b200 import ops
    from opaque_b200.ops import lib
    torch.manual_seed(T)
    cos, sin = ops.rope_tables(D, 512, 10000.0, device="cuda")
    q, k, v = (torch.randn(B, T, h, D, device="cuda", dtype=torch.bfloat16) for h in (Hq, Hk, Hk))
    v = v.transpose(1, 2).contiguous().transpose(1, 2)
    out = torch.empty(B * T, (Hq + 2 * Hk) * D, device="cuda", dtype=torch.bfloat16)
    strides = (ctypes.c_longlong * 9)(*(t.stride(d) for t in (q, k, v) for d in range(3)))
    lib.check(lib.load().ob_rope_qkv_gather(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), cos.data_ptr(), sin.data_ptr(),
                                            ctypes.addressof(strides), B * T, T, Hq, Hk, D, 1, lib.sm_count(), lib.stream()), "rope_qkv_gather")
    qr, kr = ops.functional._RoPE._run(q, k, cos, sin, None, 1)
    assert torch.equal(out, torch.cat([t.reshape(B * T, -1) for t in (qr, kr, v)], 1))


def test_without_the_compiled_sequences(monkeypatch):
    """Where the extension is missing, blocks run node by node and the factor gradients go through the general batch entry point."""
    from opaque_b200 import ops
    from opaque_b200.models import LlamaConfig, LlamaForCausalLM, shift_labels
    torch.manual_seed(0)
    model = LlamaForCausalLM(LlamaConfig.tiny(), device="cuda")
    model.add_lora(8, 16.0)
    ids = torch.randint(0, 256, (2, 64), device="cuda")
    batch = {"input_ids": ids, "labels": shift_labels(ids)}
    one, n1 = _run(model, batch, "capture", False)
    monkeypatch.setattr(ops, "block_steps", lambda: None)
    two, n2 = _run(model, batch, "capture", False)
    assert (n1, n2) == (4, 0)
    _close(one, two)


@pytest.mark.parametrize("B,T", [(3, 77), (2, 256), (19, 250)])           # ragged and uniform weight gradients, sums apart and in the norms
def test_packed_batches(B, T, monkeypatch):
    """Norms, sums and weight gradients whose problems are packed by the extension or in Python."""
    from opaque_b200 import ops
    from opaque_b200.models import GPT2Config, GPT2LMHeadModel, shift_labels
    torch.manual_seed(T)
    model = GPT2LMHeadModel(GPT2Config.tiny(), device="cuda")
    ids = torch.randint(0, 500, (B, T), device="cuda")
    batch = {"input_ids": ids, "labels": shift_labels(ids)}
    one, _ = _run(model, batch, "capture", True)
    monkeypatch.setattr(ops, "block_steps", lambda: None)
    two, _ = _run(model, batch, "capture", True)
    _close(one, two)


def test_batches_that_python_looks_at():
    """Problems that the packers decline raise what they raised."""
    from opaque_b200 import ops
    a, out = torch.randn(64, 128, device="cuda", dtype=torch.bfloat16), torch.zeros(128 * 128, device="cuda")
    steps = ops.block_steps()
    assert steps.wgrad_batch([dict(a=a, b=a, out_offset=1)], out, None, 0, 0) is False and steps.ghost_batch([(a, a.float(), out, 8, None, None, None)], 0) is False
    with pytest.raises(ValueError):
        ops.wgrad_clip_batch([dict(a=a, b=a, out_offset=1)], out)
    with pytest.raises(TypeError):
        ops.ghost_norm_batch([(a, a.float(), out, 8, None, None, None)])
    with pytest.raises(ValueError):
        ops.wgrad_clip_per_example_batch([(a, a, None, 0, 128)], out, 63)
    with pytest.raises(ValueError):
        ops.functional.rows_sum_batch_([(out.view(128, 128)[:7], a)], 8)
    assert float(out.abs().max()) == 0.0
    ops.wgrad_clip_batch([dict(a=a, b=a)], out)
    ref = a.double().t() @ a.double()
    assert float((out.view(128, 128) - ref).norm()) <= 2 ** -20 * float(ref.norm())


def test_errors_of_the_compiled_sequences():
    """Refused arguments and failed launches are Python exceptions."""
    from opaque_b200 import ops
    from opaque_b200.ops import lib
    steps = ops.block_steps()
    x = torch.randn(4, 128, device="cuda", dtype=torch.bfloat16)
    out, seg = torch.zeros(2, 64, device="cuda"), torch.tensor([0, 2, 4], dtype=torch.int32, device="cuda")
    with pytest.raises(TypeError):
        steps.gpt2_in(x, None, 3)
    with pytest.raises(ValueError):                      # past the end of the destination
        steps.store_wgrads(((x, x, 0, 128, 1, 128),), out, seg, 2, 64, 0)
    w = torch.ones(132, device="cuda", dtype=torch.bfloat16)[:124]
    with pytest.raises(lib.KernelLibraryError):          # a width that is no multiple of 8: refused by the kernel's entry point
        steps.gpt2_in(x[:, :124].contiguous(), None, w, w, x, w, 1e-5)


def test_blocks_that_keep_one_node_per_operation():
    """Partly frozen or partly adapted blocks, another class's projection and given positions."""
    from opaque_b200.models import GPT2Config, GPT2LMHeadModel, Linear, LlamaConfig, LlamaForCausalLM
    x = torch.randn(1, 8, 128, device="cuda", dtype=torch.bfloat16)
    gpt = GPT2LMHeadModel(GPT2Config.tiny(), device="cuda").requires_grad_(False)
    assert gpt.h[0]._two_nodes(x)
    gpt.h[0].mlp_c_fc.bias.requires_grad_(True)
    assert not gpt.h[0]._two_nodes(x) and gpt.h[1]._two_nodes(x) and not gpt.h[1]._two_nodes(x.float())

    class Other(Linear):
        pass
    model = LlamaForCausalLM(LlamaConfig.tiny(), device="cuda")
    assert not model.model.layers[0]._two_nodes(x, model.rope_cos, model.rope_sin, None)
    model.add_lora(8, 16.0)
    a, b = model.model.layers
    assert a._two_nodes(x, model.rope_cos, model.rope_sin, None) and not a._two_nodes(x, model.rope_cos, model.rope_sin, torch.arange(8, device="cuda")[None])
    a.self_attn.o_proj.__class__ = Other
    b.mlp.gate_proj.add_lora(8, 16.0)
    assert not a._two_nodes(x, model.rope_cos, model.rope_sin, None) and not b._two_nodes(x, model.rope_cos, model.rope_sin, None)


def test_gradient_of_the_residual_alone():
    """A frozen block whose ``x`` asks for no gradient while its residual does: the residual's is what it is with both."""
    from opaque_b200.models import GPT2Config, GPT2LMHeadModel
    torch.manual_seed(0)
    block = GPT2LMHeadModel(GPT2Config.tiny(), device="cuda").requires_grad_(False).h[0]
    x, r, gm, gs = (torch.randn(2, 64, 128, device="cuda", dtype=torch.bfloat16) for _ in range(4))
    assert block._two_nodes(x)
    grads = []
    for both in (False, True):
        rr = r.clone().requires_grad_(True)
        m, s = block.forward_carried(x.clone().requires_grad_(both), rr)
        torch.autograd.backward((m, s), (gm, gs))
        grads.append(rr.grad)
    _close([m, grads[0]], [m, grads[1]])


def _smaller(module, name, *shape):
    p = getattr(module, name)
    setattr(module, name, torch.nn.Parameter(torch.zeros(*shape, device="cuda", dtype=torch.bfloat16), requires_grad=p.requires_grad))


def test_operands_that_do_not_fit_together():
    """A parameter of another size is a ``ValueError`` of the product or norm that meets it, in a block that runs as two nodes."""
    from opaque_b200.models import GPT2Config, GPT2LMHeadModel, LlamaConfig, LlamaForCausalLM
    x = torch.randn(1, 8, 128, device="cuda", dtype=torch.bfloat16)
    for path, name, shape in (("attn_c_attn", "weight", (384, 64)), ("attn_c_attn", "bias", (376,)), ("attn_c_proj", "weight", (128, 64)),
                              ("mlp_c_fc", "weight", (512, 64)), ("mlp_c_fc", "bias", (504,)), ("mlp_c_proj", "weight", (128, 448)),
                              ("mlp_c_proj", "weight", (120, 512)), ("ln_1", "weight", (120,)), ("ln_1", "bias", (120,)), ("ln_2", "bias", (8,))):
        block = GPT2LMHeadModel(GPT2Config.tiny(), device="cuda").requires_grad_(False).h[0]
        _smaller(getattr(block, path), name, *shape)
        assert block._two_nodes(x)
        with pytest.raises(ValueError):
            block.forward_carried(x, x)
    for path, name, shape in (("self_attn.q_proj", "lora_A", (8, 64)), ("self_attn.k_proj", "lora_A", (8, 64)), ("self_attn.v_proj", "lora_B", (64, 16)),
                              ("self_attn.o_proj", "lora_A", (8, 64)), ("self_attn.o_proj", "lora_B", (128, 16)), ("self_attn.o_proj", "weight", (128, 64)),
                              ("input_layernorm", "weight", (64,)), ("post_attention_layernorm", "weight", (64,))):
        model = LlamaForCausalLM(LlamaConfig.tiny(), device="cuda")
        model.add_lora(8, 16.0)
        layer = model.model.layers[0]
        _smaller(layer.get_submodule(path), name, *shape)
        args = (model.rope_cos, model.rope_sin, None)
        assert layer._two_nodes(x, *args)
        with pytest.raises(ValueError):
            layer.forward_carried(x, x, *args)


def test_streams_of_two_kinds_keep_one_node_per_operation():
    """A residual of another type or of a shape that only broadcasts is added as it was before blocks ran as two nodes."""
    from opaque_b200.models import GPT2Config, GPT2LMHeadModel, LlamaConfig, LlamaForCausalLM
    torch.manual_seed(0)
    x = torch.randn(2, 8, 128, device="cuda", dtype=torch.bfloat16)
    block = GPT2LMHeadModel(GPT2Config.tiny(), device="cuda").requires_grad_(False).h[0]
    model = LlamaForCausalLM(LlamaConfig.tiny(), device="cuda")
    model.add_lora(8, 16.0)
    with torch.no_grad():
        r = torch.randn(1, 8, 128, device="cuda", dtype=torch.bfloat16)
        got, want = block.forward_carried(x, r), block.forward_carried(x, r.expand(2, 8, 128).contiguous())
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
        args = (model.rope_cos, model.rope_sin, None)
        got, want = model.model.layers[0].forward_carried(x, x.float(), *args), model.model.layers[0].forward_carried(x, x.clone(), *args)
        assert torch.equal(got[1], want[1]) and float((got[0] - want[0]).norm()) <= 2 ** -8 * float(want[0].norm())


def test_allocations_that_fail():
    """A sequence that finds no memory raises what torch's allocations raise, and the next call works."""
    from opaque_b200 import ops
    steps, kept = ops.block_steps(), []
    x, w = torch.zeros(1 << 18, 128, device="cuda", dtype=torch.bfloat16), torch.ones(128, device="cuda", dtype=torch.bfloat16)
    proj = torch.zeros(128, 128, device="cuda", dtype=torch.bfloat16)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    # results of 64 MB each, in what is left of the blocks that this process holds
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + 1) / torch.cuda.get_device_properties(0).total_memory)
    try:
        with pytest.raises(torch.OutOfMemoryError):
            for _ in range(32):
                kept.append(steps.gpt2_in(x, None, w, w, proj, w, 1e-5))
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert steps.gpt2_in(x, None, w, w, proj, w, 1e-5)[3].shape == x.shape


@pytest.mark.parametrize("family", ["gpt2", "llama"])
def test_memory_kept_for_the_backward_pass(family):
    """A block with frozen weights keeps no more as two nodes than with one node per operation."""
    from opaque_b200.models import GPT2Config, GPT2LMHeadModel, LlamaConfig, LlamaForCausalLM
    if family == "gpt2":
        block, args = GPT2LMHeadModel(GPT2Config.tiny(), device="cuda").requires_grad_(False).h[0], ()
        part = block.mlp_c_fc
    else:
        model = LlamaForCausalLM(LlamaConfig.tiny(), device="cuda")
        model.add_lora(8, 16.0)
        block, args = model.model.layers[0], (model.rope_cos, model.rope_sin, None)
        part = block.mlp.down_proj
    held = []
    for unsplit in (False, True):
        hook = part.register_forward_hook(lambda *a: None) if unsplit else None
        x, r = (torch.randn(2, 64, 128, device="cuda", dtype=torch.bfloat16, requires_grad=True) for _ in range(2))
        kept = {}
        with torch.autograd.graph.saved_tensors_hooks(lambda t: kept.setdefault(t.untyped_storage().data_ptr(), t), lambda t: t):
            out = block.forward_carried(x, r, *args)
        held.append(sum(t.untyped_storage().nbytes() for t in kept.values()))
        del out
        if hook is not None:
            hook.remove()
    assert held[0] <= held[1]


def test_pitches_and_groups_that_are_refused():
    """A negative pitch is no pitch left out, and no group is no problem: refused by the packer and by the Python form alike."""
    from opaque_b200 import ops
    a, out = torch.ones(64, 128, device="cuda", dtype=torch.bfloat16), torch.zeros(128 * 128, device="cuda")
    for bad, error in ((dict(ldm=-1), ValueError), (dict(num_groups=0), (ValueError, ZeroDivisionError))):
        assert ops.block_steps().wgrad_batch([dict(a=a, b=a, **bad)], out, None, 0, 0) is False
        with pytest.raises(error):
            ops.wgrad_clip_batch([dict(a=a, b=a, **bad)], out)
    assert float(out.abs().max()) == 0.0


def test_sequences_longer_than_the_rotary_tables():
    from opaque_b200.models import LlamaConfig, LlamaForCausalLM
    model = LlamaForCausalLM(LlamaConfig.tiny(), device="cuda")
    ids = torch.zeros(1, 257, dtype=torch.int64, device="cuda")
    for adapters in (False, True):                       # one node per operation, and two nodes
        if adapters:
            model.add_lora(8, 16.0)
        with torch.no_grad(), pytest.raises(ValueError):
            model.token_nll(ids, ids)
        model.token_nll(ids[:, :256], ids[:, :256])


def _attention(q, k, v, is_causal=True, enable_gqa=False, scale=None):
    """Attention whose backward pass gives the same bits every time (the library's varies)."""
    B, H, T, hd = q.shape
    if enable_gqa:
        k, v = (t[:, :, None].expand(B, t.shape[1], H // t.shape[1], T, hd).reshape(B, H, T, hd) for t in (k, v))
    s = (q @ k.transpose(2, 3)).float() * (hd ** -0.5 if scale is None else scale)
    s = s.masked_fill(torch.ones(T, T, dtype=torch.bool, device=q.device).triu(1), float("-inf"))
    return torch.softmax(s, -1).to(v.dtype) @ v


@pytest.mark.parametrize("family,B,T", [("gpt2", 2, 64), ("gpt2", 3, 77), ("gpt2", 17, 250), ("llama", 2, 64), ("llama", 3, 77)])
def test_same_operands_and_every_gradient(family, B, T, monkeypatch):
    """With an attention that repeats its bits: what a pass hands to the capture is equal bit for bit, in the same order, and the gradient of
    every parameter by itself differs by no more than the order of its fp32 sums.

    The sums' terms are the same; a value of n terms moves by at most sqrt(n) 2^-24 of their size (n up to 4250 rows), and ten times that
    allows for the terms that cancel."""
    from opaque_b200.engine.fused import Capture, FusedDPEngine
    from opaque_b200.models import GPT2Config, GPT2LMHeadModel, LlamaConfig, LlamaForCausalLM, shift_labels
    from opaque_b200.random import key
    monkeypatch.setattr(torch.nn.functional, "scaled_dot_product_attention", _attention)
    handed, results = [], []                             # per run: (method, its operands without the parameters)
    for name in ("add_linear", "add_embedding", "add_lora", "add_lora_qkv"):
        def spy(self, *a, f=getattr(Capture, name), name=name):
            flat = [t for x in a for t in (x if isinstance(x, (tuple, list)) else (x,)) if isinstance(t, torch.Tensor) and not isinstance(t, torch.nn.Parameter)]
            handed[-1].append((name, [t.clone() for t in flat]))
            return f(self, *a)
        monkeypatch.setattr(Capture, name, spy)
    for unsplit in (False, True):
        handed.append([])
        torch.manual_seed(T)
        model = (GPT2LMHeadModel(GPT2Config.tiny(), device="cuda") if family == "gpt2" else LlamaForCausalLM(LlamaConfig.tiny(), device="cuda"))
        if family == "llama":
            model.add_lora(8, 16.0)
        for n, p in model.named_parameters():
            if n.endswith(("bias", "lora_B")):
                torch.nn.init.normal_(p, std=0.1)
        for blk in (model.h if family == "gpt2" else model.model.layers) if unsplit else ():
            (blk.mlp_c_fc if family == "gpt2" else blk.mlp.down_proj).register_forward_hook(lambda *a: None)
        eng = FusedDPEngine(model, clipping_norm=1.0, noise_multiplier=0.0, normalize_by=2.0, key=key(0), microbatch_size=B)
        ids = torch.randint(0, 256, (B, T), device="cuda")
        res = eng.accumulate(model.per_example_loss, {"input_ids": ids, "labels": shift_labels(ids)})
        results.append((res, {n: eng.space.grad.local[s.offset:s.offset + s.numel].clone() for n, s in eng.space.slots.items()}))
    two, one = handed
    assert [n for n, _ in two] == [n for n, _ in one] and len(two) >= 4
    for (name, a), (_, b) in zip(two, one):
        assert len(a) == len(b) and all(torch.equal(x, y) for x, y in zip(a, b)), name
    assert torch.equal(results[0][0].losses, results[1][0].losses)
    for name, g in results[0][1].items():
        ref = results[1][1][name]
        assert float((g - ref).norm()) <= 10 * (B * T) ** 0.5 * 2 ** -24 * float(ref.norm()), (name, float((g - ref).norm() / ref.norm()))


@pytest.mark.parametrize("family", ["gpt2", "llama"])
@pytest.mark.parametrize("carried", [False, True])
def test_gradients_through_frozen_weights_bit_for_bit(family, carried, monkeypatch):
    """Data gradients of a block, and the factors' without a capture, with fixed incoming gradients and a repeatable attention."""
    from opaque_b200.models import GPT2Config, GPT2LMHeadModel, LlamaConfig, LlamaForCausalLM
    monkeypatch.setattr(torch.nn.functional, "scaled_dot_product_attention", _attention)
    torch.manual_seed(0)
    model = (GPT2LMHeadModel(GPT2Config.tiny(), device="cuda").requires_grad_(False) if family == "gpt2" else LlamaForCausalLM(LlamaConfig.tiny(), device="cuda"))
    if family == "llama":
        model.add_lora(8, 16.0)
    for n, p in model.named_parameters():
        if n.endswith(("bias", "lora_B")):
            torch.nn.init.normal_(p, std=0.1)
    block, args = (model.h[0], ()) if family == "gpt2" else (model.model.layers[0], (model.rope_cos, model.rope_sin, None))
    x, r, gm, gs = (torch.randn(3, 77, 128, device="cuda", dtype=torch.bfloat16) for _ in range(4))
    results = []
    for unsplit in (False, True):
        hook = (block.mlp_c_fc if family == "gpt2" else block.mlp.down_proj).register_forward_hook(lambda *a: None) if unsplit else None
        xx, rr = x.clone().requires_grad_(True), (r.clone().requires_grad_(True) if carried else None)
        out = block.forward_carried(xx, rr, *args)
        inputs = [xx] + ([rr] if carried else []) + [p for p in block.parameters() if p.requires_grad]
        results.append([*out, *torch.autograd.grad(out, inputs, (gm, gs))])
        if hook is not None:
            hook.remove()
    assert len(results[0]) >= 3
    for a, b in zip(*results):
        assert torch.equal(a, b)
