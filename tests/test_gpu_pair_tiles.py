"""The two tiles of the pair GEMM give the same bits, and the forms that take the small one alone equal fp32 references."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one row, the edges of the 256- and 512-row tiles, of the 256-column tile and of the six stages; ragged everything
@pytest.mark.parametrize("M,N,K", [(1, 8, 64), (255, 256, 384), (257, 264, 448), (511, 520, 72), (513, 1032, 2048), (1300, 2304, 768)])
@pytest.mark.parametrize("layout", ["nk", "kn"])
def test_tiles_agree_bit_for_bit(M, N, K, layout):
    from opaque_b200 import ops
    torch.manual_seed(M)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(*((N, K) if layout == "nk" else (K, N)), device="cuda", dtype=torch.bfloat16)
    a2, b2 = torch.randn(M, 16, device="cuda", dtype=torch.bfloat16), torch.randn(N, 16, device="cuda", dtype=torch.bfloat16)
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    kw = dict(b_layout=layout, a2=a2, b2=b2, bias=bias)
    small = ops.gemm_pair(a, b, tile="256x256", **kw)
    assert torch.equal(small, ops.gemm_pair(a, b, tile="512x256", **kw)) and torch.equal(small, ops.gemm_pair(a, b, **kw))
    assert torch.equal(small, ops.gemm(a, b, kernel="single", **kw))
    with pytest.raises(ValueError):
        ops.gemm_pair(a, b, tile="128x256", **kw)


@pytest.mark.parametrize("M,inter,K", [(1, 64, 64), (255, 128, 448), (257, 136, 384), (600, 1000, 1032)])
@pytest.mark.parametrize("act", ["silu", "gelu", "gelu_tanh"])
def test_gated_up_projection(M, inter, K, act):
    from opaque_b200 import ops
    torch.manual_seed(M)
    x, wg, wu = (torch.randn(*s, device="cuda", dtype=torch.bfloat16) / K ** 0.25 for s in ((M, K), (inter, K), (inter, K)))
    h, g, u = ops.gemm_glu(x, wg, wu, act=act)
    only, _, _ = ops.gemm_glu(x, wg, wu, act=act, save_preact=False)
    assert torch.equal(h, only)
    # the pre-activations are rounded sums, so they equal a plain product's; h is formed from them in fp32 and rounded once more
    # (2^-9), with the approximate exponential's few units of 2^-21 beside it
    assert torch.equal(g, ops.gemm_pair(x, wg)) and torch.equal(u, ops.gemm_pair(x, wu))
    f = torch.nn.functional.silu(g.float()) if act == "silu" else torch.nn.functional.gelu(g.float(), approximate="tanh" if act == "gelu_tanh" else "none")
    ref = f * u.float()
    assert float((h.float() - ref).norm() / ref.norm()) < 3e-3


@pytest.mark.parametrize("M,V,K", [(1, 40, 64), (255, 257, 448), (257, 512, 72), (700, 1111, 768)])
@pytest.mark.parametrize("softcap", [0.0, 5.0])
def test_head_statistics(M, V, K, softcap):
    from opaque_b200 import ops
    torch.manual_seed(M)
    h, w = (torch.randn(*s, device="cuda", dtype=torch.bfloat16) / K ** 0.25 for s in ((M, K), (V, K)))
    lab = torch.randint(0, V, (M,), device="cuda")
    lab[0] = -100
    z = (h.double() @ w.double().t()).float()
    if softcap:
        z = softcap * torch.tanh(z / softcap)
    for store in (False, True):
        nll, lse, logits = ops.linear_ce_forward(h, w, lab, softcap=softcap, store_logits=store)
        zz = logits.float() if store else z              # the statistics are those of the stored, rounded logits
        ref = torch.nn.functional.cross_entropy(zz, lab, reduction="none", ignore_index=-100)
        # fp32 exponentials (2 units of 2^-23 each) and sums over V of them: 1e-5 of the size of the logits
        assert float((nll - ref).abs().max()) < 1e-5 * max(1.0, float(zz.abs().max())) * 4
        if store:
            assert float((logits.float() - z).abs().max()) <= 2 ** -8 * float(z.abs().max())


# one row; the edges of the epilogue's 64-column rounds and 128-column halves, of the tile and of its five stages; several waves
@pytest.mark.parametrize("M,inter,K", [(1, 64, 64), (255, 192, 320), (257, 320, 384), (600, 448, 72), (2600, 2368, 200)])
@pytest.mark.parametrize("act", ["silu", "gelu", "gelu_tanh"])
def test_gated_activation_backward(M, inter, K, act):
    """The fused launch equals the data gradient and the element-wise kernel bit for bit, with pre-activations of a wider pitch too."""
    from opaque_b200 import ops
    torch.manual_seed(M)
    dy, wd = (torch.randn(*s, device="cuda", dtype=torch.bfloat16) / K ** 0.25 for s in ((M, K), (K, inter)))
    g, u = (torch.randn(M, inter + 8, device="cuda", dtype=torch.bfloat16)[:, :inter] for _ in range(2))
    g[0, :3] = torch.tensor([float("inf"), -100.0, 100.0])
    want = ops.functional.glu_backward(ops.gemm(dy, wd, b_layout="kn"), g.contiguous(), u.contiguous(), act)
    for pair in ((g, u), (g.contiguous(), u.contiguous())):
        for got, ref in zip(ops.gemm_glu_bwd(dy, wd, *pair, act=act), want):
            assert torch.equal(got.view(torch.int16), ref.view(torch.int16))


@pytest.mark.parametrize("rows,inter", [(40, 192), (2600, 2368)])             # two launches and one (ops.pick_glu_bwd)
@pytest.mark.parametrize("trainable", [False, True])
def test_gated_mlp_as_one_function(rows, inter, trainable):
    """Outputs and every gradient of the one-node MLP equal the separate nodes'; with a hook on the down projection it is not taken."""
    from opaque_b200.engine import fused
    from opaque_b200.engine.fused import FusedDPEngine
    from opaque_b200.models import LlamaConfig, LlamaForCausalLM, shift_labels
    from opaque_b200.random import key
    results, nodes = [], []
    for on in (True, False, "hook"):
        torch.manual_seed(rows)
        cfg = LlamaConfig.tiny()
        cfg.intermediate_size, cfg.num_hidden_layers, cfg.max_position_embeddings = inter, 1, 4096
        model = LlamaForCausalLM(cfg, device="cuda")
        if not trainable:
            model.add_lora(8, 16.0)
            for n, p in model.named_parameters():
                if n.endswith("lora_B"):
                    torch.nn.init.normal_(p, std=0.05)
        eng = FusedDPEngine(model, clipping_norm=1.0, noise_multiplier=0.0, normalize_by=2.0, key=key(0), microbatch_size=2)
        if on == "hook":
            model.model.layers[0].mlp.down_proj.register_forward_hook(lambda *a: nodes.append(1))
        ids = torch.randint(0, 256, (2, rows // 2), device="cuda")
        old, fused.FUSE_GLU_MLP = fused.FUSE_GLU_MLP, bool(on)
        try:
            res = eng.accumulate(model.per_example_loss, {"input_ids": ids, "labels": shift_labels(ids)})
        finally:
            fused.FUSE_GLU_MLP = old
        results.append((res.losses, res.norms, eng.space.grad.local.clone()))
    assert nodes == [1]
    for other in results[1:]:
        assert torch.equal(results[0][0], other[0])
        # bf16 products and activations are the same bits; norms and gradients add fp32 values with atomics, and the library
        # attention's backward may round differently between two runs (2^-8 of single values)
        for a, b in zip(results[0][1:], other[1:]):
            assert float((a - b).norm()) <= 2e-3 * float(b.norm())


# one row, edges of the 64-, 128- and 256-wide tiles and of the rounds, several waves of either kernel
@pytest.mark.parametrize("M,N,K", [(1, 64, 64), (127, 192, 320), (129, 320, 72), (257, 448, 384), (2600, 2368, 200)])
@pytest.mark.parametrize("act", ["silu", "gelu", "gelu_tanh"])
@pytest.mark.parametrize("kernel", ["single", "pair", "auto"])
def test_plain_activation_epilogues(M, N, K, act, kernel):
    """Forward and backward equal the product and the element-wise kernel bit for bit."""
    from opaque_b200 import ops
    from opaque_b200.ops import lib
    code = {"silu": 0, "gelu": 1, "gelu_tanh": 2}[act]

    def elementwise(x, dy=None):
        out = torch.empty_like(x)
        lib.check(lib.load().ob_activation(x.data_ptr(), lib.ptr(dy), out.data_ptr(), x.numel(), code, lib.sm_count(), lib.stream()), "activation")
        return out
    torch.manual_seed(M)
    a, b, w = (torch.randn(*s, device="cuda", dtype=torch.bfloat16) / K ** 0.25 for s in ((M, K), (N, K), (K, N)))
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    bias[:3] = torch.tensor([float("inf"), -100.0, 100.0])
    st = ops.StatusWord("cuda")
    f = ops.gemm(a, b, bias=bias)
    h, x = ops.gemm_act(a, b, bias, act=act, kernel=kernel, status=st)
    only, none = ops.gemm_act(a, b, bias, act=act, kernel=kernel, save_preact=False, status=st)
    df = ops.gemm_act_bwd(a, w, f, act=act, kernel=kernel, status=st)
    assert none is None and st.read() == 0
    for got, want in ((x, f), (h, elementwise(f)), (only, h), (df, elementwise(f, ops.gemm(a, w, b_layout="kn")))):
        assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    with pytest.raises(ValueError):
        ops.gemm_act_bwd(a, w[:, :-8].contiguous(), f[:, :-8].contiguous(), act=act)


@pytest.mark.parametrize("M,N,K", [(300, 264, 4608), (513, 520, 4616), (2600, 1032, 4672)])
def test_tiles_agree_around_the_line_between_them(M, N, K):
    """The last K that always takes the small tile, and the first ones that weigh the waves of both."""
    test_tiles_agree_bit_for_bit(M, N, K, "nk")
