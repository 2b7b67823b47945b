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
