"""Row kernels of the mixture of experts against fp64 (one rounding to bf16: 2^-9 relative)."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(x, y):
    return float((x.double() - y.double()).norm() / y.double().norm())


@pytest.mark.parametrize("T,k,H", [(1, 1, 8), (5, 4, 264), (130, 6, 2048), (33, 5, 72)])
def test_combine_and_row_gradients(T, k, H):
    from opaque_b200.ops import functional as F
    g = torch.Generator(device="cuda").manual_seed(T)
    y = torch.randn(T * k, H, device="cuda", generator=g, dtype=torch.bfloat16)
    w = torch.rand(T, k, device="cuda", generator=g).to(torch.bfloat16)
    dout = torch.randn(T, H, device="cuda", generator=g, dtype=torch.bfloat16)
    slot = torch.randperm(T * k, device="cuda", generator=g)          # slot of every sorted row
    token = slot // k
    pos = torch.empty_like(slot)
    pos[slot] = torch.arange(T * k, device="cuda")
    rows = y.double()[pos].view(T, k, H)
    assert _rel(F.moe_combine(y, pos, k, w), (rows * w.double()[..., None]).sum(1)) < 4e-3
    assert _rel(F.moe_combine(y, pos, k), rows.sum(1)) < 4e-3
    dy, dw = F.moe_row_grad(dout, y, w, token, slot)
    gd = dout.double()[token]
    assert _rel(dy, gd * w.double().view(-1)[slot][:, None]) < 4e-3
    ref = torch.empty(T * k, device="cuda", dtype=torch.float64)
    ref[slot] = (gd * y.double()).sum(1)
    assert float((dw - ref).abs().max()) < 1e-6 * H * 16
    with pytest.raises(ValueError):
        F.moe_combine(y, pos[:-1], k, w)


def test_experts_take_gradients_that_start_anywhere():
    """The gradient of an output that was flattened into a longer vector starts off the 16-byte boundary."""
    from opaque_b200.models import MoEConfig, MoEForCausalLM
    cfg = MoEConfig.tiny()
    torch.manual_seed(0)
    experts = MoEForCausalLM(cfg, device="cuda").layers[0].mlp.experts
    T, k, H = 18, cfg.num_experts_per_tok, cfg.hidden_size
    x, up = (torch.randn(T, H, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    idx = torch.stack([torch.randperm(cfg.num_experts, device="cuda")[:k] for _ in range(T)])
    w = torch.rand(T, k, device="cuda").to(torch.bfloat16)
    grads = []
    for shift in (0, 1):
        xi = x.clone().requires_grad_(True)
        y = experts(xi, idx, w, 2, 9)
        torch.cat([y.new_zeros(shift), y.flatten()]).backward(torch.cat([up.new_zeros(shift), up.flatten()]))
        grads.append(xi.grad)
    assert torch.equal(*grads)


def test_packed_gated_backward():
    from opaque_b200.ops import functional as F
    for rows, I in ((1, 8), (37, 136)):
        gu = torch.randn(rows, 2 * I, device="cuda", dtype=torch.bfloat16)
        dh = torch.randn(rows, I, device="cuda", dtype=torch.bfloat16)
        x = gu.double().requires_grad_(True)
        (torch.nn.functional.silu(x[:, :I]) * x[:, I:]).backward(dh.double())
        assert _rel(F.glu_backward_packed(dh, gu), x.grad) < 4e-3


@pytest.mark.parametrize("rows,I", [(1, 8), (37, 136), (900, 1408)])
def test_packed_gated_backward_has_the_bits_of_the_separate_operations(rows, I):
    """Of the 2.5 million values of the largest case about 30 round otherwise with an approximate sigmoid."""
    from opaque_b200.ops import functional as F
    g = torch.Generator(device="cuda").manual_seed(rows)
    gu = 3 * torch.randn(rows, 2 * I, device="cuda", generator=g, dtype=torch.bfloat16)
    gu.view(-1)[:6] = torch.tensor([0.0, -0.0, 100.0, -100.0, 88.0, -88.0])
    dh = torch.randn(rows, I, device="cuda", generator=g, dtype=torch.bfloat16)
    gate, up, d = gu[:, :I].float(), gu[:, I:].float(), dh.float()
    sig = torch.sigmoid(gate)
    ref = torch.cat([d * up * sig * (1 + gate * (1 - sig)), d * (gate * sig)], dim=1).to(gu.dtype)
    assert torch.equal(F.glu_backward_packed(dh, gu), ref)
