"""Residual addition fused into LayerNorm, and bias sums of many layers in one launch, against fp64 / the single-layer kernels."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(x, y):
    return float((x.double() - y.double()).norm() / y.double().norm())


@pytest.mark.parametrize("rows,H", [(1, 8), (7, 256), (9, 264), (130, 512), (33, 768), (5, 776), (17, 1024), (4, 1032)])
@pytest.mark.parametrize("bias", [True, False])
def test_add_layer_norm(rows, H, bias):
    from opaque_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(rows)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g, dtype=torch.bfloat16)          # noqa: E731
    x, res, w, b = r(rows, H).requires_grad_(True), r(rows, H).requires_grad_(True), r(H).requires_grad_(True), r(H).requires_grad_(True) if bias else None
    gy, gs = r(rows, H), r(rows, H)
    s64 = (x.double() + res.double()).bfloat16().double().detach().requires_grad_(True)
    w64, b64 = w.double().detach().requires_grad_(True), b.double().detach().requires_grad_(True) if bias else None
    y64 = torch.nn.functional.layer_norm(s64, (H,), w64, b64, 1e-5)
    for grads in ((gy, gs), (gy, None), (None, gs)):
        leaves = [t for t in (x, res, w, b) if t is not None]
        for t in leaves + [s64, w64] + ([b64] if bias else []):
            t.grad = None
        y, s = ops.add_layer_norm(x, res, w, b)
        assert torch.equal(s.double(), s64) and _rel(y, y64) < 4e-3
        used = [(o, q) for o, q in zip((y, s), grads) if q is not None]
        torch.autograd.backward([o for o, _ in used], [q for _, q in used])
        torch.autograd.backward([o for o, q in zip((y64, s64), grads) if q is not None], [q.double() for q in grads if q is not None], retain_graph=True)
        assert torch.equal(x.grad, res.grad) and _rel(x.grad, s64.grad) < 6e-3
        if grads[0] is not None:                 # parameters: fp32 sums over the rows, rounded to bf16
            assert _rel(w.grad, w64.grad) < 6e-3 and (not bias or _rel(b.grad, b64.grad) < 6e-3)


@pytest.mark.parametrize("rows,H", [(1, 8), (9, 264), (130, 512), (333, 768), (17, 1024)])
def test_add_layer_norm_has_the_bits_of_the_separate_operations(rows, H):
    """Addition, norm and the sum of both gradients as three bf16 operations: the same bits, forward and backward."""
    from opaque_b200 import ops
    x, res, gy, gs = (torch.randn(rows, H, device="cuda", dtype=torch.bfloat16) for _ in range(4))
    w, b = (torch.randn(H, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    xf, rf = x.clone().requires_grad_(True), res.clone().requires_grad_(True)
    y, s = ops.add_layer_norm(xf, rf, w, b)
    torch.autograd.backward([y, s], [gy, gs])
    s2 = (x + res).requires_grad_(True)
    y2 = ops.layer_norm(s2, w, b)
    y2.backward(gy)
    assert torch.equal(y, y2) and torch.equal(s, s2)
    assert torch.equal(xf.grad, s2.grad + gs) and torch.equal(rf.grad, xf.grad)


def test_norms_and_activations_of_views_that_start_anywhere():
    """Contiguous views off the 16-byte boundary give what their aligned copies give, in both directions."""
    from opaque_b200 import ops
    off = lambda t: torch.cat([t.new_zeros(1), t.flatten()])[1:].view(t.shape)            # noqa: E731
    x, res, gy, gs = (torch.randn(5, 64, device="cuda", dtype=torch.bfloat16) for _ in range(4))
    w, b = (torch.randn(64, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    assert off(x).is_contiguous() and off(x).data_ptr() % 16 == 2
    for fn, grads in ((lambda p, q: ops.add_layer_norm(p, q, w, b), 2), (lambda p, q: ops.fused_add_rms_norm(p, q, w), 2),
                      (lambda p, q: (ops.layer_norm(p + q, w, b),), 1), (lambda p, q: (ops.layer_norm(p, w, b),), 1),
                      (lambda p, q: (ops.rms_norm(p, w),), 1), (lambda p, q: (ops.activation(p, "silu"),), 1),
                      (lambda p, q: (ops.swiglu(p, q),), 1), (lambda p, q: (ops.geglu(p, q),), 1)):
        out = []
        for shift in (lambda t: t, off):
            p, q = shift(x).detach().requires_grad_(True), shift(res).detach().requires_grad_(True)
            ys = fn(p, q)
            torch.autograd.backward(list(ys), [shift(g) for g in (gy, gs)[:grads]])
            out.append((*ys, p.grad, q.grad))
        assert all(torch.equal(u, v) if u is not None else v is None for u, v in zip(*out))
    # gate and up as slices of rows that start elsewhere: one pitch for both, neither aligned
    rows = torch.randn(5, 136, device="cuda", dtype=torch.bfloat16)
    assert torch.equal(ops.swiglu(rows[:, 1:65], rows[:, 66:130]), ops.swiglu(rows[:, 1:65].contiguous(), rows[:, 66:130].contiguous()))
    for fn in (lambda: ops.layer_norm(x, off(w)), lambda: ops.rms_norm(x, off(w)), lambda: ops.add_layer_norm(x, res, w, off(b)),
               lambda: ops.fused_add_rms_norm(x, res, off(w))):
        with pytest.raises(ops.KernelLibraryError):         # parameters are not copied: the entry points refuse what would fault
            fn()


@pytest.mark.parametrize("count", [1, 3, 130])
@pytest.mark.parametrize("B,T", [(1, 1), (3, 70), (2, 513)])
def test_bias_sums_batched(count, B, T):
    from opaque_b200.ops import functional as F
    jobs, refs = [], []
    for i in range(count):
        N = 8 * (1 + (37 * i) % 70)
        g = torch.randn(B * T, N + 8, device="cuda", dtype=torch.bfloat16)[:, :N]
        buf = torch.full((B, N + 3), 2.0, device="cuda")
        jobs.append((buf[:, :N], g))
        refs.append((buf, g.double().view(B, T, N).sum(1) + 2.0))
    F.rows_sum_batch_(jobs, B)
    for buf, ref in refs:
        # fp32 sums of T values of size one: T * 2^-24 * sqrt(T)
        assert float((buf[:, :-3].double() - ref).abs().max()) < 1e-5 * max(T, 8) and bool((buf[:, -3:] == 2.0).all())
    with pytest.raises(ValueError):
        F.rows_sum_batch_([(jobs[0][0][:, :4], jobs[0][1])], B)


@pytest.mark.parametrize("B,T", [(1, 1), (3, 70), (2, 513)])
def test_norm_weight_sums_batched(B, T):
    from opaque_b200.ops import functional as F
    jobs, one = [], []
    for i, N in enumerate((8, 264, 768, 1032, 16)):
        g, x = (torch.randn(B * T, N, device="cuda", dtype=torch.bfloat16) for _ in range(2))
        mean, rstd = torch.randn(B * T, device="cuda"), torch.rand(B * T, device="cuda")
        args = (x, mean if i % 2 == 0 else None, rstd)
        a, b, pa, pb = (torch.ones(B, N, device="cuda") for _ in range(4))
        plain = i % 3 != 1
        jobs.append((a, g, *args, pa if plain else None))
        F.rows_group_sum_(b, g, B, x2d=x, mean=args[1], rstd=rstd, out_plain=pb if plain else None)
        one.append((a, b, pa, pb))
    jobs.append((torch.zeros(B, 8, device="cuda"), torch.randn(B * T, 8, device="cuda", dtype=torch.bfloat16)))
    F.rows_sum_batch_(jobs, B)
    for a, b, pa, pb in one:                     # the same arithmetic; only the order of the atomics differs
        assert torch.allclose(a, b, rtol=1e-5, atol=1e-4) and torch.allclose(pa, pb, rtol=1e-5, atol=1e-4)


def test_gpt2_blocks_with_hooks_see_the_unsplit_stream():
    from opaque_b200.models import GPT2Config, GPT2LMHeadModel
    torch.manual_seed(0)
    m = GPT2LMHeadModel(GPT2Config.tiny(), device="cuda")
    ids = torch.randint(0, 500, (2, 33), device="cuda")
    assert m._carries()
    with torch.no_grad():
        plain = m.hidden_states(ids)
        seen = []
        handle = m.h[1].register_forward_hook(lambda mod, args, out: seen.append((args[0].shape, out.shape)))
        hooked = m.hidden_states(ids)
        handle.remove()
    assert not m.h[1]._forward_hooks and seen == [((2, 33, 128), (2, 33, 128))]
    # the split stream adds in the norm's kernel what the plain one adds before it: the same bf16 sums
    assert torch.equal(plain, hooked)


@pytest.mark.parametrize("rows,I,pitched", [(1, 8, False), (3, 264, True), (700, 1032, False), (700, 1032, True)])
@pytest.mark.parametrize("act", ["silu", "gelu", "gelu_tanh", "relu"])
def test_activation_variants(rows, I, pitched, act):
    """Every activation's own kernel, forward and backward, contiguous and with rows further apart than their length."""
    from opaque_b200.ops import functional as F
    fn = {"silu": torch.nn.functional.silu, "gelu": torch.nn.functional.gelu, "relu": torch.relu,
          "gelu_tanh": lambda v: torch.nn.functional.gelu(v, approximate="tanh")}[act]
    both = torch.randn(rows, 2 * I, device="cuda", dtype=torch.bfloat16)
    gate, up = both[:, :I], both[:, I:]
    if not pitched:
        gate, up = gate.contiguous(), up.contiguous()
    dh = torch.randn(rows, I, device="cuda", dtype=torch.bfloat16)
    x = gate.double().requires_grad_(True)
    fn(x).backward(dh.double())
    d_act = x.grad
    xb = gate.clone().requires_grad_(True)
    y = F.activation(xb, act)
    y.backward(dh)
    # one bf16 rounding of the result (2^-9 of it) on top of fp32 arithmetic.  The single-precision hardware tanh is good to 2^-11:
    # half of that times |x| in x (1 + t) / 2, and |x| (1 - t^2) u' besides in its derivative, with |u'| <= 0.8 (1 + 0.135 x^2)
    v = gate.double().abs()
    err = 2.0 ** -11 if act == "gelu_tanh" else 1e-6
    e_fwd, e_bwd = err * (0.5 * v + 0.01), err * (0.5 + 0.8 * v * (1 + 0.135 * v * v)) + 1e-6
    close = lambda got, want, tol: bool(((got.double() - want).abs() <= 2 ** -8 * want.abs() + tol + 1e-6).all())
    d, u = dh.double().abs(), up.double().abs()
    assert close(y, fn(gate.double()), e_fwd) and close(xb.grad, d_act, d * e_bwd)
    if act != "relu":
        dg, du = F.glu_backward(dh, gate, up, act)
        assert close(dg, d_act * up.double(), d * u * e_bwd) and close(du, dh.double() * fn(gate.double()), d * e_fwd)


# one row per example, fewer rows than warps, ragged chunks, several rows per warp; widths at the edges of the vectors per lane
@pytest.mark.parametrize("E,T,H", [(1, 1, 8), (3, 7, 256), (300, 2, 264), (5, 333, 512), (2, 1000, 768), (7, 130, 776), (9, 600, 1024)])
@pytest.mark.parametrize("residual", [True, False])
def test_layer_norm_backward_with_sums(E, T, H, residual):
    """Data gradient: the bits of the kernels without the sums.  Sums: against 64 bits; fp32 sums of T terms, 2^-24 each times a factor
    of two for the terms' own roundings and sqrt(T) for their number."""
    from opaque_b200.ops import lib
    torch.manual_seed(T)
    rows = E * T
    dy, x, ds = (torch.randn(rows, H, device="cuda").bfloat16() for _ in range(3))
    w = torch.randn(H, device="cuda").bfloat16()
    stats = torch.stack([x.float().mean(1), 1 / x.float().std(1, unbiased=False).clamp_min(0.1)]).contiguous()
    mean, rstd = stats.data_ptr(), stats.data_ptr() + 4 * rows
    L, want, got = lib.load(), torch.empty_like(dy), torch.empty_like(dy)
    if residual:
        lib.check(L.ob_add_layernorm_bwd_dx(dy.data_ptr(), x.data_ptr(), w.data_ptr(), mean, rstd, ds.data_ptr(), want.data_ptr(), rows, H, lib.stream()), "")
    else:
        lib.check(L.ob_layernorm_bwd_dx(dy.data_ptr(), x.data_ptr(), w.data_ptr(), mean, rstd, want.data_ptr(), rows, H, lib.stream()), "")
    pe = torch.ones(E, 2 * H + 8, device="cuda")
    lib.check(L.ob_layernorm_bwd_sums(dy.data_ptr(), x.data_ptr(), w.data_ptr(), mean, rstd, ds.data_ptr() if residual else None, got.data_ptr(), E, T, H,
                                      pe.data_ptr(), pe.data_ptr() + 4 * H, pe.stride(0), lib.stream()), "layernorm_bwd_sums")
    assert torch.equal(got, want)
    xh = (x.double() - stats[0].double()[:, None]) * stats[1].double()[:, None]
    ref = torch.cat([(dy.double() * xh).view(E, T, H).sum(1), dy.double().view(E, T, H).sum(1)], 1)
    assert torch.all(pe[:, 2 * H:] == 1) and float((pe[:, :2 * H].double() - 1 - ref).norm()) <= 2 ** -23 * (T ** 0.5 + 2) * float((1 + ref.abs()).norm())


# where 16 chunks per example are a few blocks more than SMs: one block per SM with longer chunks instead, down to the last row
@pytest.mark.parametrize("E,T,H", [(10, 129, 256), (12, 140, 768), (10, 1024, 776), (16, 131, 1024), (74, 60, 1024)])
@pytest.mark.parametrize("residual", [True, False])
def test_layer_norm_backward_with_sums_in_one_wave(E, T, H, residual):
    test_layer_norm_backward_with_sums(E, T, H, residual)


@pytest.mark.parametrize("rows,H", [(4737, 520), (4800, 768), (9473, 776), (5000, 1024)])
def test_add_layer_norm_of_many_rows(rows, H):
    """Rows that come through the ring: against the fp32 statement, and the bits that the same rows have in a short call."""
    from opaque_b200 import ops
    torch.manual_seed(rows)
    x, r = (torch.randn(rows, H, device="cuda").bfloat16() for _ in range(2))
    w, b = (torch.randn(H, device="cuda").bfloat16() for _ in range(2))
    y, s = ops.add_layer_norm(x, r, w, b)
    assert torch.equal(s, x + r)
    for lo in (0, rows - 100):
        ys, _ = ops.add_layer_norm(x[lo:lo + 100], r[lo:lo + 100], w, b)
        assert torch.equal(ys, y[lo:lo + 100])
