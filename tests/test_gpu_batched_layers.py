"""Batched launches of the norm and weight-gradient kernels: the same problems one by one give the same numbers, whatever
their number (one launch holds 56), shapes, order and destination.  Sums are fp32 in both; only atomics' order differs."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(x, y):
    return float((x.double() - y.double()).norm() / y.double().norm().clamp_min(1e-30))


def _r(*s):
    return torch.randn(*s, device="cuda", dtype=torch.bfloat16)


@pytest.mark.parametrize("count,T", [(1, 64), (3, 130), (65, 40), (5, 1100)])
def test_ghost_norms_batched(count, T):
    from opaque_b200 import ops
    B = 3
    ids = torch.randint(0, 9, (B * T,), device="cuda", dtype=torch.int32)
    seg = torch.tensor([0, 5, 5, T, 2 * T + 7, 3 * T], device="cuda", dtype=torch.int32)
    seg_out = torch.tensor([0, 1, 2, 0, 1], device="cuda", dtype=torch.int32)
    longest = T + 7
    jobs, one = [], []
    got = torch.zeros(count, B, device="cuda")
    for i in range(count):
        a, g = _r(B * T, 8 * (i % 5 + 1)), _r(B * T, 72 + 8 * (i % 3))
        kind = i % 3
        extra = dict(ids=ids) if kind == 1 else (dict(seg_offsets=seg, seg_out=seg_out) if kind == 2 else {})
        tokens = longest if kind == 2 else T
        n2 = torch.zeros(B, device="cuda")
        ops.ghost_norm(None if kind == 1 else a, g, n2, tokens, **extra)
        one.append(n2)
        jobs.append((None if kind == 1 else a, g, got[i], tokens, extra.get("ids"), extra.get("seg_offsets"), extra.get("seg_out")))
        if kind == 0:
            assert _rel(n2, ops.ghost_norm_ref(a, g, T)) < 2e-5
    st = ops.StatusWord()
    ops.ghost_norm_batch(jobs, status=st)
    assert st.read() == 0 and all(_rel(got[i], one[i]) < 1e-6 for i in range(count))


@pytest.mark.parametrize("count", [1, 7, 66])
def test_weight_gradients_batched(count):
    from opaque_b200 import ops
    T = 200
    scale = torch.rand(T, device="cuda")
    shapes = [(64 + 8 * (i % 7), 136 + 8 * (i % 4)) for i in range(count)]
    offs, total = [], 0
    for m, n in shapes:
        offs.append(total)
        total += m * n
    out = torch.ones(total, device="cuda")
    probs = [dict(a=_r(T, m), b=_r(T, n), out_offset=o, row_scale=scale if i % 2 else None) for i, ((m, n), o) in enumerate(zip(shapes, offs))]
    st = ops.StatusWord()
    ops.wgrad_clip_batch(probs, out, status=st)
    assert st.read() == 0
    for pr, (m, n), o in zip(probs, shapes, offs):
        ref = ops.wgrad_clip_ref(pr["a"], pr["b"], row_scale=pr["row_scale"])[0] + 1.0
        # with factors the scaled operand is rounded to bf16 (twice at most): 2^-8 relative
        assert _rel(out[o:o + m * n].view(m, n), ref) < (1e-5 if pr["row_scale"] is None else 6e-3)
    with pytest.raises(ValueError):
        ops.wgrad_clip_batch(probs, torch.zeros(total - 1, device="cuda"))


def test_weight_gradients_batched_store_mode_per_example():
    from opaque_b200 import ops
    B, T, r = 3, 50, 16
    seg = torch.arange(0, (B + 1) * T, T, device="cuda", dtype=torch.int32)
    x, g, q, xa = _r(B * T, 72), _r(B * T, 40), _r(B * T, r), _r(B * T, r)
    pe = torch.full((B, 72 * r + 40 * r), 5.0, device="cuda")
    common = dict(seg_offsets=seg, num_groups=B, group_stride=pe.stride(0), n_valid=r)
    ops.wgrad_clip_batch([dict(a=x, b=q, out_offset=0, ldm=1, ldn=72, **common), dict(a=g, b=xa, out_offset=72 * r, ldm=r, ldn=1, **common)],
                         pe, accumulate=False, block_n=64)
    ra = ops.wgrad_clip_ref(x, q, seg_offsets=seg, num_groups=B).transpose(1, 2).reshape(B, -1)
    rb = ops.wgrad_clip_ref(g, xa, seg_offsets=seg, num_groups=B).reshape(B, -1)
    assert _rel(pe, torch.cat([ra, rb], 1)) < 1e-5


@pytest.mark.parametrize("count", [2, 65])
def test_per_example_kernels_batched(count):
    from opaque_b200 import ops
    B, R = 3, 128
    c = torch.tensor([0.5, 0.0, 1.5], device="cuda")
    probs, refs, norms, total = [], [], [], 0
    for i in range(count):
        m, n = 136 + 8 * (i % 3), 264 - 8 * (i % 5)
        a, b = _r(B * R, m), _r(B * R, n)
        probs.append((a, b, c, total, n))
        refs.append(ops.wgrad_clip_ref(a, b, row_scale=c.repeat_interleave(R))[0].reshape(-1))
        norms.append(torch.stack([(a[e * R:(e + 1) * R].float().t() @ b[e * R:(e + 1) * R].float()).square().sum() for e in range(B)]))
        total += m * n
    out, st = torch.zeros(total, device="cuda"), ops.StatusWord()
    ops.wgrad_clip_per_example_batch(probs, out, R, status=st)
    assert st.read() == 0 and _rel(out, torch.cat(refs)) < 2e-5
    n2 = torch.zeros(count, B, device="cuda")
    ops.direct_norm2_batch([(p[0], p[1], n2[i]) for i, p in enumerate(probs)], R, status=st)
    assert st.read() == 0 and _rel(n2, torch.stack(norms)) < 2e-5


@pytest.mark.parametrize("offset", [0, 4, 1])
@pytest.mark.parametrize("M,N,ldm", [(8, 136, 136), (130, 140, 140), (257, 264, 300), (40, 520, 521)])
def test_accumulating_destinations(offset, M, N, ldm):
    """Grouped and dense accumulation into aligned destinations (reduced by the TMA engine) and unaligned ones (by the warps):
    nothing outside the matrices is touched, empty groups add nothing."""
    from opaque_b200 import ops
    offs = torch.tensor([0, 70, 70, 199, 200], device="cuda", dtype=torch.int32)
    a, b = (_r(200, (w + 7) // 8 * 8)[:, :w] for w in (M, N))
    gstride = M * ldm + 4
    ref = ops.wgrad_clip_ref(a, b, seg_offsets=offs, num_groups=4)
    out = torch.full((offset + 5 * gstride,), 3.0, device="cuda")
    want, inside = out.clone(), torch.zeros_like(out, dtype=torch.bool)
    for g in range(5):
        want[offset + g * gstride:][:M * ldm].view(M, ldm)[:, :N] += 2 * ref[g] if g < 4 else ref.sum(0)
        inside[offset + g * gstride:][:M * ldm].view(M, ldm)[:, :N] = True
    st = ops.StatusWord()
    for _ in range(2):
        ops.wgrad_clip_batch([dict(a=a, b=b, seg_offsets=offs, num_groups=4, out_offset=offset, ldm=ldm, group_stride=gstride)], out, status=st)
    ops.wgrad_clip_batch([dict(a=a, b=b, out_offset=offset + 4 * gstride, ldm=ldm)], out, status=st)
    assert st.read() == 0 and _rel(out, want) < 1e-5 and bool((out[~inside] == 3.0).all())
    if offset == 0:                                       # the per-example kernel's destination, two examples of 64 rows
        c = torch.tensor([0.5, 2.0], device="cuda")
        out2 = torch.full((M * ldm + 8,), 3.0, device="cuda")
        ops.wgrad_clip_per_example_batch([(a[:128], b[:128], c, 0, ldm)], out2, 64, status=st)
        w2 = torch.full_like(out2, 3.0)
        w2[:M * ldm].view(M, ldm)[:, :N] += ops.wgrad_clip_ref(a[:128], b[:128], row_scale=c.repeat_interleave(64))[0]
        assert st.read() == 0 and _rel(out2, w2) < 1e-5 and bool((out2[:M * ldm].view(M, ldm)[:, N:] == 3.0).all()) and bool((out2[M * ldm:] == 3.0).all())


@pytest.mark.parametrize("R", [1, 40, 63, 65, 129, 333])
def test_per_example_kernels_take_any_length(R):
    """An example's last 64-row block must not see the next example's rows."""
    from opaque_b200 import ops
    B, M, N = 3, 136, 264
    a, b = _r(B * R, M), _r(B * R, N)
    c = torch.tensor([0.5, 0.0, 1.5], device="cuda")
    out, st = torch.zeros(M * N, device="cuda"), ops.StatusWord()
    ops.wgrad_clip_per_example_batch([(a, b, c, 0, N)], out, R, status=st)
    assert st.read() == 0 and _rel(out.view(M, N), ops.wgrad_clip_ref(a, b, row_scale=c.repeat_interleave(R))[0]) < 2e-5
    n2 = torch.zeros(B, device="cuda")
    ops.direct_norm2_batch([(a, b, n2)], R, status=st)
    assert st.read() == 0 and _rel(n2, ops.ghost_norm_ref(a, b, R)) < 5e-5
    if R % 64:
        with pytest.raises(ValueError):                   # the single call still wants whole blocks
            ops.wgrad_clip_per_example(a, b, out, ex_scale=c, rows_per_example=R)


def test_few_records_on_a_wide_head_take_the_direct_norm():
    from opaque_b200 import ops
    assert ops.pick_norm_path(64, 768, 50304, 2) == "direct" and ops.pick_norm_path(199, 2048, 151936, 3) == "direct"
    assert ops.pick_norm_path(64, 768, 50304) == "ghost" and ops.pick_norm_path(512, 768, 50304, 32) == "ghost"
    assert ops.pick_norm_path(64, 768, 3072, 2) == "ghost"
