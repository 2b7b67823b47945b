"""Fused clipping of a materialised gradient tree against the tensor operations it replaces and against fp64."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _tree(E, shapes, seed, strided=False):
    g = torch.Generator(device="cuda").manual_seed(seed)
    leaves = [torch.randn(E, *s, device="cuda", generator=g) * 3.0 ** (i % 4) for i, s in enumerate(shapes)]
    return [x.transpose(-1, -2) if strided and x.ndim > 2 else x for x in leaves]


@pytest.mark.parametrize("E,shapes", [(1, [(1,)]), (3, [(5,), ()]), (65, [(256, 33), (256,), (10, 256), (10,)]), (2, [(8192,), (8193,), (3, 4097)]),
                                      (9, [(4,)] * 64)])
@pytest.mark.parametrize("mode", ["clip", "auto"])
def test_matches_the_tensor_operations(E, shapes, mode):
    from opaque_b200.engine import clipping as C
    for strided in (False, True):
        leaves = _tree(E, shapes, E, strided)
        if E > 2:
            leaves[0][1].reshape(-1)[0] = float("inf")            # counts as zero, like NaN
            leaves[-1][2].reshape(-1)[-1] = float("nan")
            leaves = [x * (torch.arange(E, device="cuda") != 0).view(-1, *[1] * (x.ndim - 1)) if torch.isfinite(x[0]).all() else x for x in leaves]
        clean = [C._sanitize(x) for x in leaves]
        scale_for, norms, _, _ = C.batched_clip_scales(clean, 2.5, mode=mode, gamma=0.01)
        want = [C._weighted_sum(x, scale_for((i,), x.dtype), torch.float32) for i, x in enumerate(clean)]
        assert C._tree_kernel_ok(leaves, None, None)
        sums, n32, cn = C._clip_tree(leaves, 2.5, mode, 0.01, 0.5)
        # both round an fp64 norm to fp32 and the factor to fp32; the sum here is fp64, there fp32 (E terms: E * 2^-24)
        assert torch.allclose(n32, norms, rtol=2e-7, atol=0) and torch.allclose(cn, scale_for((0,), torch.float32).float() * norms, rtol=5e-7, atol=0)
        for a, b, x in zip(sums, want, clean):
            exact = 0.5 * (scale_for((0,), torch.float32).float().double().view(-1, *[1] * (x.ndim - 1)) * x.double()).sum(0)
            bound = 4e-7 * (x.double().abs() * scale_for((0,), torch.float32).view(-1, *[1] * (x.ndim - 1))).sum(0) + 1e-30
            assert a.shape == b.shape and bool(((a - exact).abs() <= bound).all()) and bool(((a - 0.5 * b).abs() <= bound * (E + 2)).all())


def test_clipped_grad_takes_it_and_agrees_over_microbatches():
    from opaque_b200.dpsgd import clipped_grad
    from opaque_b200.engine import clipping as C
    from opaque_b200.functional import make_functional
    torch.manual_seed(0)
    fmodel, params = make_functional(torch.nn.Sequential(torch.nn.Linear(20, 9), torch.nn.Tanh(), torch.nn.Linear(9, 3)).cuda(), disable_autograd_tracking=True)
    x, y = torch.randn(13, 20, device="cuda"), torch.randint(0, 3, (13,), device="cuda")

    def loss(p, a, b):
        return torch.nn.functional.cross_entropy(fmodel(p, a.unsqueeze(0)), b.unsqueeze(0))
    out = {}
    for mb in (None, 5):
        for kernel in (True, False):
            old = C._tree_kernel_ok
            C._tree_kernel_ok = old if kernel else (lambda *a: False)
            try:
                fn, st = clipped_grad(loss, clipping_norm=0.3, normalize_by=7.0, batch_argnums=(1, 2), return_aux=True, microbatch_size=mb)
                (g, aux), _ = fn(params, x, y, state=st)
            finally:
                C._tree_kernel_ok = old
            out[mb, kernel] = (torch.cat([t.reshape(-1) for t in g.pytree]), aux.grad_norms, aux.clipped_grad_norms, aux.clipping_rate, g.max_norm)
    ref = out[None, False]
    for got in out.values():
        assert all(torch.allclose(a, b, rtol=2e-6, atol=2e-7) for a, b in zip(got[:3], ref[:3])) and got[3:] == ref[3:]


def test_what_the_kernels_do_not_take_keeps_the_tensor_path():
    from opaque_b200.engine import clipping as C
    ok = torch.randn(3, 4, device="cuda")
    assert C._tree_kernel_ok([ok], None, None) and C._tree_kernel_ok([ok], torch.float32, torch.float32)
    assert not C._tree_kernel_ok([ok.double()], None, None) and not C._tree_kernel_ok([ok.cpu()], None, None)
    assert not C._tree_kernel_ok([ok], torch.float64, None) and not C._tree_kernel_ok([ok], None, torch.float64)
    assert not C._tree_kernel_ok([ok, 3.0], None, None) and not C._tree_kernel_ok([ok] * 65, None, None) and not C._tree_kernel_ok([], None, None)
    assert not C._tree_kernel_ok([ok[:0]], None, None) and not C._tree_kernel_ok([ok.clone().requires_grad_(True)], None, None)
    assert not C._tree_kernel_ok([torch._neg_view(ok)], None, None) and not C._tree_kernel_ok([ok.to_sparse()], None, None)
    torch.func.vmap(lambda t: (C._tree_kernel_ok([t], None, None), t)[1] if not C._tree_kernel_ok([t], None, None) else 1 / 0)(ok)


@pytest.mark.parametrize("E", [1, 5])                 # one record's view is contiguous as it stands
def test_negated_views_are_clipped_as_they_read(E):
    from opaque_b200.dpsgd.clipping import clipped_fun
    x, c = torch.randn(E, 3, device="cuda"), torch._neg_view(torch.ones(4, device="cuda"))
    fn, st = clipped_fun(lambda a: {"a": 2 * a, "c": c}, clipping_norm=1e3)
    got, _ = fn(x, state=st)
    assert torch.allclose(got.pytree["c"], torch.full_like(x[0, :1], -E).expand(4), rtol=1e-5)
    assert torch.allclose(got.pytree["a"], 2 * x.sum(0), rtol=1e-5, atol=1e-5)
