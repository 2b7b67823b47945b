"""Products on the single-CTA kernel: edges of rows, columns and k-blocks, both layouts of both segments, scale and bias, pitched
outputs, narrow tiles; and the same bits from every kernel and tile shape that ``auto`` chooses between.

Tolerance: operands are bf16 and products exact in fp32; the fp32 sum of K terms and the final rounding to bf16 leave a relative
2-norm error of 2^-9 (rounding) + K * 2^-24, below 4e-3 for every K here.
"""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 4e-3


def _rel(x, y):
    return float((x.float() - y.float()).norm() / y.float().norm())


@pytest.mark.parametrize("M,N,K,K2", [(1, 8, 64, 0), (127, 64, 520, 16), (128, 264, 512, 64), (129, 136, 1000, 48), (300, 520, 4096, 8), (257, 200, 768, 768),
                                      (128, 768, 3072, 0), (1285, 768, 3072, 0), (256, 2048, 8192, 0), (300, 768, 50304, 0)])
@pytest.mark.parametrize("layout,layout2", [("nk", "nk"), ("kn", "kn"), ("nk", "kn"), ("kn", "nk")])
def test_products_match_fp32_and_have_the_same_bits_in_every_kernel(M, N, K, K2, layout, layout2):
    """The choice of a kernel by size must not show in a result: the k-blocks of a tile are added in one order everywhere."""
    from opaque_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g, dtype=torch.bfloat16)      # noqa: E731
    a, w, bias = r(M, K), r(N, K), r(N)
    a2, w2 = (r(M, K2), r(N, K2)) if K2 else (None, None)
    prod = a.float() @ w.float().t() + (a2.float() @ w2.float().t() if K2 else 0.0)
    b = w if layout == "nk" else w.t().contiguous()
    b2 = None if not K2 else (w2 if layout2 == "nk" else w2.t().contiguous())
    kw = dict(b_layout=layout, a2=a2, b2=b2, b2_layout=layout2, bias=bias)
    st = ops.StatusWord()
    ref = ops.gemm(a, b, kernel="single", block_n=256, status=st, **kw)
    assert st.read() == 0 and _rel(ref, prod + bias.float()) < TOL
    for choice in (dict(), dict(kernel="single"), dict(kernel="single", block_n=64), dict(kernel="pair")):
        assert torch.equal(ops.gemm(a, b, **choice, **kw), ref), choice
    assert torch.equal(ops.gemm_pair(a, b, tile="256x256", **kw), ref)
    assert _rel(ops.gemm(a, b, alpha=0.5, **kw), 0.5 * prod + bias.float()) < TOL


def test_products_write_inside_a_pitched_output_only():
    from opaque_b200 import ops
    a, w = torch.randn(130, 256, device="cuda", dtype=torch.bfloat16), torch.randn(72, 256, device="cuda", dtype=torch.bfloat16)
    for pitch in (80, 75):                               # rows for vector stores and rows that need scalar stores
        buf = torch.full((130, pitch), 7.0, device="cuda", dtype=torch.bfloat16)
        ops.gemm(a, w, out=buf[:, :72], kernel="single")
        assert _rel(buf[:, :72], a.float() @ w.float().t()) < TOL and bool((buf[:, 72:] == 7.0).all())


def test_scale_runs_on_the_single_cta_kernel():
    from opaque_b200 import ops
    a, w = torch.randn(64, 128, device="cuda", dtype=torch.bfloat16), torch.randn(64, 128, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(ValueError):
        ops.gemm(a, w, kernel="pair", alpha=2.0)


def test_lora_operands_packed_in_one_launch():
    from opaque_b200 import ops
    for r, d, outs in ((8, 8, (8, 16, 24)), (16, 200, (64, 8, 8)), (32, 72, (40, 40, 136))):
        f = [(torch.randn(r, d, device="cuda", dtype=torch.bfloat16), torch.randn(o, r, device="cuda", dtype=torch.bfloat16)) for o in outs]
        a, b = ops.lora_pack(f)
        assert torch.equal(a, torch.cat([x for x, _ in f])) and torch.equal(b, torch.block_diag(*[y for _, y in f]))


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (128, 64, 64), (130, 72, 1000), (257, 328, 136), (64, 16, 2048), (20000, 56, 72)])
def test_narrow_tiles(M, N, K):
    from opaque_b200 import ops
    torch.manual_seed(M + N)
    a, bias = torch.randn(M, K, device="cuda", dtype=torch.bfloat16), torch.randn(N, device="cuda", dtype=torch.bfloat16)
    a2 = torch.randn(M, 16, device="cuda", dtype=torch.bfloat16)
    for layout, layout2 in (("nk", "kn"), ("kn", "nk")):
        w = torch.randn((N, K) if layout == "nk" else (K, N), device="cuda", dtype=torch.bfloat16)
        b2 = torch.randn((N, 16) if layout2 == "nk" else (16, N), device="cuda", dtype=torch.bfloat16)
        prod = a.float() @ (w.float().t() if layout == "nk" else w.float()) + a2.float() @ (b2.float().t() if layout2 == "nk" else b2.float())
        buf = torch.full((M, N + 8), 7.0, device="cuda", dtype=torch.bfloat16)
        kw = dict(b_layout=layout, a2=a2, b2=b2, b2_layout=layout2, bias=bias, alpha=0.5, kernel="single")
        ops.gemm(a, w, out=buf[:, :N], block_n=64, **kw)
        assert _rel(buf[:, :N], 0.5 * prod + bias.float()) < TOL and bool((buf[:, N:] == 7.0).all())
        # a tile's k-blocks are added in the same order whatever its width
        assert torch.equal(buf[:, :N], ops.gemm(a, w, block_n=256, **kw))
    with pytest.raises(ops.KernelLibraryError):
        ops.gemm(a, w, b_layout="kn", kernel="single", block_n=128)


def test_tile_width_follows_the_number_of_narrow_tiles():
    from opaque_b200 import ops
    assert ops.pick_tile_width(10 ** 6, 64, 2) == 64 and ops.pick_tile_width(128, 768, 12) == 64
    assert ops.pick_tile_width(2048, 768, 12) == 256 and ops.pick_tile_width(16384, 3072, 12) == 256 and ops.pick_tile_width(128, 50304, 12) == 256
