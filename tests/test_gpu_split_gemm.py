"""Products whose k-blocks are split over several CTAs per tile: edges of rows, columns and k-blocks, both layouts of both
segments, scale and bias, pitched outputs.

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


@pytest.mark.parametrize("M,N,K,K2", [(1, 8, 64, 0), (127, 64, 520, 16), (128, 264, 512, 64), (129, 136, 1000, 48), (300, 520, 4096, 8), (257, 200, 768, 768)])
@pytest.mark.parametrize("layout,layout2", [("nk", "nk"), ("kn", "kn"), ("nk", "kn"), ("kn", "nk")])
def test_split_products_match_fp32(M, N, K, K2, layout, layout2):
    from opaque_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g, dtype=torch.bfloat16)      # noqa: E731
    a, w, bias = r(M, K), r(N, K), r(N)
    a2, w2 = (r(M, K2), r(N, K2)) if K2 else (None, None)
    prod = a.float() @ w.float().t() + (a2.float() @ w2.float().t() if K2 else 0.0)
    b = w if layout == "nk" else w.t().contiguous()
    b2 = None if not K2 else (w2 if layout2 == "nk" else w2.t().contiguous())
    st = ops.StatusWord()
    nk = -(-K // 64) + -(-K2 // 64)
    for splits in sorted({1, min(2, nk), min(3, nk), min(7, nk), min(24, nk), nk}):
        for alpha, bb in ((1.0, None), (0.5, bias)):
            kw = dict(b_layout=layout, a2=a2, b2=b2, b2_layout=layout2, bias=bb, kernel="single", splits=splits, alpha=alpha)
            got = ops.gemm(a, b, status=st, **kw)
            assert st.read() == 0 and _rel(got, alpha * prod + (0.0 if bb is None else bb.float())) < TOL, (splits, alpha)
            assert torch.equal(got, ops.gemm(a, b, **kw))
    auto = ops.gemm(a, b, b_layout=layout, a2=a2, b2=b2, b2_layout=layout2, bias=bias)
    assert _rel(auto, prod + bias.float()) < TOL


def test_split_products_write_inside_a_pitched_output_only():
    from opaque_b200 import ops
    a, w = torch.randn(130, 256, device="cuda", dtype=torch.bfloat16), torch.randn(72, 256, device="cuda", dtype=torch.bfloat16)
    for pitch in (80, 75):                               # rows for vector stores and rows that need scalar stores
        buf = torch.full((130, pitch), 7.0, device="cuda", dtype=torch.bfloat16)
        ops.gemm(a, w, out=buf[:, :72], kernel="single", splits=4)
        assert _rel(buf[:, :72], a.float() @ w.float().t()) < TOL and bool((buf[:, 72:] == 7.0).all())


def test_split_argument_errors():
    from opaque_b200 import ops
    a, w = torch.randn(64, 128, device="cuda", dtype=torch.bfloat16), torch.randn(64, 128, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(ops.KernelLibraryError):
        ops.gemm(a, w, kernel="single", splits=3)        # two k-blocks
    with pytest.raises(ValueError):
        ops.gemm(a, w, kernel="pair", alpha=2.0)


def test_small_products_are_split_and_large_ones_are_not():
    from opaque_b200 import ops
    for M, N, K in [(1, 768, 3072), (128, 768, 50304), (130, 48, 4096), (256, 2048, 8192)]:
        kernel, splits = ops.pick_gemm_plan(M, N, K)
        assert kernel == "single" and splits > 1
    for M, N, K in [(16384, 4096, 4096), (16384, 2304, 768), (8192, 128256, 4096)]:
        assert ops.pick_gemm_plan(M, N, K) == (ops.pick_gemm_kernel(M, N, K), 1)


def test_lora_operands_packed_in_one_launch():
    from opaque_b200 import ops
    for r, d, outs in ((8, 8, (8, 16, 24)), (16, 200, (64, 8, 8)), (32, 72, (40, 40, 136))):
        f = [(torch.randn(r, d, device="cuda", dtype=torch.bfloat16), torch.randn(o, r, device="cuda", dtype=torch.bfloat16)) for o in outs]
        a, b = ops.lora_pack(f)
        assert torch.equal(a, torch.cat([x for x, _ in f])) and torch.equal(b, torch.block_diag(*[y for _, y in f]))


@pytest.mark.parametrize("M,N,K,splits", [(1, 8, 8, 1), (128, 64, 64, 1), (130, 72, 1000, 1), (130, 72, 1000, 5), (257, 328, 136, 2), (64, 16, 2048, 8),
                                          (20000, 56, 72, 1)])
def test_narrow_tiles(M, N, K, splits):
    from opaque_b200 import ops
    torch.manual_seed(M + N)
    a, bias = torch.randn(M, K, device="cuda", dtype=torch.bfloat16), torch.randn(N, device="cuda", dtype=torch.bfloat16)
    a2 = torch.randn(M, 16, device="cuda", dtype=torch.bfloat16)
    for layout, layout2 in (("nk", "kn"), ("kn", "nk")):
        w = torch.randn((N, K) if layout == "nk" else (K, N), device="cuda", dtype=torch.bfloat16)
        b2 = torch.randn((N, 16) if layout2 == "nk" else (16, N), device="cuda", dtype=torch.bfloat16)
        prod = a.float() @ (w.float().t() if layout == "nk" else w.float()) + a2.float() @ (b2.float().t() if layout2 == "nk" else b2.float())
        buf = torch.full((M, N + 8), 7.0, device="cuda", dtype=torch.bfloat16)
        kw = dict(b_layout=layout, a2=a2, b2=b2, b2_layout=layout2, bias=bias, alpha=0.5, kernel="single", splits=splits)
        ops.gemm(a, w, out=buf[:, :N], block_n=64, **kw)
        assert _rel(buf[:, :N], 0.5 * prod + bias.float()) < TOL and bool((buf[:, N:] == 7.0).all())
        # a tile's k-blocks are added in the same order whatever its width
        assert torch.equal(buf[:, :N], ops.gemm(a, w, block_n=256, **kw))
    with pytest.raises(ops.KernelLibraryError):
        ops.gemm(a, w, b_layout="kn", kernel="single", block_n=128)


def test_tile_width_follows_the_number_of_narrow_tiles():
    from opaque_b200 import ops
    assert ops.pick_tile_width(10 ** 6, 64, 2) == 64 and ops.pick_tile_width(128, 768, 12) == 64 and ops.pick_tile_width(128, 768, 48, 12) == 64
    assert ops.pick_tile_width(2048, 768, 12) == 256 and ops.pick_tile_width(16384, 3072, 12) == 256 and ops.pick_tile_width(128, 50304, 12) == 256
