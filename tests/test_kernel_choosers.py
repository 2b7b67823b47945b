"""Shape-based choices between kernel variants (pure functions: no GPU needed)."""
from opaque_b200 import ops


def test_gemm_plan_takes_the_kernel_that_measured_faster():
    # both sides of the crossover in width at 3663 rows, and in size: (pair, single) us 18.7 / 20.5 and 10.3 / 9.3, 42.1 / 27.3 and 167 / 182
    assert ops.pick_gemm_plan(3663, 3072, 768) == "pair" and ops.pick_gemm_plan(3663, 768, 768) == "single"
    assert ops.pick_gemm_plan(256, 2048, 8192) == "single" and ops.pick_gemm_plan(8192, 4096, 4096) == "pair"
    # large products run on pairs at any K, products of few tiles on single CTAs
    for shape in [(16384, 4096, 4096), (16384, 14336, 4096), (16384, 4096, 14336), (16384, 2304, 768), (16384, 768, 3072)]:
        assert ops.pick_gemm_plan(*shape) == "pair", shape
    for shape in [(1, 8, 64), (128, 768, 768), (2048, 512, 4096), (16384, 48, 4096)]:
        assert ops.pick_gemm_plan(*shape) == "single", shape
    # a second K segment counts as its k-blocks
    assert ops.pick_gemm_plan(3663, 768, 704, 64) == ops.pick_gemm_plan(3663, 768, 768)


def test_tile_width_of_the_single_cta_kernel():
    assert ops.pick_tile_width(16384, 48, 64) == 64 and ops.pick_tile_width(16384, 64, 64) == 64      # one narrow tile covers the columns
    assert ops.pick_tile_width(128, 768, 12) == 64 and ops.pick_tile_width(128, 2048, 128) == 64      # all narrow tiles at once, and faster
    assert ops.pick_tile_width(3663, 768, 12) == 256                                                  # beyond one wave


def test_plan_code_is_the_plan_and_knows_activations(monkeypatch):
    monkeypatch.setattr(ops.lib, "sm_count", lambda *a: 148)
    for shape in [(3663, 3072, 768), (3663, 768, 768), (128, 768, 768), (16384, 768, 3072), (512, 256, 64), (1, 8, 64)]:
        code = ops._plan_code(*shape, 0, 0)
        assert (code == 0) == (ops.pick_gemm_plan(*shape) == "pair")
        assert code in (0, ops.pick_tile_width(shape[0], shape[1], -(-shape[2] // 64)))
        assert ops._plan_code(*shape, 0, 1) == ops.pick_tile_width(shape[0], shape[1], -(-shape[2] // 64))      # single CTAs only
    # with an activation: 64-column tiles for few rows, pairs from where they measured faster (1285 rows: 14.2 us against 19.0)
    assert [ops._plan_code(rows, 3072, 768, 0, 2) for rows in (128, 512, 1285, 3663, 16384)] == [64, 64, 0, 0, 0]


def test_gated_backward_runs_in_the_epilogue_beyond_one_wave():
    assert not ops.pick_glu_bwd(128, 8192) and not ops.pick_glu_bwd(597, 5632)
    assert ops.pick_glu_bwd(1024, 14336) and ops.pick_glu_bwd(5439, 8192)
    assert not ops.pick_glu_bwd(256, 74 * 256) and ops.pick_glu_bwd(256, 74 * 256 + 1)                # 74 SM pairs


def test_norm_path_choice_crosses_over_with_sequence_length():
    # Gram matrices cost T^2 (d_in + d_out), the product 2 T d_in d_out: short sequences on big layers take the Gram form
    assert ops.pick_norm_path(512, 768, 768) == "ghost"
    assert ops.pick_norm_path(1024, 4096, 4096) == "ghost"
    assert ops.pick_norm_path(1024, 2048, 8192) == "ghost"
    # long sequences on small layers take the product
    assert ops.pick_norm_path(4096, 128, 256) == "direct"
    assert ops.pick_norm_path(2048, 768, 768) == "direct"
    # the product kernel needs examples of a multiple of 64 rows
    assert ops.pick_norm_path(4100, 128, 256) == "ghost"
    # monotone in T for a fixed layer
    seen_direct = False
    for t in range(64, 8192 + 1, 64):
        path = ops.pick_norm_path(t, 1024, 1024)
        assert not (seen_direct and path == "ghost")
        seen_direct = seen_direct or path == "direct"
    assert seen_direct
