"""What a capture keeps alive until the backward pass is over."""
import pytest
import torch

from opaque_b200 import ops
from opaque_b200.engine import fused


def _capture(batch):
    cap = object.__new__(fused.Capture)
    cap.batch_size, cap.sum_jobs, cap.sum_held = batch, [], 0
    return cap


@pytest.mark.parametrize("rows,cols,layers", [(4096, 8192, 3), (4096, 4096, 3), (1024, 4096, 40), (4096, 1024, 40), (3663, 768, 40), (64, 768, 70),
                                              (4097, 64, 3), (4104, 1024, 2)])
def test_waiting_norm_sums_hold_a_bounded_number_of_bytes(monkeypatch, rows, cols, layers):
    done, peak = [], 0
    monkeypatch.setattr(ops.functional, "rows_sum_batch_", lambda jobs, n: done.extend(j[0] for j in jobs))
    monkeypatch.setattr(ops.functional, "rows_group_sum_", lambda out, *a, **k: done.append(out))
    cap = _capture(1)
    g = torch.empty(rows, cols, dtype=torch.bfloat16)
    for i in range(layers):
        cap.add_row_sums(i, g, g, None, None, None)
        waiting = sum(j[1].nbytes + j[2].nbytes for j in cap.sum_jobs)
        assert waiting == cap.sum_held
        peak = max(peak, waiting)
    assert peak <= 256 << 20
    if rows > 4096 or rows * cols > 4 << 20:
        assert peak == 0                      # wide or long matrices wait for nothing
    cap._launch_sums()
    assert sorted(done) == list(range(layers)) and not cap.sum_jobs and cap.sum_held == 0

