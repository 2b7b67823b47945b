"""The fused shard step with 4 coordinates per thread (parameters stay on this GPU) and with 8 (written through a peer table)
does the same arithmetic per coordinate: equal bits, for every remainder of the length and every noise form."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 7, 8, 1021, 4096, 100004])
@pytest.mark.parametrize("mode,nbuf,coef", [(0, 0, ()), (1, 4, (0.31, 0.18, 0.09, 0.04, 0.55, 0.85, 0.96, 0.995)),
                                            (1, 9, tuple([0.1] * 9 + [0.5] * 9)), (2, 3, (1.0, 0.4, 0.2, 0.1)), (3, 2, (1.0, -0.5, 0.2))])
def test_both_widths_give_the_same_bits(n, mode, nbuf, coef):
    from opaque_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(n)
    base = dict(grad=torch.randn(n, device="cuda", generator=gen), master=torch.randn(n, device="cuda", generator=gen),
                m=torch.randn(n, device="cuda", generator=gen), v=torch.rand(n, device="cuda", generator=gen))
    state = torch.randn(max(nbuf, 1), n, device="cuda", generator=gen)
    results = []
    for wide in (False, True):
        t = {k: x.clone() for k, x in base.items()}
        st, pl = state.clone(), torch.zeros(n + 16, device="cuda", dtype=torch.bfloat16)
        dest = dict(peer_params=torch.tensor([pl.data_ptr()], device="cuda", dtype=torch.int64)) if wide else dict(params_local=pl)
        no = torch.zeros(n, device="cuda")
        for step in (1, 2):
            t["grad"].copy_(base["grad"])
            ops.shard_step(**t, **dest, global_offset=8, seed=5 + step, noise_std=0.7, inv_normalize=0.25, lr=0.01, weight_decay=0.1,
                           step=step, ftrl_state=st if mode else None, ftrl_mode=mode, ftrl_coef=coef, nbuf=nbuf,
                           ring_head=step % nbuf if mode in (2, 3) else 0, noisy_out=no)
            assert not bool(t["grad"].any())
        assert not bool(pl[:8].any()) and not bool(pl[8 + n:].any())
        results.append([t["master"], t["m"], t["v"], st, pl, no])
    assert all(torch.equal(a, b) for a, b in zip(*results))
