"""Prompt attention's rows beyond a sequence's last: they hold the next sequence's queries, and leave no trace in this one's outputs."""
import math

import pytest
import torch

from test_kernels_gpu import DEV, _prefill_plan, dense_attention, make_paged, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("new,start", [(65, 0), (100, 200), (129, 3), (200, 0), (255, 64)])
def test_a_prompt_has_the_same_bits_whatever_follows_it(hd, window, new, start):
    nh, nkv = 4, 2
    lengths, news = [start + new, 140], [new, 140]
    k_pool, v_pool, table, dense = make_paged(2, lengths, nkv, hd, torch.bfloat16, seed=5)
    g = torch.Generator().manual_seed(6)
    q = torch.randn(sum(news), nh * hd, generator=g).to(torch.bfloat16)
    seq = torch.tensor([0] * new + [1] * 140, dtype=torch.int32, device=DEV)
    pos = torch.tensor(list(range(start, start + new)) + list(range(140)), dtype=torch.int32, device=DEV)
    scale = 1.0 / math.sqrt(hd)

    def run(q, n_seqs):
        n = sum(news[:n_seqs])
        return ops().attention(q[:n].to(DEV), k_pool.to(DEV), v_pool.to(DEV), seq[:n], pos[:n], table.to(DEV), nh, nkv, hd, scale, window,
                               plan=_prefill_plan(lengths[:n_seqs], news[:n_seqs]))[:new]

    alone = run(q, 1)
    loud = q.clone()
    loud[new:] = (loud[new:].float() * 1e4).to(torch.bfloat16)     # scores far above this sequence's, in rows of its tiles
    loud[new + 1::3] = float("inf")
    assert torch.equal(run(q, 2), alone)
    assert torch.equal(run(loud, 2), alone)
    want = torch.stack([dense_attention(q[t], *dense[0], nh, nkv, scale, start + t, window) for t in range(new)]).to(alone.device)
    # weights rounded to bfloat16 (half a step: 2^-9) for the product with the values, and the output's own rounding
    bound = 2 ** -9 * float(dense[0][1].abs().max()) + 1e-3 + 2 ** -8 * want.abs()
    assert bool(((alone.float() - want.float()).abs() <= bound).all())
