"""Routed experts around the number of (token, choice) rows from which they run as tensor-core tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("tokens,top,E", [(5, 4, 8), (23, 1, 4), (12, 2, 16), (6, 4, 32), (25, 1, 3), (20, 3, 5)])
@pytest.mark.parametrize("kind", ["clamped_sigmoid", "relu2"])
def test_tiles_and_rows_agree(tokens, top, E, kind):
    """Both ways against float64, with an addend; the rule sends a step to the tiles from 24 rows on."""
    from dotllm_b200.kernels import library, ops
    K, ff = 256, 128
    g = torch.Generator().manual_seed(tokens)
    make = lambda *s, scale=1.0: (torch.randn(*s, generator=g) * scale).to(torch.bfloat16).to(DEV)
    halves = 1 if kind in ops.UNGATED else 2
    x, w_in, w_out = make(tokens, K), make(E, halves * ff, K, scale=0.06), make(E, K, ff, scale=0.09)
    ids = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(tokens)]).to(torch.int32).to(DEV)
    weights = torch.rand(tokens, top, generator=g).to(DEV)
    addend = torch.randn(tokens, K, generator=g).to(DEV)
    assert ops.experts_grouped_takes(x, ids, w_in, w_out) == (tokens * top >= 24)
    want = addend.double().clone()
    for t in range(tokens):
        for j in range(top):
            e = int(ids[t, j])
            z = w_in[e].double() @ x[t].double()
            if kind == "relu2":
                h = z.clamp(min=0).square()
            else:
                a, b = z[:ff].clamp(max=1.5), z[ff:].clamp(-1.5, 1.5)
                h = a * torch.sigmoid(1.702 * a) * (b + 1)
            want[t] += weights[t, j].double() * (w_out[e].double() @ h)
    tiles = ops.experts_grouped(x, ids, weights, w_in, w_out, kind, 1.5, 1.702, addend=addend)
    rows = ops.expert_down(ops.expert_gate_up(x, ids, w_in, kind, 1.5, 1.702), ids, weights, w_out, addend=addend)
    library.check_status()
    for got in (tiles, rows):
        # the intermediate rows are rounded to bfloat16 (2^-9 each, independent over ff of them): relative to the result's size
        assert float((got.double() - want).norm() / want.norm()) < 2.0 ** -8
