"""Routed experts around the number of (token, choice) rows from which they run as tensor-core tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("tokens,top,E", [(5, 4, 8), (23, 1, 4), (12, 2, 16), (6, 4, 32), (25, 1, 3), (20, 3, 5)])
@pytest.mark.parametrize("kind", ["clamped_sigmoid", "relu2"])
def test_tiles_and_rows_agree(tokens, top, E, kind):
    """Both ways against float64, with an addend; the tiles are open to a step from 24 rows on."""
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


def step(tokens, top, E, K=512, ff=256, seed=0):
    g = torch.Generator().manual_seed(seed)
    make = lambda *s, scale=1.0: (torch.randn(*s, generator=g) * scale).to(torch.bfloat16).to(DEV)
    ids = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(tokens)]).to(torch.int32).to(DEV)
    return make(tokens, K), make(E, 2 * ff, K, scale=0.05), make(E, K, ff, scale=0.06), ids, torch.rand(tokens, top, generator=g).to(DEV)


@pytest.mark.parametrize("tokens,top,E,K,ff,tiles", [(8, 2, 16, 2048, 2048, False), (12, 2, 16, 2048, 2048, True), (12, 2, 16, 1024, 512, False), (32, 2, 16, 1024, 512, False),
                                                     (6, 4, 32, 4096, 2048, True), (6, 4, 32, 2048, 768, False), (24, 4, 32, 2048, 768, True),
                                                     (8, 6, 64, 2048, 1408, False), (3, 8, 128, 2048, 768, False), (16, 8, 128, 2048, 768, True),
                                                     (12, 8, 256, 2048, 768, False)])
def test_tiles_where_they_pay(tokens, top, E, K, ff, tiles):
    """Few rows that hardly share an expert, or small experts, go row by row; from 128 rows on all go as tiles."""
    from dotllm_b200.kernels import ops
    x, ids = torch.empty(tokens, K, dtype=torch.bfloat16, device=DEV), torch.zeros(tokens, top, dtype=torch.int32, device=DEV)
    w_in, w_out = (torch.empty(s, dtype=torch.bfloat16, device=DEV) for s in ((E, 2 * ff, K), (E, K, ff)))
    assert ops.experts_as_tiles(x, ids, w_in, w_out) == tiles


@pytest.mark.parametrize("tokens,top,E", [(3, 8, 256), (16, 8, 256), (1, 1, 40), (130, 1, 3), (43, 3, 5), (256, 1, 1)])
def test_tiles_for_the_experts_that_have_rows(tokens, top, E):
    """The rows are padded to tiles of the experts that can have any, and the result is the row kernels'."""
    from dotllm_b200.kernels import library, ops
    x, w_in, w_out, ids, weights = step(tokens, top, E, seed=tokens)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    tiles = ops.experts_grouped(x, ids, weights, w_in, w_out, "silu")
    peak = torch.cuda.max_memory_allocated() - before
    rows = ops.expert_down(ops.expert_gate_up(x, ids, w_in, "silu"), ids, weights, w_out)
    library.check_status()
    # both round the same intermediate rows to bfloat16; a sum that lies near a rounding's edge may fall to either side (2^-9 of one of 256)
    assert float((tiles - rows).norm() / rows.norm()) < 2.0 ** -8
    n = (tokens * top + 127 * min(E, tokens * top)) // 128
    assert peak < n * 128 * (2 * 512 + 2 * 256 + 4 * 512) + 4 * tokens * 512 + (2 << 20)          # (small buffers share segments of 2 MB)


@pytest.mark.parametrize("tokens", [32, 63, 64])
def test_scaled_rows_keep_their_digits(tokens):
    """An expert's input times its weight: row by row the product stays float32, and steps below 128 rows stay there."""
    from dotllm_b200.kernels import ops
    x, w_in, w_out, ids, weights = step(tokens, 2, 4, 2048, 1536)
    assert ops.experts_as_tiles(x, ids, w_in, w_out)
    assert ops.experts_as_tiles(x, ids, w_in, w_out, row_scale=weights) == (2 * tokens >= 128)
