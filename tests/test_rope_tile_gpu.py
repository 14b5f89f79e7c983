"""Rotation and cache write of many tokens at once (16 bytes a thread) against the kernel with one block per (token, head): both round every
product and sum explicitly, so their bits are equal."""
import pytest
import torch

import plain_llama

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,hd,rd,biases", [
    (3, 1, 64, 64, False),       # every channel rotated
    (4, 2, 128, 96, True),       # channels beyond the rotation, with biases
    (2, 1, 48, 16, False),       # fewer units than a batch holds; the query's channels beyond the rotation stay
    (2, 2, 112, 0, True),        # no rotation, biases alone
    (2, 1, 24, 8, False),        # float32 takes 16 bytes at a time, bfloat16 does not (8 channels are half a pair of units)
])
@pytest.mark.parametrize("tokens", [64, 65, 127, 300])
def test_tile_form_writes_what_the_token_form_writes(dtype, nh, nkv, hd, rd, biases, tokens):
    from dotllm_b200.kernels import ops
    g = torch.Generator().manual_seed(tokens)
    first = tokens // 3                                     # two sequences; the second starts inside a page
    seq = torch.tensor([0] * first + [1] * (tokens - first), dtype=torch.int32, device=DEV)
    pos = torch.tensor(list(range(first)) + list(range(37, 37 + tokens - first)), dtype=torch.int32, device=DEV)
    table = torch.tensor([[5, 0, 3, 9, 1, 10], [2, 8, 4, 11, 6, 7]], dtype=torch.int32, device=DEV)
    x = torch.randn(tokens, (nh + 2 * nkv) * hd, generator=g).to(dtype).to(DEV)
    cos, sin = (t.to(DEV) for t in plain_llama.rope_tables(range(512), rd, 10000.0)) if rd else (None, None)
    b = [torch.randn(n * hd, generator=g).to(DEV) for n in (nh, nkv, nkv)] if biases else None

    def run(cuts):
        y = x.clone()
        pools = [torch.zeros(12, nkv, 64, hd, dtype=dtype, device=DEV), torch.zeros(12, nkv, hd, 64, dtype=dtype, device=DEV)]
        for lo in range(0, tokens, cuts):
            s = slice(lo, lo + cuts)
            ops.rope_cache_write(y[s, :nh * hd], y[s, nh * hd:(nh + nkv) * hd], y[s, (nh + nkv) * hd:], cos, sin, rd, seq[s].contiguous(),
                                 pos[s].contiguous(), table, *pools, nh, nkv, hd, **({"biases": b} if b else {}))
        return y, *pools

    for got, want in zip(run(tokens), run(50)):             # runs of fewer than 64 tokens: a block per (token, head)
        assert torch.equal(got, want)
