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


@pytest.mark.parametrize("tokens,top,E,K,ff,N", [(1, 1, 1, 8, 8, 8), (1, 4, 40, 264, 24, 136), (5, 3, 7, 520, 148 * 8 + 8, 160), (8, 2, 16, 2048, 512, 2048),
                                                 (8, 16, 20, 136, 40, 296), (9, 4, 33, 1024, 2376, 264), (16, 8, 300, 256, 72, 2376), (16, 1, 3, 392, 4744, 7120),
                                                 (12, 2, 5, 128, 264, 4744)])
def test_chosen_experts_read_once(tokens, top, E, K, ff, N, monkeypatch):
    """The kernels that read each chosen expert once, against float64: edges of a block's rows, tiles and passes, more rows of one expert than an instruction
    has columns (a token may name an expert twice), ids without matrices, identity experts, no weights; and a token's bits do not depend on
    the others.  Bounds: float32 sums of K products of bfloat16 (K / 16 additions deep), h rounded to bfloat16 once."""
    from dotllm_b200.kernels import library, ops
    monkeypatch.setattr(ops, "EXPERT_ROWS_MB", (0.0, 0.0))
    g = torch.Generator().manual_seed(tokens * 31 + K)
    make = lambda *s, scale=1.0: (torch.randn(*s, generator=g) * scale).to(torch.bfloat16).to(DEV)
    x, w_in, w_out, other = make(tokens, K), make(E, 2 * ff, K, scale=0.06), make(E, N, ff, scale=0.09), make(tokens, N)
    ids = torch.randint(0, E + 2, (tokens, top), generator=g).to(torch.int32)
    if tokens > 4:
        ids[:, 0] = 0                                        # one expert for every token
        ids[2, -1] = -1
    ids = ids.to(DEV)
    weights, addend, gate = torch.rand(tokens, top, generator=g).to(DEV), torch.randn(tokens, N, generator=g).to(DEV), torch.randn(tokens, 3, generator=g).to(DEV)
    assert ops.experts_by_rows(x, ids, w_in, w_out, "silu")
    h = ops.expert_gate_up(x, ids, w_in, "clamped_sigmoid", 1.5, 1.702)
    flat = ids.flatten().tolist()
    for r, e in enumerate(flat):
        if not 0 <= e < E:
            assert (h[r] == 0).all()
            continue
        z = w_in[e].double() @ x[r // top].double()
        size = (K / 16 + 16) * 2.0 ** -24 * (w_in[e].double().abs() @ x[r // top].double().abs())
        a, b = z[:ff].clamp(max=1.5), z[ff:].clamp(-1.5, 1.5)
        want = a * torch.sigmoid(1.702 * a) * (b + 1)
        # |d/da a sigmoid(1.702 a)| <= 1.1, |b + 1| <= 2.5, |a sigmoid| <= 1.5
        assert ((h[r].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.75 * size[:ff] + 1.5 * size[ff:] + 1e-6).all()
    for kw in (dict(weights=weights, addend=addend, addend_gate=gate, identity=(other, 1)), dict(weights=None), dict(weights=weights, addend=addend)):
        got = ops.expert_down(h, ids, kw.get("weights"), w_out, addend=kw.get("addend"), addend_gate=kw.get("addend_gate"), identity=kw.get("identity"), read_once=True)
        want, bound = torch.zeros(tokens, N, dtype=torch.float64, device=DEV), torch.zeros(tokens, N, dtype=torch.float64, device=DEV)
        if "addend" in kw:
            want += addend.double() * (torch.sigmoid(gate[:, :1].double()) if "addend_gate" in kw else 1.0)
        for r, e in enumerate(flat):
            f = weights.flatten()[r].double() if kw["weights"] is not None else 1.0
            if 0 <= e < E:
                want[r // top] += f * (w_out[e].double() @ h[r].double())
                bound[r // top] += f * (w_out[e].double().abs() @ h[r].double().abs())
            elif e == E and "identity" in kw:
                want[r // top] += f * other[r // top].double()
        assert ((got.double() - want).abs() <= (ff / 16 + 16 + top) * 2.0 ** -24 * (bound + want.abs()) + 1e-5 * want.abs() + 1e-6).all()
        alone = ops.expert_down(h[-top:].contiguous(), ids[-1:].contiguous(), kw["weights"][-1:].contiguous() if kw["weights"] is not None else None, w_out,
                                addend=addend[-1:].contiguous() if "addend" in kw else None, addend_gate=gate[-1:] if "addend_gate" in kw else None,
                                identity=(other[-1:], 1) if "identity" in kw else None, read_once=True)
        assert torch.equal(alone, got[-1:])
    assert torch.equal(ops.expert_gate_up(x[-1:].contiguous(), ids[-1:].contiguous(), w_in, "clamped_sigmoid", 1.5, 1.702), h[-top:])
    library.check_status()


@pytest.mark.parametrize("tokens,top,E,K,ff,once", [(8, 2, 16, 2048, 2048, True), (16, 2, 16, 2048, 2048, True), (17, 2, 16, 2048, 2048, False), (8, 4, 32, 2048, 768, True),
                                                    (9, 4, 32, 2048, 768, False), (8, 2, 16, 1024, 512, False), (16, 9, 16, 2048, 2048, False)])
def test_experts_read_once_where_it_pays(tokens, top, E, K, ff, once):
    """Experts of some size and steps of few tokens; never an activation of one product, a row scale or unaligned rows."""
    from dotllm_b200.kernels import ops
    x, ids = torch.empty(tokens, K, dtype=torch.bfloat16, device=DEV), torch.zeros(tokens, top, dtype=torch.int32, device=DEV)
    w_in, w_out = (torch.empty(s, dtype=torch.bfloat16, device=DEV) for s in ((E, 2 * ff, K), (E, K, ff)))
    assert ops.experts_by_rows(x, ids, w_in, w_out, "silu") == once
    assert not ops.experts_by_rows(x, ids, w_in, w_out, "relu2") and not ops.experts_by_rows(x, ids, w_in, w_out, "silu", row_scale=x)
    odd = torch.empty(tokens, K + 1, dtype=torch.bfloat16, device=DEV)[:, 1:]
    assert not ops.experts_by_rows(odd, ids, w_in, w_out, "silu")


@pytest.mark.parametrize("tokens,top,E,ff,N", [(1, 2, 4, 2048, 2048), (8, 2, 8, 768, 2048), (8, 1, 4, 8192, 2048), (16, 4, 8, 2048, 4096), (5, 1, 2, 14336, 4096),
                                               (16, 1, 3, 1408, 7104)])
def test_sums_of_chosen_experts_keep_float32(tokens, top, E, ff, N, monkeypatch):
    """The float32 results of experts read once are as near the exact sums as those of the kernel that goes row by row (chains of float32 multiply-adds).
    A chain of m rounded additions is sqrt(m / 2) 2^-24 / sqrt(3) off (the partial sums grow as a random walk), a tree of m sqrt(log2 m) of it: at
    most 4 for the widest here, so 2^-22 would be a chain that drifts; the kernels differ by a quarter at most."""
    from dotllm_b200.kernels import library, ops
    g = torch.Generator().manual_seed(ff + N)
    h = torch.randn(tokens * top, ff, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(E, N, ff, generator=g) * 0.02).to(torch.bfloat16).to(DEV)
    ids = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(tokens)]).to(torch.int32).to(DEV)
    weights = torch.rand(tokens, top, generator=g).to(DEV)
    want = torch.stack([sum(weights[t, j].double() * (w[int(ids[t, j])].double() @ h[t * top + j].double()) for j in range(top)) for t in range(tokens)])
    error = {}
    for name, limit in (("once", 0.0), ("by rows", float("inf"))):
        monkeypatch.setattr(ops, "EXPERT_ROWS_MB", (limit, limit))
        got = ops.expert_down(h, ids, weights, w, read_once=True)
        error[name] = float((got.double() - want).norm() / want.norm())
    library.check_status()
    assert error["once"] < 1.25 * error["by rows"] and error["once"] < 2.0 ** -22, error


@pytest.mark.parametrize("tokens,top,ff,N,E,once", [(1, 1, 768, 2048, 8, False), (8, 1, 768, 2048, 8, False), (8, 1, 1024, 2048, 64, False), (8, 1, 1408, 2048, 16, True),
                                                    (8, 2, 704, 2048, 64, False), (2, 2, 512, 4096, 128, False), (1, 4, 768, 2048, 32, True), (8, 2, 768, 2048, 32, True),
                                                    (8, 2, 664, 2048, 32, False), (1, 2, 1024, 2048, 16, False), (2, 2, 1024, 2048, 16, True),
                                                    (9, 2, 1024, 2048, 16, False), (9, 2, 1408, 2048, 16, True), (9, 1, 1408, 2048, 16, True)])
def test_down_products_read_once_where_that_pays(tokens, top, ff, N, E, once, monkeypatch):
    """Whatever came before them (a gate or none, weights on the way in): by the down matrices' own size, and short sums row by row."""
    from dotllm_b200.kernels import library, ops
    called = []
    real = library.call
    monkeypatch.setattr(library, "call", lambda name, *a: (called.append(name), real(name, *a))[1])
    h, w = torch.zeros(tokens * top, ff, dtype=torch.bfloat16, device=DEV), torch.zeros(E, N, ff, dtype=torch.bfloat16, device=DEV)
    ids = torch.zeros(tokens, top, dtype=torch.int32, device=DEV)
    assert (ops.expert_down(h, ids, None, w) == 0).all()
    assert called == ["dl_expert_down_rows" if once else "dl_expert_down"]


@pytest.mark.parametrize("tokens,top,ff,K,E,once", [(6, 8, 700, 2048, 16, False), (6, 8, 704, 2048, 16, True), (8, 2, 512, 4096, 32, False), (4, 2, 512, 4096, 32, True),
                                                    (8, 2, 600, 4096, 32, True), (8, 2, 512, 6144, 16, True)])
def test_gate_up_products_read_once_where_that_pays(tokens, top, ff, K, E, once, monkeypatch):
    from dotllm_b200.kernels import library, ops
    called = []
    real = library.call
    monkeypatch.setattr(library, "call", lambda name, *a: (called.append(name), real(name, *a))[1])
    x, w = torch.zeros(tokens, K, dtype=torch.bfloat16, device=DEV), torch.zeros(E, 2 * ff, K, dtype=torch.bfloat16, device=DEV)
    ids = torch.zeros(tokens, top, dtype=torch.int32, device=DEV)
    assert (ops.expert_gate_up(x, ids, w, "silu") == 0).all()
    assert called == ["dl_expert_gate_up_rows" if once else "dl_expert_gate_up"]


@pytest.mark.parametrize("tokens,top,E,K,ff,N", [(16, 8, 64, 4096, 1024, 2048), (8, 16, 128, 1024, 1408, 4736), (16, 1, 16, 2048, 9472, 2048)])
def test_chosen_experts_repeat_with_full_rings(tokens, top, E, K, ff, N, monkeypatch):
    """Many entries, of several passes in the last, with every column of the instructions in use: slots are refilled the moment they are released, and 30
    launches give the bits of the first, which are near the exact ones (a slot released before its reads are done shows as wrong columns)."""
    from dotllm_b200.kernels import library, ops
    monkeypatch.setattr(ops, "EXPERT_ROWS_MB", (0.0, 0.0))
    g = torch.Generator(device=DEV).manual_seed(E)
    make = lambda *s: (torch.randn(*s, generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    x, w_in, w_out = make(tokens, K), make(E, 2 * ff, K), make(E, N, ff)
    ids = torch.stack([torch.randperm(E, generator=g, device=DEV)[:top] for _ in range(tokens)]).to(torch.int32)
    weights = torch.rand(tokens, top, generator=g, device=DEV)
    assert ops.experts_by_rows(x, ids, w_in, w_out, "silu")
    h = ops.expert_gate_up(x, ids, w_in, "silu")
    y = ops.expert_down(h, ids, weights, w_out, read_once=True)
    flat = ids.flatten().tolist()
    z = torch.stack([w_in[e].double() @ x[r // top].double() for r, e in enumerate(flat)])
    want_h = torch.nn.functional.silu(z[:, :ff]) * z[:, ff:]
    assert float((h.double() - want_h).norm() / want_h.norm()) < 2.0 ** -8       # rounded once to bfloat16
    want = (weights.flatten()[:, None].double() * torch.stack([w_out[e].double() @ h[r].double() for r, e in enumerate(flat)])).view(tokens, top, N).sum(1)
    assert float((y.double() - want).norm() / want.norm()) < 2.0 ** -22          # float32 sums (test_sums_of_chosen_experts_keep_float32)
    for _ in range(30):
        again = ops.expert_gate_up(x, ids, w_in, "silu")
        assert torch.equal(again, h) and torch.equal(ops.expert_down(again, ids, weights, w_out, read_once=True), y)
    library.check_status()
