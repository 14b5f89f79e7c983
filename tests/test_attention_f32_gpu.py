"""The float32 attention kernels against float64: prompts, a few new tokens, and the same bits from both."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
PAGE = 64


class Case:
    """Sequences of given lengths over scattered pages, NaN in every place that holds no token, and one query row per token."""

    def __init__(self, lens, nh, nkv, hd, seed=0):
        g = torch.Generator().manual_seed(seed)
        self.lens, self.nh, self.nkv, self.hd = lens, nh, nkv, hd
        need = [-(-n // PAGE) for n in lens]
        order = torch.randperm(sum(need) + 2, generator=g).tolist()
        self.table = torch.full((len(lens), max(need) + 1), -1, dtype=torch.int32)
        k_pool, v_pool = torch.full((len(order), nkv, PAGE, hd), float("nan")), torch.full((len(order), nkv, hd, PAGE), float("nan"))
        self.q, self.k, self.v = [], [], []
        for b, n in enumerate(lens):
            k, v = torch.randn(n, nkv, hd, generator=g), torch.randn(n, nkv, hd, generator=g)
            self.q.append(torch.randn(n, nh, hd, generator=g).to(DEV))
            self.k.append(k.to(DEV))
            self.v.append(v.to(DEV))
            for p in range(need[b]):
                page, m = order.pop(), min(PAGE, n - PAGE * p)
                self.table[b, p] = page
                k_pool[page, :, :m] = k[PAGE * p:PAGE * p + m].permute(1, 0, 2)
                v_pool[page, :, :, :m] = v[PAGE * p:PAGE * p + m].permute(1, 2, 0)
        self.table, self.k_pool, self.v_pool = self.table.to(DEV), k_pool.to(DEV), v_pool.to(DEV)

    def run(self, starts, news, gates=None, **kw):
        """The rows of tokens starts[b] .. starts[b] + news[b] - 1 of every sequence, through ``ops.attention`` with the step's plan."""
        from dotllm_b200.engine.step import AttentionPlan
        from dotllm_b200.kernels import library, ops
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
        totals = [s + n for s, n in zip(starts, news)]
        cu = [0]
        for n in news:
            cu.append(cu[-1] + n)
        plan = AttentionPlan(len(news), max(news), max(totals), all(n == 1 for n in news), i32(starts), i32(news), i32(cu), i32(totals),
                             list(starts), list(news))
        rows = lambda parts: torch.cat([x[s:s + n] for x, s, n in zip(parts, starts, news)])
        q = rows(self.q).reshape(cu[-1], -1).contiguous()
        if gates is not None:
            kw["gate"] = rows(gates).contiguous()
        out = ops.attention(q, self.k_pool, self.v_pool, i32([b for b, n in enumerate(news) for _ in range(n)]),
                            i32([s + i for s, n in zip(starts, news) for i in range(n)]), self.table, self.nh, self.nkv, self.hd,
                            kw.pop("scale", self.hd ** -0.5), plan=plan, **kw)
        library.check_status()
        return list(out.split(news))

    def exact(self, b, window=0, keep_first=0, sinks=None, hook=None, gates=None):
        n, G = self.lens[b], self.nh // self.nkv
        at = torch.arange(n, device=DEV)
        d = at[None, :] - at[:, None]
        seen = d <= 0
        if window:
            seen &= (d > -window) | (at[None, :] < keep_first)
        q, k, v = self.q[b].double(), self.k[b].double(), self.v[b].double()
        s = torch.einsum("thd,shd->hts", q, k.repeat_interleave(G, 1)) * self.hd ** -0.5
        if hook is not None and hook.softcap > 0:
            s = hook.softcap * torch.tanh(s / hook.softcap)
        if hook is not None and hook.slopes is not None:
            s = s + hook.slopes.double()[:, None, None] * d
        s = s.masked_fill(~seen, -math.inf)
        if sinks is not None:
            s = torch.cat([s, sinks.double()[:, None, None].expand(-1, n, 1)], dim=-1)
        w = torch.softmax(s, dim=-1)[..., :n]
        o = torch.einsum("hts,shd->thd", w, v.repeat_interleave(G, 1))
        if gates is not None:
            o = o * torch.sigmoid(gates[b].double())[..., None]
        return o.reshape(n, -1)


def options(name, nh):
    from dotllm_b200.kernels import ops
    g = torch.Generator().manual_seed(11)
    vec = lambda s: (torch.randn(nh, generator=g) * s).to(DEV)
    return {"plain": {}, "window": dict(window=70), "wide window": dict(window=300, keep_first=5),
            "kept and sinks": dict(window=129, keep_first=66, sinks=vec(2.0)), "sinks": dict(sinks=vec(2.0)),
            "capped": dict(score_hook=ops.ScoreHook(3.0)), "slopes": dict(score_hook=ops.ScoreHook(0.0, vec(0.1))),
            "capped slopes": dict(score_hook=ops.ScoreHook(2.0, vec(0.05)))}[name]


def bound(n, hook):
    """Weights that sum to one, values of up to 5: 5 times the relative error of a weight, which is the absolute error of its score
    (twice: the row's maximum is subtracted) and the exponential's.  Scores of up to 8 are off by about 1e-6; a penalty of size
    slope * distance adds two roundings at that size."""
    far = float(hook.slopes.abs().max()) * n if hook is not None and hook.slopes is not None else 0.0
    return 1e-5 + 5 * 2 * 2 * far * 2.0 ** -24


@pytest.mark.parametrize("nh,nkv,hd", [(8, 2, 64), (3, 3, 128), (16, 1, 128), (8, 1, 64), (10, 2, 64)])
@pytest.mark.parametrize("name", ["plain", "window", "wide window", "kept and sinks", "sinks", "capped", "slopes", "capped slopes"])
def test_prompts_and_tokens(nh, nkv, hd, name):
    from dotllm_b200.kernels import ops
    lens = [1, 64, 65, 257, 700]
    case, kw = Case(lens, nh, nkv, hd), options(name, nh)
    gates = [torch.randn(n, nh, generator=torch.Generator().manual_seed(7 + n)).to(DEV) for n in lens] if name in ("plain", "sinks") else None
    whole = case.run([0] * 5, lens, gates=gates, **kw)
    hook = kw.get("score_hook")
    for b in range(5):
        want = case.exact(b, kw.get("window", 0), kw.get("keep_first", 0), kw.get("sinks"), hook, gates)
        assert float((whole[b].double() - want).abs().max()) < bound(lens[b], hook), b
    # a portion of a prompt, a few tokens and one token: the same bits, through either kernel
    for news in ([1, 30, 40, 150, 333], [1, 8, 3, 5, 8], [1, 1, 1, 1, 1]):
        starts = [n - m for n, m in zip(lens, news)]
        got = case.run(starts, news, gates=gates, **kw)
        for b in range(5):
            assert torch.equal(got[b], whole[b][starts[b]:]), (news, b)


def test_a_later_value_that_is_no_number_stays_unseen():
    """Rows of a tile that do not see a token are not touched by an infinity among its values."""
    case = Case([200], 4, 2, 64, seed=3)
    clean = case.run([0], [200])[0]
    page = int(case.table[0, 2])
    case.v_pool[page, 0, 5, 140 % PAGE] = float("inf")
    got = case.run([0], [200])[0]
    assert torch.equal(got[:140], clean[:140]) and bool(torch.isinf(got[140:, 5]).all())
    assert torch.equal(case.run([139], [1])[0], clean[139:140]) and torch.equal(case.run([130], [70])[0], got[130:])


@pytest.mark.parametrize("what", ["newest key", "page of keys", "first page of keys", "query", "page beyond the window", "scores of -inf", "first scores of -inf"])
@pytest.mark.parametrize("with_sinks", [False, True])
def test_keys_and_queries_that_are_no_numbers(what, with_sinks):
    """A NaN among the visible scores makes the output NaN, through either kernel, and nothing else does: exactly where float64 says so.
    A page whose scores are all -inf has no weight beside others."""
    nan, inf = float("nan"), float("inf")
    case = Case([193, 260], 8, 2, 64, seed=8)                  # the first one's newest key is a page's only one
    kw = dict(sinks=torch.linspace(-1, 1, 8, device=DEV)) if with_sinks else {}
    if what == "page beyond the window":
        kw["window"] = 70

    def put(b, lo, hi, channels, value):                       # keys of the first KV head
        case.k[b][lo:hi, 0, channels] = value
        for at in range(lo, hi):
            case.k_pool[int(case.table[b, at // PAGE]), 0, at % PAGE, channels] = value

    if what == "newest key":
        put(0, 192, 193, slice(None), nan)
        put(1, 256, 257, slice(None), nan)
    elif what == "page of keys":
        put(0, 64, 128, slice(5, 6), nan)
        put(1, 128, 192, slice(None), nan)
    elif what in ("first page of keys", "page beyond the window"):
        put(0, 0, 64, slice(None), nan)
        put(1, 0, 64, slice(None), nan)
    elif what == "query":
        case.q[0][192, 3] = nan
        case.q[1][258, 0, 7] = nan
    else:
        page = 0 if what.startswith("first") else 64
        for b in (0, 1):
            case.q[b][:, :, 0] = 1.0
            put(b, page, page + 64, slice(0, 1), -inf)
    whole = case.run([0, 0], [193, 260], **kw)
    few = case.run([192, 257], [1, 3], **kw)
    for b in (0, 1):
        want = case.exact(b, kw.get("window", 0), sinks=kw.get("sinks"))
        assert bool(torch.isnan(want).any()) == (what != "scores of -inf" and (what != "first scores of -inf" or not with_sinks))
        assert torch.equal(torch.isnan(whole[b]), torch.isnan(want)), b
        fine = ~torch.isnan(want)
        assert float((whole[b].double() - want)[fine].abs().max()) < bound(260, None)
        assert torch.equal(few[b].nan_to_num(nan=9.0), whole[b][-few[b].shape[0]:].nan_to_num(nan=9.0)), b


def test_longer_tables():
    """Columns of a table beyond a sequence's pages change nothing."""
    case = Case([100, 30], 8, 2, 64, seed=4)
    short = case.run([99, 29], [1, 1])
    case.table = torch.cat([case.table, torch.full((2, 30), -1, dtype=torch.int32, device=DEV)], dim=1).contiguous()
    assert all(torch.equal(a, b) for a, b in zip(short, case.run([99, 29], [1, 1])))


@pytest.mark.parametrize("tokens_at_once", [1, 2, 5])
def test_a_few_tokens_in_several_launches(monkeypatch, tokens_at_once):
    """Where the pages' parts of all tokens would take too much room, a launch takes as many tokens as fit: the same bits."""
    from dotllm_b200.kernels import attention_fast
    nh, hd = 8, 64
    lens, news = [100, 300, 64, 7], [3, 2, 1, 1]
    starts = [n - m for n, m in zip(lens, news)]
    case = Case(lens, nh, 2, hd, seed=5)
    gates = [torch.randn(n, nh, generator=torch.Generator().manual_seed(n)).to(DEV) for n in lens]
    whole = case.run(starts, news, gates=gates)
    monkeypatch.setattr(attention_fast, "F32_PARTS_BYTES", tokens_at_once * 4 * nh * case.table.shape[1] * (hd + 2) + 3)
    assert all(torch.equal(a, b) for a, b in zip(whole, case.run(starts, news, gates=gates)))


def test_blocks_that_walk_several_pages():
    """So many tokens and pages that a block takes more than one: the bits of the whole prompts."""
    case = Case([2500, 2450, 70, 2500, 1900], 4, 2, 64, seed=6)
    for kw in ({}, dict(window=700, keep_first=70)):
        whole = case.run([0] * 5, case.lens, **kw)
        starts = [n - 8 for n in case.lens]
        assert 2 * 40 * case.table.shape[1] > 16 * 148
        assert all(torch.equal(a, b[-8:]) for a, b in zip(case.run(starts, [8] * 5, **kw), whole))


def test_a_wide_table_costs_nothing():
    """Short sequences in a step whose tables are as wide as a long one's (a captured step keeps its width): the columns beyond cost no time."""
    n = 64
    case = Case([30] * n, 8, 8, 64, seed=7)

    def time():
        times = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            out = case.run([29] * n, [1] * n)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times), out                                 # (the host may be slow, the device is not slow by chance)

    narrow, out = time()
    case.table = torch.cat([case.table, torch.full((n, 2500), -1, dtype=torch.int32, device=DEV)], dim=1).contiguous()
    wide, got = time()
    print(f"observed: {narrow * 1e3:.0f} us, a table of 2,500 columns more {wide * 1e3:.0f} us")
    assert all(torch.equal(a, b) for a, b in zip(out, got))
    assert wide < narrow + 0.8                                 # (blocks for 1.3 million columns took 1.3 ms)
