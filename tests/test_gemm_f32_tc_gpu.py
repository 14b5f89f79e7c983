"""The float32 product on the tensor cores against float64, at the edges of its tiles, segments and cuts."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
U = 2.0 ** -24


def make(M, N, K, seed=0):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(M, K, generator=g).to(DEV), (torch.randn(N, K, generator=g) * 0.05).to(DEV)


def bound(x, w):
    """Of one output: the three products left out are each below 2^-25 of theirs (2 U in all); an accumulator of 256 k is truncated
    at most 16 times where the large products are summed (2 U each; the small ones' count 2^-8 of that), their sum rounds twice, and
    runs and segments add once each (U), all of partial sums that are no larger than sum |x w|."""
    runs = (x.shape[1] + 31) // 32                             # at least: a short segment's runs are short too
    return (2 + 33 + 2 + runs) * U * (x.abs().double() @ w.abs().double().T)


@pytest.mark.parametrize("M,N,K", [(1, 16, 256), (40, 20, 260), (1, 64, 512), (3, 130, 516), (16, 128, 2048), (17, 200, 544), (32, 64, 1000), (33, 96, 640), (64, 257, 768),
                                   (65, 128, 4096), (128, 300, 1024), (129, 128, 516), (300, 384, 1536), (5, 19000, 512), (700, 2500, 512)])
def test_against_float64(M, N, K):
    from dotllm_b200.kernels import gemm_f32_tc, library, ops
    x, w = make(M, N, K)
    assert gemm_f32_tc.takes(w)
    y = ops.linear(x, w)
    want = x.double() @ w.double().T
    err = (y.double() - want).abs()
    assert bool((err <= bound(x, w)).all()), float((err / bound(x, w)).max())
    # the bits of a row do not depend on the rows beside it, nor on the strides of x
    for m in sorted({1, min(M, 16), min(M, 17), min(M, 40), min(M, 70)}):
        assert torch.equal(ops.linear(x[M - m:], w), y[M - m:]), m
    wide = torch.full((M, K + 3), 7.0, device=DEV)
    wide[:, :K] = x
    assert torch.equal(ops.linear(wide[:, :K], w, resident=True), y)
    library.check_status()


def test_cuts_give_the_same_bits():
    """One matrix at row counts whose plans cut the segments differently."""
    from dotllm_b200.kernels import ops
    x, w = make(1100, 1024, 8192, seed=3)
    whole = ops.linear(x, w)
    for m in (1, 20, 50, 128, 400):
        assert torch.equal(ops.linear(x[:m], w), whole[:m]), m


def test_infinities_nans_and_overflow():
    from dotllm_b200.kernels import library, ops
    for M in (4, 200):
        x, w = make(M, 192, 1024, seed=5)
        x[0, 7], x[1, 900], x[2, 3] = float("inf"), float("nan"), -float("inf")
        x[3, :] = 3.0e38                                   # sums beyond float32: some on the way only, some for good
        w[10, 7] = 0.0                                     # inf * 0
        w[20, :] = 1.0
        y = ops.linear(x, w)
        chain = torch.empty_like(y)                        # what the FFMA kernel says
        library.call("dl_gemm_f32", x.data_ptr(), 1024, w.data_ptr(), chain.data_ptr(), 192, M, 192, 1024, library.current_stream())
        assert bool(torch.isnan(y[0, 10])) and bool(torch.isnan(y[1]).all()) and float(y[3, 20]) == float("inf")
        assert torch.equal(y[:3].nan_to_num(nan=1.25), chain[:3].nan_to_num(nan=1.25))
        # where a sum overflows on the way in one order and not in the other, the finite result is the right one
        fine = torch.isfinite(y[3])
        assert torch.equal(y[3][~fine].nan_to_num(nan=1.25), chain[3][~fine].nan_to_num(nan=1.25))
        want = x[3].double() @ w.double().T
        assert bool(((y[3].double() - want).abs() <= bound(x[3:4], w)[0])[fine].all())


def test_small_and_large_values_keep_their_digits():
    """Pieces far from one: the three pieces of a value cover float32's exponents down to about 1e-33."""
    from dotllm_b200.kernels import ops
    x, w = make(24, 128, 2048, seed=6)
    for sx, sw in ((1e-25, 1e20), (1e18, 1e-12), (1e-12, 1e-15)):
        xs, ws = x * sx, w * sw
        err = (ops.linear(xs, ws).double() - xs.double() @ ws.double().T).abs()
        assert bool((err <= bound(xs, ws)).all())


@pytest.mark.parametrize("M", [1, 24, 50, 200])
@pytest.mark.parametrize("sx,sw", [(1e-36, 1.0), (1.0, 1e-35), (1.0, 2e-37), (1e-18, 1e-17), (1e-34, 1e3), (3e30, 1e-34), (2e-38, 2e4)])
def test_the_smallest_values_keep_their_digits(M, sx, sw):
    """Down to numbers below the normal ones: every bit of a value counts (the result's own rounding may be that of such a number)."""
    from dotllm_b200.kernels import ops
    x, w = make(M, 144, 1024, seed=7)
    xs, ws = x * sx, w * sw
    want = xs.double() @ ws.double().T
    err = (ops.linear(xs, ws).double() - want).abs()
    assert bool((err <= bound(xs, ws) + 2.0 ** -149).all())
    assert float(err.norm() / want.norm()) < 5e-7


@pytest.mark.parametrize("M,N,K", [(700, 2048, 2048), (700, 2500, 516), (300, 1024, 8192), (40, 4096, 2048), (8, 2048, 2048), (1, 2048, 1024)])
def test_results_that_are_not_finite_cost_an_ffma_product(M, N, K):
    """Every output infinite: the bits of the FFMA kernel, and a few of its times on top of this one's (not thousands of loads one after the other)."""
    from dotllm_b200.kernels import library, ops
    x, w = make(M, N, K, seed=9)
    bad = x.clone()
    bad[:, K - 3] = float("inf")
    chain = torch.empty(M, N, device=DEV)

    def ffma(x):
        library.call("dl_gemm_f32", x.data_ptr(), K, w.data_ptr(), chain.data_ptr(), N, M, N, K, library.current_stream())

    def time(f):
        times = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            f()
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[3:])                                  # (the host may be slow, the device is not slow by chance)

    y = ops.linear(bad, w)
    ffma(bad)
    assert torch.equal(y.nan_to_num(nan=1.25), chain.nan_to_num(nan=1.25)) and not bool(torch.isfinite(y).any())
    library.check_status()
    finite, infinite, product = time(lambda: ops.linear(x, w)), time(lambda: ops.linear(bad, w)), time(lambda: ffma(x))
    print(f"observed {M} x {N} x {K}: finite {finite * 1e3:.0f} us, not finite {infinite * 1e3:.0f}, FFMA {product * 1e3:.0f}")
    assert infinite < finite + 10 * product                    # (8 rows: 7.8 times; a cut tile's chains are single lanes' and read rows of W side by side)


@pytest.mark.parametrize("M,N,K", [(4, 300, 256), (9, 256, 2048), (24, 200, 516), (50, 256, 768), (200, 256, 2048), (300, 128, 4096), (20, 144, 14336)])
def test_no_further_off_than_the_ffma_product(M, N, K):
    """Norms: the bound above leaves room for a product without its smallest pieces (4e-6 off), this does not.  Every number of tokens a
    tile may have, whole and cut tiles."""
    from dotllm_b200.kernels import library, ops
    x, w = make(M, N, K, seed=12)
    want = x.double() @ w.double().T
    chain = torch.empty(M, N, device=DEV)
    library.call("dl_gemm_f32", x.data_ptr(), K, w.data_ptr(), chain.data_ptr(), N, M, N, K, library.current_stream())
    far = lambda y: float((y.double() - want).norm() / want.norm())
    assert far(ops.linear(x, w)) < min(5e-7, 1.1 * far(chain) + 2e-8), (far(ops.linear(x, w)), far(chain))


@pytest.mark.parametrize("M", [4, 24, 50, 200])
@pytest.mark.parametrize("K", [512, 8192])
@pytest.mark.parametrize("whose", ["x", "w"])
def test_the_last_eight_bits_alone(M, K, whose):
    """Neighbours in k that cancel but for their last pieces: what is left is 2^-17 of the terms, the sums' own rounding 2^-24 of them."""
    from dotllm_b200.kernels import ops
    a, b = make(M, 144, K, seed=13)
    a, b = (a, b) if whose == "x" else (b, a)

    def last(t):                                               # pairs (v, -(v without its last piece)); the other side's pairs are equal
        v = t[:, ::2].contiguous()
        hi = v.to(torch.bfloat16).float()
        mid = (v - hi).to(torch.bfloat16).float()
        return torch.stack([v, -(hi + mid)], dim=2).reshape(t.shape).contiguous()

    first, second = last(a), b[:, ::2].to(torch.bfloat16).float().repeat_interleave(2, 1).contiguous()
    x, w = (first, second) if whose == "x" else (second, first)
    want = x.double() @ w.double().T
    assert 0 < float(want.norm()) < 1e-4 * float((x.abs().double() @ w.abs().double().T).norm())
    assert float((ops.linear(x, w).double() - want).norm() / want.norm()) < 0.1
