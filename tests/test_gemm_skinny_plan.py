"""Which weight-streaming products go by rows and which by shares, and how the shares are cut (no GPU is needed: the plan is the library's)."""
import pytest

from dotllm_b200.kernels import gemm_skinny


@pytest.mark.parametrize("N,K,gated,form", [
    (2048, 2048, False, "rows"), (16, 4096, False, "rows"), (16, 4104, False, "shares"), (512, 8192, False, "shares"), (1024, 12288, False, "shares"),
    (512, 14336, False, "shares"), (64, 16384, False, "shares"), (1536, 16384, False, "shares"), (13 * 148, 12288, False, "shares"),
    (13 * 148 + 1, 12288, False, "rows"), (2048, 5120, False, "rows"), (2048, 5128, False, "shares"), (2048, 8192, False, "shares"),
    (2048, 12280, False, "shares"), (2368, 14336, False, "rows"), (2369, 14336, False, "shares"), (2400, 4096, False, "rows"), (20 * 148, 8192, False, "shares"),
    (20 * 148 + 1, 8192, False, "rows"), (4096, 14336, False, "rows"), (128256, 2048, False, "rows"),
    (8192, 2048, True, "rows"), (512, 4096, True, "rows"), (6 * 148, 8192, True, "shares"), (6 * 148 + 1, 8192, True, "rows"), (64, 14336, True, "shares"),
    (1024, 14336, True, "rows")])
def test_the_form_follows_the_measured_sizes(N, K, gated, form):
    """Few rows of long k are read by shares: by rows every block reads all of x (512 x 14,336 of eight rows took 10.7 us where shares take 8)."""
    assert gemm_skinny.plan(N, K, gated)[0] == form


@pytest.mark.parametrize("sms", [148, 132, 8, 1])
def test_shares_cover_the_product_and_hand_over_few_parts(sms):
    """Every chunk has a warp, no more blocks than multiprocessors, and a tile of long k is not cut into single chunks, whose sums one warp would add."""
    for N in (1, 16, 17, 256, 512, 1024, 1536, 2000, 2400, 2960):
        for K in (4104, 5120, 6144, 8192, 10240, 12280, 14336, 24576):
            for gated in (False, True):
                form, warps, share, blocks = gemm_skinny.plan(N, K, gated, sms)
                if form != "shares":
                    continue
                tiles, chunks = (N + (7 if gated else 15)) // (8 if gated else 16), -(-K // 256)
                assert 4 <= warps <= gemm_skinny.CONSUMER_WARPS and 1 <= blocks <= sms
                assert (blocks - 1) * warps * share < tiles * chunks <= blocks * warps * share
                assert share >= (4 if chunks >= 48 else 2 if chunks >= 32 else 1)
                floats, counters = gemm_skinny.scratch_need(16, N, K, gated, sms)
                assert floats >= blocks * warps * 2 * 2 * 128 and counters == tiles
