"""Rules by which a launcher chooses among its kernels, asked without a GPU (148 SMs)."""
import time

import pytest

from megalodon_b200.ops._ext import have_ext, require

pytestmark = pytest.mark.skipif(not have_ext(), reason="extension not built")
_BF16, _FP16 = 1, 2


def test_attention_of_one_query_in_one_launch():
    """Where its clusters run at once and fill the SMs (figures beside the rule); fp16 not at all."""
    plan = require().decode_attend_plan
    for heads, want in ((1, 128), (2, 64), (3, 0), (18, 0), (19, 0), (24, 0), (28, 8), (32, 8), (34, 0), (36, 0), (40, 0),
                        (48, 0), (60, 4), (64, 4), (68, 0), (72, 0), (96, 0), (112, 2), (148, 2), (150, 1), (400, 1)):
        ctas = plan(heads, 2048, 256, 2048 if heads < 3 else 1024, _BF16, 148)
        assert ctas == want, (heads, ctas)
        assert plan(heads, 2048, 256, 1024, _FP16, 148) == 0
    for heads, want in ((19, 8), (32, 8), (36, 0), (37, 4), (64, 4), (72, 0), (75, 2)):      # narrow rows
        assert plan(heads, 2048, 64, 256, _BF16, 148) == want, heads
    for heads, want in ((28, 0), (64, 0), (128, 2), (200, 1)):                              # scores from FMAs
        assert plan(heads, 2048, 72, 264, _BF16, 148) == want, heads
    # whatever the heads: never more CTAs in clusters than run at once, never too few for the SMs
    for heads in range(3, 600):
        ctas = plan(heads, 2048, 128, 1024, _BF16, 148)
        if ctas > 1:
            assert 214 <= ctas * heads <= (296 if ctas == 2 else 259), heads


def test_sequences_to_a_cta_of_the_ema():
    """Every number of CTAs is looked at, and nothing else: a batch of 65535 costs a call less than its launches."""
    plan = require().cema_tensor_plan

    def want(B, L, D, sms=148):
        groups, tiles = -(-D // 16), -(-L // 256)
        cost, per = min((-(-groups * -(-B // n) // sms) * (5.0 + 2.85 * tiles * n), n) for n in range(1, B + 1))
        return cost, per
    for B in (*range(1, 70), 100, 777, 1000, 4097):
        for L, D in ((300, 1024), (777, 1024), (2048, 2048), (5003, 512), (600, 64)):
            cost, per = want(B, L, D)
            assert plan(B, L, D, 148) == (0 if cost > 32.0 + 8e-6 * B * L * D else per), (B, L, D)
    # one pass of the scan: few sequences on the tensor cores, many not
    for B, L, D, tensor in ((1, 2, 1024, False), (1, 37, 1024, True), (4, 64, 512, True), (4, 128, 1024, True),
                            (16, 128, 1024, False), (128, 100, 128, False), (8, 40, 1024, False), (4, 100, 4096, False)):
        assert (plan(B, L, D, 148) > 0) == tensor, (B, L, D)
    t0 = time.perf_counter()
    for B in range(65436, 65536):
        plan(B, 2, 16, 148)
    assert time.perf_counter() - t0 < 100 * 50e-6


@pytest.mark.parametrize("M,N,K,tiles", [
    # us measured as 128 x 64, 128 x 128, 128 x 256 and CTA pair (512); what may be chosen is within 4 % of the best
    (130, 4096, 16384, {64}),               # 50.5  61.0 101.2  78.8
    (513, 4096, 16384, {512}),              # 140   111  101    84
    (1000, 512, 20000, {64}),               # 59.6  70.5 110    94
    (1000, 4096, 8192, {512}),              # 95.6  62.7  57.3  50.0
    (600, 4096, 11264, {512}),              # 104   82.2  75.3  64.7
    (2000, 2048, 512, {128, 256}),          # 11.4   8.5   8.5   9.2
    (2000, 1024, 4096, {128}),              # 27.4  16.5  24.1  24.1
    (1000, 512, 4096, {64}),                # 15.1  15.5  23.6  23.8
    (4096, 4096, 4096, {512}),              # 172   109   111    92
    (513, 1024, 16384, {64, 128}),          # 51.2  49.8  77.6  77.8
    (6216, 1024, 2048, {128, 512}),         # 40.3  24.3  26.2  24.7
])
def test_tile_of_a_product(M, N, K, tiles):
    assert require().gemm_tile(M, N, K, 1, 148) in tiles
