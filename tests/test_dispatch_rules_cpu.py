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
