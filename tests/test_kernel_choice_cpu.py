"""The rules that choose a call's kernels, on the CPU: what they count, and where they change over."""
import math

import pytest

from zerocool_b200.moe import kernel_choice
from zerocool_b200.records import MoeConfig

SMS = 148


def router_cut(tokens, experts, shared, sms=SMS):
    c = kernel_choice(MoeConfig(hidden=128, ffn=128, experts=experts, top_k=4, has_shared=shared, max_tokens=max(tokens, 1)), tokens, sms)
    return c["router_ranks"], c["router_tokens"]


@pytest.mark.parametrize("experts,shared", [(512, 1), (512, 0), (128, 1), (96, 1), (1024, 1)])
def test_whole_router_tiles_are_at_most_two_per_sm(experts, shared):
    """Whole-K tiles of 64 tokens live as long as the kernel: a third one on some SM makes the launch half as long again."""
    whole = 0
    for tokens in range(129, 9000, 7):
        ranks, rows = router_cut(tokens, experts, shared)
        if rows == 64 and ranks == 1:
            whole += 1
            assert math.ceil(tokens / 64) * math.ceil((experts + shared) / 64) <= 2 * SMS, tokens
    assert whole or experts in (96, 128)          # with few experts the gate's row tile is a third of the tiles or more


def test_router_cut_at_its_edges():
    assert [router_cut(t, 512, 1) for t in (1, 8, 9, 128, 129)] == [(8, 8), (8, 8), (8, 16), (8, 16), (8, 64)]
    assert router_cut(1856, 512, 1) == (8, 64) and router_cut(1920, 512, 1) == (1, 64)
    assert router_cut(2048, 512, 1) == (1, 64) and router_cut(2049, 512, 1) == (8, 64)         # 288 and 297 tiles
    assert router_cut(2368, 512, 0) == (1, 64) and router_cut(2369, 512, 0) == (8, 64)         # 296 and 304
    assert router_cut(8192, 128, 1) == (8, 64)                                                 # 384
    assert router_cut(3776, 512, 1) == (8, 64) and router_cut(3777, 512, 1) == (1, 128)
    assert router_cut(2048, 512, 1, sms=132) == (8, 64)                                        # 288 tiles on fewer SMs
