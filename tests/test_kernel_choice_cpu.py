"""The rules that choose a call's kernels, on the CPU: what they count, and where they change over."""
import math

import pytest

from zerocool_b200.moe import kernel_choice
from zerocool_b200.records import ARITH_REFERENCE, BF16, F32, MoeConfig

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


ITEM, STREAMING = 1, 2


def expert_kernels(tokens, sms=SMS, **kw):
    base = dict(hidden=2048, ffn=512, experts=512, top_k=10, has_shared=1, max_tokens=max(tokens, 1))
    base.update(kw)
    return kernel_choice(MoeConfig(**base), tokens, sms)["expert_kernels"]


@pytest.mark.parametrize("kw", [dict(experts=128, top_k=8), dict(experts=128, top_k=8, has_shared=0), dict(experts=64, top_k=10), dict(experts=64, top_k=8, has_shared=0),
                                dict(experts=512, first_expert=128, local_experts=128)])
def test_experts_with_several_passes_stream(kw):
    """The rule counts eight-row passes, not experts: 64 to 128 experts at 64 tokens and more are many passes, however few experts."""
    for tokens in range(64, 400, 3):
        assert expert_kernels(tokens, **kw) == STREAMING, tokens


NATIVE = dict(hidden=2560, ffn=640, meta_dtype=BF16)


@pytest.mark.parametrize("tokens,kw,kernels", [
    (1, {}, ITEM), (2, {}, ITEM), (3, {}, STREAMING), (5, {}, STREAMING), (14, {}, STREAMING), (15, {}, ITEM), (16, {}, ITEM), (17, {}, STREAMING), (64, {}, STREAMING),
    (24, dict(experts=256, top_k=8), ITEM), (28, dict(experts=256, top_k=8), STREAMING), (14, dict(experts=256, top_k=8, ffn=768), ITEM),
    (1, dict(act_dtype=F32), ITEM), (2, dict(act_dtype=F32), STREAMING), (2, dict(act_dtype=F32, arith=ARITH_REFERENCE), ITEM),
    (2, NATIVE, ITEM), (5, NATIVE, STREAMING), (8, NATIVE, ITEM), (9, NATIVE, ITEM), (13, NATIVE, ITEM), (14, NATIVE, ITEM), (15, NATIVE, ITEM), (18, NATIVE, STREAMING), (22, NATIVE, STREAMING),
    (40, NATIVE, STREAMING), (24, dict(NATIVE, experts=64, top_k=8, has_shared=0), ITEM), (48, dict(NATIVE, experts=64, top_k=8, has_shared=0), STREAMING),
    (16, dict(NATIVE, down_bits=8), STREAMING),                # ten 8-bit groups are whole stages
    (1, dict(hidden=3072), ITEM), (2, dict(hidden=3072), STREAMING), (1, dict(hidden=4096), ITEM), (2, dict(hidden=4096), STREAMING), (16, dict(hidden=4096), STREAMING),
    (3, dict(hidden=1024, experts=128, top_k=8), ITEM), (4, dict(hidden=1024, experts=128, top_k=8), STREAMING),
])
def test_expert_kernels_at_the_measured_edges(tokens, kw, kernels):
    assert expert_kernels(tokens, **kw) == kernels
