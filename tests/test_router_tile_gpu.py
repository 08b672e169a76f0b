"""Router logits beyond 128 tokens (the register-tiled kernel) against the CPU checker, bit for bit: the pinned order of
additions holds for every way the kernel is cut."""
import numpy as np
import pytest

from oracle import oracle
from zerocool_b200 import synth
from zerocool_b200.records import BF16, F32, MoeConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,experts,hidden,act,router_dtype,shared", [
    (129, 512, 2048, BF16, F32, 1),      # partitions over a cluster, one token in the last tile, the gate row on its own
    (256, 512, 4096, BF16, F32, 0),
    (300, 96, 2560, BF16, BF16, 1),      # a row tile of 33 rows (the gate row shares it), partitions of 160
    (191, 32, 128, F32, F32, 1),         # partitions of eight k
    (200, 1024, 640, F32, BF16, 0),
    (1000, 1024, 384, BF16, F32, 1),     # 256 tiles: whole tiles, running totals
    (1930, 1024, 128, BF16, F32, 1),     # 496 tiles: 128-token tiles, ten tokens in the last one
    (2050, 992, 256, F32, F32, 0),
])
def test_router_logits_of_long_batches_are_bit_exact(tokens, experts, hidden, act, router_dtype, shared):
    torch = pytest.importorskip("torch")
    from zerocool_b200.moe import Moe
    cfg = MoeConfig(hidden=hidden, ffn=128, experts=experts, top_k=4, layers=1, max_tokens=tokens, act_dtype=act, router_dtype=router_dtype, has_shared=shared)
    m = Moe(cfg, 0)
    w = synth.router(cfg, 7, 0)
    m.load_layer(0, router_w=w, shared_gate_w=synth.shared_gate(cfg, 7, 0) if shared else None)
    x = synth.activations(cfg, 7, 0, tokens)
    dev = torch.from_numpy(x).to(device="cuda", dtype=torch.bfloat16 if act == BF16 else torch.float32)
    got = m.router(0, dev).cpu().numpy()
    want = oracle.router_logits(x, w, router_dtype)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert np.array_equal(m.router(0, dev).cpu().numpy().view(np.uint32), got.view(np.uint32))
