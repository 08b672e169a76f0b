"""Router logits beyond 128 tokens (the register-tiled kernel) against the CPU checker, bit for bit: the pinned order of
additions holds for every way the kernel is cut."""
import numpy as np
import pytest

from oracle import oracle
from zerocool_b200 import synth
from zerocool_b200.moe import kernel_choice
from zerocool_b200.records import BF16, F16, F32, MoeConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,experts,hidden,act,router_dtype,shared", [
    (129, 512, 2048, BF16, F32, 1),      # partitions over a cluster, one token in the last tile, the gate row in a tile of its own
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


def test_router_bias_is_added_to_the_finished_sum():
    torch = pytest.importorskip("torch")
    from zerocool_b200.moe import Moe
    cfg = MoeConfig(hidden=256, ffn=128, experts=96, top_k=4, max_tokens=300, act_dtype=BF16, router_dtype=F32)
    m = Moe(cfg, 0)
    w, bias = synth.router(cfg, 7, 0), np.random.default_rng(1).standard_normal(96).astype(np.float32)
    m.load_layer(0, router_w=w)
    m.set_router_bias(0, bias)
    x = synth.activations(cfg, 7, 0, 300)
    got = m.router(0, torch.from_numpy(x).to(device="cuda", dtype=torch.bfloat16)).cpu().numpy()
    want = oracle.router_logits(x, w, F32) + bias
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("tokens,experts,cut", [(100, 512, (8, 16)), (129, 512, (8, 64)), (300, 96, (8, 64)), (2048, 512, (1, 64)), (3900, 512, (1, 128)), (3000, 1024, (1, 128))])
def test_shared_gate_value_is_bit_exact(tokens, experts, cut):
    """The gate value of the shared expert, which a layer call does not hand out. Experts of zeros leave out = sigmoid(gate) x shared row;
    a layer whose gate row makes the sigmoid 1 gives the shared rows, and combining those with the checker's gate values must
    give the first layer's result, bit for bit."""
    torch = pytest.importorskip("torch")
    from zerocool_b200.moe import Moe
    cfg = MoeConfig(hidden=128, ffn=128, experts=experts, top_k=4, layers=2, max_tokens=tokens, meta_dtype=F16, act_dtype=BF16, out_dtype=F32, router_dtype=F32, has_shared=1)
    choice = kernel_choice(cfg, tokens)
    assert (choice["router_ranks"], choice["router_tokens"]) == cut
    rng = np.random.default_rng(tokens)
    gate = (rng.standard_normal((1, 128)) * 0.2).astype(np.float32)
    one = np.zeros((1, 128), np.float32)
    one[0, 0] = 200.0
    w = synth.router(cfg, 7, 0)
    shared = synth.record(cfg, 7, 0, synth.SHARED_EXPERT)
    m = Moe(cfg, 0)
    for layer, row in enumerate((gate, one)):
        m.load_layer(layer, np.zeros((experts, cfg.record_stride), np.uint8), router_w=w, shared_record=shared, shared_gate_w=row)
    x = synth.activations(cfg, 7, 0, tokens)
    x[:, 0] = 1.0
    dev = torch.from_numpy(x).to(device="cuda", dtype=torch.bfloat16)
    got, rows = m.decode(0, dev).clone(), m.decode(1, dev).clone()
    routing = m.last_routing(tokens)
    values = oracle.router_logits(x, gate, F32)[:, 0]
    zeros = torch.zeros(tokens * 4, 128, device="cuda")
    again = m.combine(zeros, torch.from_numpy(routing["weights"]).cuda(), torch.from_numpy(routing["ids"]).cuda(), rows, torch.from_numpy(values.copy()).cuda())
    assert m.status() == 0 and rows.abs().max() > 0
    assert torch.equal(again, got)
