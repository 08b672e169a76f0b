"""The persistent streaming expert kernels against the CPU checker, at the sizes where their cut can go wrong: K that is not
whole stages or pairs of stages, one staged row block, warps sharing a tile, more passes per CTA than its table holds, long
items, more list entries than threads, FP32 activations, 8-bit codes, and biases that do not follow the scales (the bias product
on its own). The option expert_kernels names them, so that no case runs on the item kernels unnoticed."""
import numpy as np
import pytest

from oracle import oracle
from tests import util
from zerocool_b200 import synth
from zerocool_b200.records import ARITH_REFERENCE, BF16, F16, F32, MoeConfig

pytestmark = pytest.mark.gpu
SEED = 11
TOL = 2e-3          # max-abs error over the output's RMS, the specification's bound for FP32 accumulation and FP16 SwiGLU rows


@pytest.mark.parametrize("tokens,kw", [
    (5, dict(experts=512)),                                              # four warps per gate/up tile
    (40, dict(hidden=4096, experts=128)),                                # one row block, four warps per tile
    (40, dict(hidden=3072, experts=64)),
    (33, dict(hidden=384, ffn=128, experts=32)),                         # six groups; a row of 64 code bytes
    (70, dict(hidden=2560, ffn=640, experts=64, meta_dtype=BF16)),       # ten groups: an odd number of stages, half of the last one
    (70, dict(hidden=1280, ffn=384, experts=64, act_dtype=F32)),         # two FP16 terms per activation, three pairs of which the last has one stage
    (130, dict(hidden=512, ffn=256, experts=32)),                        # items of about forty rows
    (5000, dict(hidden=128, ffn=128, experts=32, top_k=8, act_dtype=F32)),   # 5,600 passes: more than a table of 32 per CTA
    (45, dict(hidden=2048, experts=64, down_bits=8, q8_signed=1)),
    (45, dict(hidden=640, ffn=128, experts=32, gate_bits=8, up_bits=8, down_bits=8)),
    (30, dict(hidden=2048, experts=64, gate_bits=8, up_bits=8, down_bits=4)),
    (200, dict(hidden=256, ffn=128, experts=1024, top_k=8)),             # two list entries per thread
    (40, dict(hidden=4096, experts=32, act_dtype=F32)),                  # one row block of two terms, eight warps of their own tiles
    (64, dict(hidden=2560, ffn=640, experts=64, meta_dtype=BF16, act_dtype=F32, router_dtype=BF16, arith=ARITH_REFERENCE)),
])
def test_streamed_experts_against_the_checker(tokens, kw):
    torch = pytest.importorskip("torch")
    from zerocool_b200.moe import Moe
    base = dict(hidden=2048, ffn=512, experts=64, top_k=10, layers=1, meta_dtype=F16, act_dtype=BF16, out_dtype=F32, router_dtype=F32, has_shared=1, max_tokens=tokens)
    base.update(kw)
    cfg = MoeConfig(**base)
    rng = np.random.default_rng(tokens)
    records = [util.asymmetric_record(cfg, SEED, 0, e, rng) for e in range(cfg.experts)]
    shared = util.asymmetric_record(cfg, SEED, 0, synth.SHARED_EXPERT, rng)
    m = Moe(cfg, 0)
    w, gate = synth.router(cfg, SEED, 0), synth.shared_gate(cfg, SEED, 0)
    m.load_layer(0, np.stack(records), router_w=w, shared_record=shared, shared_gate_w=gate)
    m.set_option("expert_kernels", 2)
    x = synth.activations(cfg, SEED, 0, tokens)
    if cfg.gate_bits > cfg.down_bits:
        # 8-bit gate and up weights reach 2.5: activations of 1/16 keep the SwiGLU rows inside the 4-bit down projection's range
        x = x / 16
        assert max(np.abs(oracle.expert(cfg.as_dict(), r, x)[0]).max() for r in records + [shared]) < 4094
    dev = torch.from_numpy(x).to(device="cuda", dtype=m.act_torch)
    got = m.decode(0, dev)
    assert m.status() == 0
    ids = m.last_routing(tokens)["ids"]
    want = oracle.moe_layer(cfg.as_dict(), records, w, x, shared_record=shared, shared_gate_w=gate)
    assert np.array_equal(ids, want["ids"])
    err = util.rel_max_error(got.cpu().numpy(), want["out"])
    # The reference arithmetic rounds to BF16 at every boundary: one step (2^-8 of a value of a few RMS) where a sum lies on one.
    assert err <= (0.05 if cfg.arith == ARITH_REFERENCE else TOL), err
    assert torch.equal(m.decode(0, dev), got)


@pytest.mark.parametrize("kernels", [1, 2])
def test_a_token_does_not_depend_on_its_place_in_the_batch(kernels):
    torch = pytest.importorskip("torch")
    from zerocool_b200.moe import Moe
    cfg = util.cfg2(experts=64, max_tokens=200)
    m = Moe(cfg, 0)
    m.synth_fill_layer(0, SEED)
    m.set_option("expert_kernels", kernels)
    x = torch.from_numpy(synth.activations(cfg, SEED, 0, 200)).to(device="cuda", dtype=torch.bfloat16)
    order = torch.from_numpy(np.random.default_rng(3).permutation(200)).cuda()
    assert torch.equal(m.decode(0, x)[order], m.decode(0, x[order].contiguous()))


def expert_rows_against_64_bits(kw, kernels, fold=1, bias_only=False, rows=1024):
    """(relative 2-norm error of the expert products of 32 experts with two-term SwiGLU rows, the handle's status)."""
    import torch
    from zerocool_b200.moe import Moe
    from zerocool_b200.records import build_record, dequantise, float_to_meta, meta_to_float
    base = dict(hidden=2048, ffn=512, experts=64, top_k=8, layers=1, local_experts=32, meta_dtype=F16, act_dtype=BF16, out_dtype=F32, max_tokens=64, q8_signed=1)
    base.update(kw)
    cfg = MoeConfig(**base)
    rng = np.random.default_rng(5)
    records = []
    for e in range(32):
        parts = []
        for p in range(3):
            codes, scales, _ = synth.projection_parts(cfg, SEED, 0, e, p)
            s = meta_to_float(scales, cfg.meta_dtype)
            if bias_only:
                s, b = np.zeros_like(s), rng.uniform(0.01, 0.03, size=s.shape)
            else:
                b = (-8.0 if cfg.bits(p) == 4 else 0.0) * s + rng.uniform(-0.03, 0.03, size=s.shape)
            parts.append((codes, float_to_meta(s.astype(np.float32), cfg.meta_dtype).reshape(scales.shape), float_to_meta(b.astype(np.float32), cfg.meta_dtype).reshape(scales.shape)))
        records.append(build_record(cfg, parts))
    m = Moe(cfg, 0)
    m.load_layer(0, np.stack(records))
    m.set_option("exact_h", 1)
    m.set_option("fold_q4", fold)
    m.set_option("expert_kernels", kernels)
    x = torch.from_numpy(rng.standard_normal((rows, cfg.hidden)).astype(np.float32)).cuda()
    x = (x.abs() * 0.05 if bias_only else x).to(m.act_torch)
    ids = torch.arange(rows, device="cuda", dtype=torch.int32) % 32
    y = m.ep_experts(0, x, ids).double()
    error = norm = 0.0
    for e in range(32):
        w = [torch.from_numpy(dequantise(cfg, records[e], p)).cuda() for p in range(3)]
        mine = x[ids == e].double()
        gate = mine @ w[0].T
        want = (gate * torch.sigmoid(gate) * (mine @ w[1].T)) @ w[2].T
        error += float(((y[ids == e] - want) ** 2).sum())
        norm += float((want ** 2).sum())
    return (error / norm) ** 0.5, m.status()


@pytest.mark.parametrize("kw", [dict(), dict(act_dtype=F32), dict(gate_bits=8, up_bits=8, down_bits=8)])
def test_bias_terms_keep_the_group_sums_24_bits(kw):
    """Scales of zero leave the sums of bias x group sum, here all of one sign, so that every rounding shows. Each of the three
    products may lose one step of 2^-23 of a partial sum over eight groups (the tensor core's adder) and half of one in each FP32
    addition: on average below 2^-23 together. Group sums cut to 22 bits and added in the tensor core lose two to four times that."""
    pytest.importorskip("torch")
    error, status = expert_rows_against_64_bits(kw, 2, bias_only=True)
    assert status == 0
    assert error <= 3 * 2.0 ** -23, error


@pytest.mark.parametrize("kw,fold", [(dict(act_dtype=F32), 1), (dict(), 0), (dict(act_dtype=F32), 0), (dict(hidden=2560, ffn=640, meta_dtype=BF16), 0),
                                     (dict(gate_bits=8, up_bits=8, down_bits=8), 0)])
def test_streaming_kernels_are_as_close_to_64_bits_as_the_item_kernels(kw, fold):
    """Both accumulate the same products. The error is that of a few thousand group sums (1,024 rows x 8 groups of down, with
    heavy-tailed rows): 8 % covers its scatter."""
    pytest.importorskip("torch")
    stream, status = expert_rows_against_64_bits(kw, 2, fold)
    item, item_status = expert_rows_against_64_bits(kw, 1, fold)
    assert status == 0 and item_status == 0
    assert stream <= 1.08 * item, (stream, item)


@pytest.mark.parametrize("tokens,kernels", [(4, 1), (8, 2), (40, 2)])
def test_the_shared_expert_alone_counts_no_routed_rows(tokens, kernels):
    """A launch with an empty item list has the shared expert's passes only: a few tokens of it run on the item kernels, whatever
    the layer's routed rows would be. The two kernels add in different orders, so equal bits tell which one ran."""
    torch = pytest.importorskip("torch")
    from zerocool_b200.moe import Moe
    m = Moe(util.cfg2(experts=64, top_k=8, local_experts=32, max_tokens=64), 0)
    m.synth_fill_layer(0, SEED)
    x = torch.from_numpy(synth.activations(m.cfg, SEED, 0, tokens)).to(device="cuda", dtype=torch.bfloat16)
    m.ep_dispatch(0, x)
    y = torch.zeros(tokens * 8, m.cfg.hidden, device="cuda")
    outs = []
    for choice in (0, 1, 2):
        m.set_option("expert_kernels", choice)
        outs.append(m.ep_combine(0, x, y).clone())
    assert m.status() == 0
    assert not torch.equal(outs[1], outs[2])
    assert torch.equal(outs[0], outs[kernels])


def test_received_rows_are_counted_by_tokens_and_not_by_capacity():
    """The owner step of expert parallelism: 128 local experts of a handle with room for 4 x 640 rows, one rank of 64 tokens
    (640 rows expected: streaming) - and the same bits as the streaming kernels when they are named."""
    torch = pytest.importorskip("torch")
    from zerocool_b200.ep import attach_local, emulate_peer
    from zerocool_b200.moe import Moe
    parts = []
    for r in range(4):
        m = Moe(util.cfg2(first_expert=r * 128, local_experts=128, max_tokens=64), 0)
        m.synth_fill_layer(0, SEED)
        parts.append(m)
    attach_local(parts)
    xs = [torch.from_numpy(synth.activations(parts[0].cfg, SEED + r, 0, 64)).to(device="cuda", dtype=torch.bfloat16) for r in range(4)]
    outs = {}
    for choice in (0, 1, 2):
        for m in parts:
            m.set_option("expert_kernels", choice)
        outs[choice] = [o.clone() for o in emulate_peer(parts, 0, xs)]
    assert all(m.status() == 0 for m in parts)
    assert any(not torch.equal(a, b) for a, b in zip(outs[1], outs[2]))
    assert all(torch.equal(a, b) for a, b in zip(outs[0], outs[2]))


@pytest.mark.parametrize("tokens", [5, 40, 1200])
def test_item_kernels_take_what_the_streaming_kernels_take(tokens):
    """A handle whose records have no TMA view runs everything on the item kernels, the few-row experts of a long batch too."""
    torch = pytest.importorskip("torch")
    from zerocool_b200.moe import Moe
    cfg = util.cfg2(experts=128, max_tokens=1280)
    m = Moe(cfg, 0)
    m.synth_fill_layer(0, SEED)
    m.set_router_bias(0, synth.zipf_router_bias(cfg, SEED, 0))
    x = torch.from_numpy(synth.activations(cfg, SEED, 0, tokens)).to(device="cuda", dtype=torch.bfloat16)
    outs = []
    for kernels in (2, 1):
        m.set_option("expert_kernels", kernels)
        outs.append(m.moe(0, x).clone())
    counts = np.diff(m.last_routing(tokens)["offsets"])
    assert tokens < 64 or (((counts > 0) & (counts <= 16)).any() and (counts > 64).any())      # both sides of a long batch
    assert m.status() == 0
    assert util.rel_max_error(outs[1].cpu().numpy(), outs[0].cpu().numpy()) <= TOL
