"""Performance cases of the MoE layer: the calls an inference engine makes, over the range of its batches.

A case is one engine step's calls to the layer: `layers` layers, each with an input of its own (in a model the other
sub-blocks of a layer stand between two MoE calls, so their inputs are independent here), through the public entry points
of `zerocool_b200.moe.Moe`. `form` says how the program issues them:
  "eager"  Moe.moe layer by layer on the current stream
  "graph"  the same calls captured once into a CUDA graph and replayed, as a serving loop does for short batches
  "hc"     Moe.moe_hc: the layer with the hyper-connection update of the residual streams as its epilogue
Weights, router and activations are seeded, with the distributions of the benchmark: uniform codes, scales U(0.004, 0.02),
bias = -8 scale (8-bit: 0-centred codes and bias = -8 scale as well), router ~N(0, 0.02), activations ~N(0, 1).
"""
import math

import numpy as np
import torch

from zerocool_b200.moe import Moe
from zerocool_b200.records import ARITH_FP32, ARITH_REFERENCE, BF16, F16, F32, MoeConfig

# The benchmark's layer: hidden 2048, 512 routed experts top-10 and a shared one, ffn 512, 4-bit groups of 64.
BASE = dict(form="graph", hidden=2048, ffn=512, experts=512, top_k=10, shared=True, down_bits=4, bf16_meta=False, bf16_router=False,
            f32_act=False, f32_out=False, reference=False, zipf=False, layers=1, tokens=1)


def case(name, **kw):
    return dict(BASE, name=name, **kw)


def listed():
    return [
        # one user generating: a token per step, everything is latency; replayed from a graph
        case("decode_1", tokens=1, layers=8),
        # a handful of users, the layer called one by one by an engine that does not capture
        case("decode_5_eager", tokens=5, layers=8, form="eager"),
        # small and full serving batches of generated tokens; 64 is the benchmark's headline batch
        case("decode_16", tokens=16, layers=4),
        case("decode_64", tokens=64, layers=4),
        # the smallest model: 64 experts, no shared expert, FP32 activations and results, one token
        case("small_model_1", tokens=1, layers=16, experts=64, top_k=8, shared=False, f32_act=True, f32_out=True),
        # the reference engine's own shape and arithmetic, with the residual-stream update it does around the layer
        case("native_hc_9", tokens=9, layers=4, form="hc", hidden=2560, ffn=640, bf16_meta=True, bf16_router=True, f32_act=True, f32_out=True, reference=True),
        # mixed artifact (8-bit down projection), generated tokens of a middling batch
        case("mixed_37", tokens=37, layers=2, down_bits=8),
        # hidden 4096: the large model of the expert-parallel configuration on one GPU, 256 tokens in flight
        case("wide_256", tokens=256, hidden=4096, form="eager"),
        # a chunk of a prompt riding with generated tokens: about ten rows per expert
        case("chunk_513", tokens=513, form="eager"),
        # prompts: 2048 and 8192 tokens with skewed expert loads
        case("prefill_2048", tokens=2048, form="eager", zipf=True),
        case("prefill_8192", tokens=8192, form="eager", zipf=True),
        # 32 requests of ragged lengths flattened into one batch, mixed artifact
        case("mixed_6430", tokens=6430, form="eager", down_bits=8),
    ]


def draw(rng):
    """One more case: a geometry, a batch size spread over its logarithm, and the options that go with both."""
    c = dict(BASE)
    c.update(rng.choice([dict(), dict(), dict(down_bits=8), dict(hidden=4096), dict(hidden=2560, ffn=640, bf16_meta=True, bf16_router=True),
                         dict(experts=64, top_k=8, shared=False), dict(experts=128, top_k=8)]))
    most = 2048 if c["hidden"] == 4096 else 4096
    c["tokens"] = int(round(math.exp(rng.uniform(0, math.log(most)))))
    if c["tokens"] <= 64:
        c["layers"] = rng.randint(2, 4)
        c["form"] = rng.choice(["graph", "eager", "hc"])
        c["f32_act"] = c["f32_out"] = rng.random() < 0.25
        c["reference"] = c["bf16_meta"] and c["f32_act"]
    else:
        c["form"] = rng.choice(["eager", "graph"])
        c["f32_out"] = rng.random() < 0.25
        c["zipf"] = rng.random() < 0.4
    return c


def config(c):
    return MoeConfig(hidden=c["hidden"], ffn=c["ffn"], experts=c["experts"], top_k=c["top_k"], layers=c["layers"], max_tokens=max(64, c["tokens"]),
                     down_bits=c["down_bits"], q8_signed=1, meta_dtype=BF16 if c["bf16_meta"] else F16, act_dtype=F32 if c["f32_act"] else BF16,
                     out_dtype=F32 if c["f32_out"] else BF16, router_dtype=BF16 if c["bf16_router"] else F32, has_shared=int(c["shared"]),
                     arith=ARITH_REFERENCE if c["reference"] else ARITH_FP32)


def generator(seed, *what):
    g = torch.Generator(device="cuda")
    g.manual_seed((seed * 1000003 + sum((v + 1) * 7919 ** (i + 1) for i, v in enumerate(what))) % (1 << 62))
    return g


def projections(c):
    """(rows, columns, bits, byte offset) of gate, up and down inside a record, and the record's length."""
    out, at = [], 0
    for n, k, bits in ((c["ffn"], c["hidden"], 4), (c["ffn"], c["hidden"], 4), (c["hidden"], c["ffn"], c["down_bits"])):
        out.append((n, k, bits, at))
        at += n * k * bits // 8 + 2 * n * (k // 64) * 2
    return out, at


def records(c, seed, layer, count, which):
    """uint8 [count, stride]: expert records with uniform codes; `which` keeps routed and shared experts apart."""
    parts, size = projections(c)
    stride = (size + 16383) // 16384 * 16384
    g = generator(seed, layer, which)
    r = torch.randint(0, 256, (count, stride), dtype=torch.uint8, device="cuda", generator=g)
    meta = torch.bfloat16 if c["bf16_meta"] else torch.float16
    for n, k, bits, at in parts:
        codes, half = n * k * bits // 8, n * (k // 64) * 2
        if bits == 8:
            r[:, at:at + codes] = torch.randint(-127, 128, (count, codes), dtype=torch.int8, device="cuda", generator=g).view(torch.uint8)
        scale = (torch.rand(count, half // 2, device="cuda", generator=g) * 0.016 + 0.004).to(meta)
        bias = (scale.float() * -8.0).to(meta)
        r[:, at + codes:at + codes + half] = scale.view(torch.uint8)
        r[:, at + codes + half:at + codes + 2 * half] = bias.view(torch.uint8)
    return r


def router_of(c, seed, layer):
    g = generator(seed, layer, 2)
    w = torch.randn(c["experts"], c["hidden"], device="cuda", generator=g) * 0.02
    gate = torch.randn(1, c["hidden"], device="cuda", generator=g) * 0.02
    t = torch.bfloat16 if c["bf16_router"] else torch.float32
    return w.to(t), gate.to(t)


def router_bias(c, seed, layer):
    """Skewed loads: -1.1 ln(rank) on the logits, ranks in a seeded order."""
    order = np.random.RandomState((seed * 31 + layer) % (1 << 31)).permutation(c["experts"])
    b = np.empty(c["experts"], np.float32)
    b[order] = -1.1 * np.log(np.arange(1, c["experts"] + 1))
    return b


def inputs(c, seed, layer):
    g = generator(seed, layer, 3)
    x = torch.randn(c["tokens"], c["hidden"], device="cuda", generator=g).to(torch.bfloat16)
    x = x.float() if c["f32_act"] and c["reference"] else torch.randn(c["tokens"], c["hidden"], device="cuda", generator=g) if c["f32_act"] else x
    hyper = inject = None
    if c["form"] == "hc":
        hyper = torch.randn(c["tokens"], 4, c["hidden"], device="cuda", generator=g).to(torch.bfloat16).float()
        inject = torch.rand(c["tokens"], 4, device="cuda", generator=g).to(torch.bfloat16).float()
    return x, hyper, inject


def calls(state):
    m, outs = state["moe"], []
    for layer, (x, hyper, inject) in enumerate(state["inputs"]):
        outs.append(m.moe_hc(layer, x, hyper, inject) if hyper is not None else m.moe(layer, x))
    return outs


def prepare(case, seed):
    m = Moe(config(case), torch.cuda.current_device())
    for layer in range(case["layers"]):
        w, gate = router_of(case, seed, layer)
        shared = records(case, seed, layer, 1, 1)[0] if case["shared"] else None
        m.load_layer(layer, records(case, seed, layer, case["experts"], 0), router_w=w, shared_record=shared, shared_gate_w=gate if case["shared"] else None)
        if case["zipf"]:
            m.set_router_bias(layer, router_bias(case, seed, layer))
    state = {"moe": m, "inputs": [inputs(case, seed, layer) for layer in range(case["layers"])]}
    if case["form"] == "graph":
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            calls(state)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            state["outs"] = calls(state)
        state["graph"] = graph
    return state


def run(state):
    if "graph" in state:
        state["graph"].replay()
        return state["outs"]
    return calls(state)


def active(c):
    """Expected number of routed experts that a batch selects."""
    if not c["zipf"]:
        return c["experts"] * (1 - (1 - c["top_k"] / c["experts"]) ** c["tokens"])
    r = np.random.RandomState(0)
    z = r.randn(min(c["tokens"], 4096), c["experts"]).astype(np.float32) * (0.02 * math.sqrt(c["hidden"])) + router_bias(c, 0, 0)
    return len(np.unique(np.argpartition(-z, c["top_k"] - 1, axis=1)[:, :c["top_k"]]))


def work(case):
    c = case
    T, H, F, E, K, S = c["tokens"], c["hidden"], c["ffn"], c["experts"], c["top_k"], int(c["shared"])
    record = projections(c)[1]
    ab, ob, rb = 4 if c["f32_act"] else 2, 4 if c["f32_out"] else 2, 2 if c["bf16_router"] else 4
    rows = T * H * (ab + (2 * 4 * 4 if c["form"] == "hc" else ob))
    return {"bytes": c["layers"] * ((active(c) + S) * record + (E + S) * H * rb + rows),
            "flops": c["layers"] * (T * (K + S) * 6.0 * H * F + 2.0 * T * (E + S) * H)}


def tolerance(case):
    # The reference arithmetic rounds to BF16 at every boundary, a BF16 result once: another order of the FP32 sums moves some
    # values to the neighbouring BF16 value (2^-8 of a value at most). FP32 results differ by the FP16 rounding of the SwiGLU rows.
    if case["reference"]:
        return {"rel": 1e-2, "max": 0.1}
    return {"rel": 2e-3, "max": 0.02} if case["f32_out"] else {"rel": 5e-3, "max": 0.04}


def dense(c, record, part):
    """One projection of a record as FP64 [rows, columns]."""
    n, k, bits, at = projections(c)[0][part]
    codes, half = n * k * bits // 8, n * (k // 64) * 2
    raw = record[at:at + codes].view(n, -1)
    q = torch.stack((raw & 15, raw >> 4), -1).view(n, k) if bits == 4 else raw.view(torch.int8)
    meta = torch.bfloat16 if c["bf16_meta"] else torch.float16
    s, b = (record[at + codes + i * half:at + codes + (i + 1) * half].clone().view(meta).view(n, k // 64, 1).double() for i in (0, 1))
    return (q.double().view(n, k // 64, 64) * s + b).view(n, k)


def expert64(c, record, x):
    gate, up = x @ dense(c, record, 0).T, x @ dense(c, record, 1).T
    return (gate * torch.sigmoid(gate) * up) @ dense(c, record, 2).T


def exact(case, seed):
    c, outs = case, []
    for layer in range(c["layers"]):
        x32, hyper, inject = inputs(c, seed, layer)
        w, gate_w = router_of(c, seed, layer)
        x = x32.double()
        logits = x @ w.double().T
        if c["zipf"]:
            logits += torch.from_numpy(router_bias(c, seed, layer)).cuda().double()
        top, ids = logits.topk(c["top_k"], dim=1)
        weights = torch.softmax(top, dim=1)
        rec = records(c, seed, layer, c["experts"], 0)
        y = torch.zeros_like(x)
        for e in torch.unique(ids).tolist():
            t, j = (ids == e).nonzero(as_tuple=True)
            y.index_add_(0, t, expert64(c, rec[e], x[t]) * weights[t, j][:, None])
        if c["shared"]:
            y += torch.sigmoid(x @ gate_w.double().T) * expert64(c, records(c, seed, layer, 1, 1)[0], x)
        outs.append(y if hyper is None else hyper.double() + y[:, None, :] * inject.double()[:, :, None])
        del rec
    return outs
