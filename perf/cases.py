"""The work users have this package do, as cases that can be prepared, run and compared.

Two kinds of programs use it.  A serving or evaluation program builds one ``MoELayer`` per layer and batch size and
calls it: replayed from its CUDA graph when the step has fixed buffers (entry ``graph``), or eagerly behind the router
gate when every step brings new ones (entry ``forward``).  A program written for MxMoE calls the operators of
``mxmoe_ops`` one after the other (entry ``ops``).  Layers have the shapes of the benchmark configurations; token
counts run from one decoded token to the largest prefill batch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mxmoe_b200 import mxmoe_ops, ops, workload
from mxmoe_b200.hadamard import hadamard_factor
from mxmoe_b200.layer import MoELayer
from mxmoe_b200.weights import parse_scheme, weight_bits

# experts, top-k, hidden, expert intermediate, shared experts (each as wide as a routed one), Zipf exponent of the
# routing (0: one favoured expert, softmax-like), 1 % outlier channels
FAMILIES = {
    "qwen15": dict(experts=60, topk=4, hidden=2048, inter=1408, shared=4, zipf=1.2, outliers=True),
    "ds2lite": dict(experts=64, topk=6, hidden=2048, inter=1408, shared=2, zipf=1.0, outliers=False),
    "mixtral": dict(experts=8, topk=2, hidden=4096, inter=14336, shared=0, zipf=0.0, outliers=True),
}
SCHEMES = {
    "qwen15": ("w4a4_g-1_sym", "w8a8_g-1_sym", "w4a16_g128_asym", "fp16", "mixed5"),
    "ds2lite": ("w4a4_g-1_sym", "w8a8_g-1_sym", "w4a16_g128_asym", "fp16", "mixed5"),
    "mixtral": ("w4a4_g-1_sym", "w8a8_g-1_sym", "mixed_w8w4"),
}


def _case(name, family, scheme, tokens, entry, shared=False, online_had=False):
    c = dict(family=family, scheme=scheme, tokens=tokens, entry=entry, shared=shared, online_had=online_had)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # one user waits for the next token: nothing but latency
        _case("decode-1", "ds2lite", "w4a16_g128_asym", 1, "graph", shared=True),
        # a decode batch of the weight-only configuration: three rows per expert
        _case("decode-32", "ds2lite", "w4a16_g128_asym", 32, "graph", shared=True),
        # a decode batch of odd size on the mixed-precision layer: every scheme in one launch
        _case("decode-61-mixed", "qwen15", "mixed5", 61, "graph", shared=True),
        # decode with few large experts: a gigabyte of weights for 32 rows
        _case("decode-16-mixtral", "mixtral", "mixed_w8w4", 16, "graph"),
        # an ordinary batch of a rotated w4a4 model, the down projection's input rotated online, behind the gate
        _case("batch-500-had", "qwen15", "w4a4_g-1_sym", 500, "forward", online_had=True),
        # a prompt chunk of odd length on the unquantised layer, behind the gate
        _case("chunk-1009-fp16", "qwen15", "fp16", 1009, "forward"),
        # the prefill batches of the benchmark configurations
        _case("prefill-8192-w4a4", "qwen15", "w4a4_g-1_sym", 8192, "graph"),
        _case("prefill-8192-mixed", "qwen15", "mixed5", 8192, "graph", shared=True),
        _case("prefill-8192-w4a16", "ds2lite", "w4a16_g128_asym", 8192, "graph", shared=True),
        _case("prefill-16384-mixtral", "mixtral", "mixed_w8w4", 16384, "graph"),
        # MxMoE's own sequence of operators: a decode batch and a prompt
        _case("ops-24-mixed", "qwen15", "mixed5", 24, "ops", shared=True),
        _case("ops-2000-mixed", "qwen15", "mixed5", 2000, "ops", shared=True),
    ]


def draw(rng):
    family = rng.choice(("qwen15", "ds2lite", "mixtral"))
    entry = rng.choice(("graph", "graph", "forward", "ops"))
    scheme = rng.choice(SCHEMES[family])
    most = 4096 if entry == "ops" else 8192
    tokens = min(most, max(1, round(math.exp(rng.uniform(0.0, math.log(most + 0.5))))))
    shared = FAMILIES[family]["shared"] > 0 and rng.random() < 0.5
    had = entry != "ops" and scheme == "w4a4_g-1_sym" and rng.random() < 0.3
    return _case(None, family, scheme, tokens, entry, shared=shared, online_had=had)


def _spec(case) -> workload.LayerSpec:
    f = FAMILIES[case["family"]]
    a4 = case["scheme"] not in ("fp16", "w4a16_g128_asym")
    return workload.LayerSpec(case["family"], f["experts"], f["topk"], f["hidden"], f["inter"],
                              f["inter"] * f["shared"] if case["shared"] else 0, case["tokens"], "zipf", f["zipf"],
                              f["outliers"], a4, case["scheme"])


def _log_popularity(case) -> np.ndarray:
    f = FAMILIES[case["family"]]
    if f["zipf"] == 0.0:
        return np.array([1.0] + [0.0] * (f["experts"] - 1))
    return -f["zipf"] * np.log(np.arange(1, f["experts"] + 1))


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    spec, f = _spec(case), FAMILIES[case["family"]]
    had = None
    if case["online_had"]:
        had = hadamard_factor(spec.inter)[0].to(dev)
    gate_up, down, signs, _ = workload.build_layer_weights(spec, seed=1000 + 4096 * seed, gen_device=dev, device=dev,
                                                           online_had=had)
    hidden = workload.make_hidden(spec, seed=seed, device=dev)
    # router logits: log popularity + Gumbel noise, so that the top-k of a token is a draw without replacement
    gen = torch.Generator(device=dev).manual_seed(seed + 77)
    u = torch.rand(spec.tokens, spec.num_experts, generator=gen, device=dev).clamp_(1e-7, 1 - 1e-7)
    logits = (torch.from_numpy(_log_popularity(case)).to(dev) - torch.log(-torch.log(u))).float().contiguous()
    ids, weights = ops.gate_topk(logits, spec.topk)
    s = dict(case=case, spec=spec, hidden=hidden, logits=logits, ids=ids, weights=weights)
    if case["entry"] == "ops":
        n_all = spec.num_experts + (1 if spec.shared_inter else 0)
        none = torch.empty(0, dtype=torch.float16, device=dev)
        for key, block in (("gate_up", gate_up), ("down", down)):
            s[key] = [block[e].data for e in range(n_all)]
            s[key + "_scale"] = [none if block[e].scale is None else block[e].scale for e in range(n_all)]
            s[key + "_q"] = [block[e].qparams for e in range(n_all)]
        s["shared"] = f["shared"] if spec.shared_inter else 0
        s["signs"] = None if signs is None else signs.to(dev)
        return s
    s["layer"] = MoELayer(spec.num_experts, spec.topk, spec.hidden, spec.inter, gate_up, down, spec.tokens,
                          shared_inter=spec.shared_inter, signs=signs, rotate=spec.rotate, device=dev,
                          online_had=None if had is None else had.half())
    return s


def run(s):
    entry = s["case"]["entry"]
    if entry == "graph":
        return s["layer"].forward_graph(s["hidden"], s["ids"], s["weights"])
    if entry == "forward":
        ids, weights = ops.gate_topk(s["logits"], s["spec"].topk)
        return {"out": s["layer"].forward(s["hidden"], ids, weights), "ids": ids, "weights": weights}
    spec, ns = s["spec"], s["shared"]
    T, k, E, H, I = spec.tokens, spec.topk, spec.num_experts, spec.hidden, spec.inter
    inp, inp_scale, out, _, _, out_store, recv, perm, experts_sorted = mxmoe_ops.quant_inp_act(
        s["hidden"], s["ids"], E, I, ns, s["gate_up_q"], rotate=spec.rotate, signs=s["signs"])
    mxmoe_ops.gg_mxmoe_share_fused(inp, s["gate_up"], inp_scale, s["gate_up_scale"], out, 2 * I, H, 2 * I * ns, H,
                                   s["gate_up_q"], recv)
    inp2, scale2, out2, _, _, out_store2 = mxmoe_ops.silu_mul_then_quant(
        out_store, len(inp), E, H, I, ns, T, k, experts_sorted, recv, s["down_q"])
    mxmoe_ops.gg_mxmoe_share_fused(inp2, s["down"], scale2, s["down_scale"], out2, H, I, H, I * ns, s["down_q"], recv)
    rows = T * k + (T if ns else 0)
    return {"out": out_store2[:rows * H], "recv": recv, "perm": perm, "experts": experts_sorted}


def work(case):
    """Hidden states and routing in, the weights of the experts that get a token, results out."""
    spec = _spec(case)
    T, H, I, E, k = spec.tokens, spec.hidden, spec.inter, spec.num_experts, spec.topk
    noise = np.random.RandomState(0).gumbel(size=(T, E))
    top = np.argpartition(-(noise + _log_popularity(case)), k - 1, axis=1)[:, :k]
    used = np.bincount(top.reshape(-1), minlength=E) > 0
    gu, dn = workload.draw_schemes(spec)
    weights = 0.0
    for e in range(len(gu)):
        inter = spec.shared_inter if e == E else I
        if e == E or used[e]:
            for scheme, n, kk in ((gu[e], 2 * inter, H), (dn[e], H, inter)):
                weights += n * kk * weight_bits(scheme) / 8 + (2 * n if parse_scheme(scheme)[2] == -1 and scheme != "fp16" else 0)
    rows_out = T * k + (T if spec.shared_inter else 0) if case["entry"] == "ops" else T
    routing = T * E * 4 + T * k * 8 if case["entry"] == "forward" else T * k * 8
    return {"bytes": T * H * 2 + routing + weights + rows_out * H * 2, "flops": float(spec.flops())}


def tolerance(case):
    """fp16 rounding of the three stages (gate_up, silu * up, down); where activations are quantised between them, a
    last-bit difference before the quantiser can move a code by one step."""
    return {"rel": 2e-3} if case["scheme"] in ("fp16", "w4a16_g128_asym") else {"rel": 1e-2}
