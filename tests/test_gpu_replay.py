"""Mixed-precision decode layers replayed back to back: thousands of launches whose weight loads land out of order (several
layers, a gigabyte of weights: more than the caches and address translations hold) must all give the first launch's bits."""
import numpy as np
import pytest
import torch

from mxmoe_b200 import gg, ops, workload
from mxmoe_b200.layer import MoELayer
from tests import util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family,tokens", [("qwen15", 61), ("mixtral", 16), ("qwen15", 1500)])
def test_replays_give_the_same_bits(cuda_device, family, tokens):
    if family == "qwen15":
        spec = workload.LayerSpec("qwen15", 60, 4, 2048, 1408, 5632, tokens, "zipf", 1.2, True, True, "mixed5")
    else:
        spec = workload.LayerSpec("mixtral", 8, 2, 4096, 14336, 0, tokens, "softmax_biased", 0.0, True, True, "mixed_w8w4")
    layers = []
    for seed in range(3):
        gu, dn, signs, _ = workload.build_layer_weights(spec, seed=1000 + 4096 * seed, gen_device=cuda_device,
                                                        device=cuda_device)
        x = workload.make_hidden(spec, seed=seed, device=cuda_device)
        ids, w = workload.make_routing(spec, seed=seed)
        ids, w = ids.to(cuda_device), w.to(cuda_device)
        layer = MoELayer(spec.num_experts, spec.topk, spec.hidden, spec.inter, gu, dn, tokens,
                         shared_inter=spec.shared_inter, signs=signs, rotate=spec.rotate, device=cuda_device)
        layers.append((layer, x, ids, w, layer.forward_graph(x, ids, w).clone()))
    for _ in range(10):
        for _ in range(60):
            for layer, x, ids, w, _ in layers:
                layer.forward_graph(x, ids, w)
        for layer, x, ids, w, first in layers:
            assert torch.equal(layer.forward_graph(x, ids, w), first)
            layer.check()


@pytest.mark.parametrize("rows", [(23, 1, 32, 17, 8, 31), (200, 33, 385, 96, 191, 64)], ids=["short-tiles", "long-tiles"])
def test_packed_activations_replay_bit_exact(cuda_device, rows):
    """Packed 4-bit activations are expanded into shared memory by threads of both CTAs of a pair and read by MMAs that one
    thread of the first CTA issues: every one of many launches gives the oracle's bits."""
    rng = np.random.default_rng(len(rows) + rows[0])
    cases = [util.WxAxCase(rng, m, n, 1408, 4) for m, n in zip(rows, (768, 640, 512, 1024, 384, 896))]
    g = gg.GroupedGemm([c.problem(cuda_device) for c in cases])
    want = [torch.from_numpy(c.ref.view(np.int16).copy()).to(cuda_device) for c in cases]
    wrong = torch.zeros((), dtype=torch.int64, device=cuda_device)
    for _ in range(300):
        for c in cases:
            c.C.fill_(float("nan"))
        g.run(kernel="swap2")
        for c, w in zip(cases, want):
            wrong += (c.C.view(torch.int16) != w).sum()
    g.check()
    assert int(wrong) == 0


@pytest.mark.parametrize("side_stream", [False, True])
def test_eager_chain_with_changing_inputs(cuda_device, side_stream):
    """Launches of the chain overlap: every step of an eager loop over two inputs and routings, whose buffers all steps share,
    gives the bits of that input alone, with nothing between the steps that would separate them."""
    spec = workload.LayerSpec("tiny", 12, 3, 1024, 768, 768, 150, "zipf", 1.2, True, True, "mixed5")
    gu, dn, signs, _ = workload.build_layer_weights(spec, gen_device=cuda_device, device=cuda_device)
    layer = MoELayer(spec.num_experts, spec.topk, spec.hidden, spec.inter, gu, dn, spec.tokens,
                     shared_inter=spec.shared_inter, signs=signs, rotate=spec.rotate, device=cuda_device)
    inputs, want = [], []
    for seed in range(2):
        gen = torch.Generator(device=cuda_device).manual_seed(seed)
        x = workload.make_hidden(spec, seed=seed, device=cuda_device)
        logits = torch.randn(spec.tokens, spec.num_experts, generator=gen, device=cuda_device)
        inputs.append((x, logits))
        ids, w = ops.gate_topk(logits, spec.topk)
        want.append(layer.forward(x, ids, w).clone())
        torch.cuda.synchronize()
    assert not torch.equal(want[0], want[1])
    stream = torch.cuda.Stream() if side_stream else torch.cuda.current_stream()
    wrong = torch.zeros((), dtype=torch.int64, device=cuda_device)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        for step in range(400):
            for i in (step & 1, 1 - (step & 1)):
                ids, w = ops.gate_topk(inputs[i][1], spec.topk)
                out = layer.forward(inputs[i][0], ids, w)
                if step % 4 == 0:      # otherwise the next step follows at once
                    wrong += (out.view(torch.int16) != want[i].view(torch.int16)).sum()
    torch.cuda.synchronize()
    layer.check()
    assert int(wrong) == 0
