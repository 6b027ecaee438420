"""Mixed-precision decode layers replayed back to back: thousands of launches whose weight loads land out of order (several
layers, a gigabyte of weights: more than the caches and address translations hold) must all give the first launch's bits."""
import numpy as np
import pytest
import torch

from mxmoe_b200 import gg, workload
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
