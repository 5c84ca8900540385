"""Routing and activation buffers of expert layers: one set a runner, made with it."""
import weakref
from types import SimpleNamespace

import pytest
import torch

from cubic_serve_b200.models.moe import MoeLayer


def _layer(n=256, top_k=2, local=4, shared=False):
    w = lambda n, k: SimpleNamespace(n=n, k=k)  # noqa: E731
    extra = dict(shared_gate_up=w(128, 64), shared_gate=w(8, 64)) if shared else {}
    return MoeLayer(None, w(n, 64), w(64, n // 2), (0, 0, 0, 0), 8, top_k, 0, local, **extra)


def test_layers_of_the_same_shapes_share_buffers():
    layers = [_layer(), _layer(shared=True), _layer(), _layer(n=512), _layer(top_k=4), _layer(local=2), _layer(shared=True), _layer()]
    for i, l in enumerate(layers):
        l.share_scratch(layers[:i], 16, 64, "cpu")
    owner = [next(j for j, o in enumerate(layers) if o.scratch is l.scratch) for l in layers]
    assert owner == [0, 1, 0, 3, 4, 5, 1, 0]
    for l, o in zip(layers, owner):
        assert l.out is layers[o].out and l.logits is layers[o].logits and l.least_rows == layers[o].least_rows == 32
        assert l.ensure_scratch(16, 64, "cpu") is l.scratch
    assert layers[6].sh_act is layers[1].sh_act
    # more tokens than the others hold: a set of its own
    more = _layer()
    more.share_scratch(layers, 17, 64, "cpu")
    assert more.scratch is not layers[0].scratch and more.scratch.topk_ids.shape[0] == 17


@pytest.mark.parametrize("shared", [False, True])
def test_buffers_of_a_smaller_runner_stay(shared):
    """A larger runner over the same weights: the graphs of the first one still write where they were captured."""
    layers = [_layer(shared=shared) for _ in range(3)]
    for i, l in enumerate(layers):
        l.share_scratch(layers[:i], 16, 64, "cpu")
    first = [weakref.ref(t) for t in (layers[0].scratch, layers[0].logits, layers[0].out, *((layers[0].sh_act, layers[0].sh_sig) if shared else ()))]
    for i, l in enumerate(layers):
        l.share_scratch(layers[:i], 32, 64, "cpu")
    assert all(l.scratch is layers[0].scratch and l.scratch.topk_ids.shape[0] == 32 for l in layers)
    assert all(r() is not None for r in first)
    for i, l in enumerate(layers):                      # the same runner again, or a smaller one: nothing new
        l.share_scratch(layers[:i], 16, 64, "cpu")
    assert [len(l.replaced) for l in layers] == [1, 1, 1]


@pytest.mark.gpu
def test_first_step_of_a_runner_makes_no_expert_buffers():
    from cubic_serve_b200.executor.gpu_executor import GpuExecutor, Segment
    from cubic_serve_b200.models.config import ModelConfig, QuantSpec
    from cubic_serve_b200.models.decoder import DecoderRunner, random_decoder_weights
    cfg = ModelConfig(name="buffers", family="gqa_moe", num_layers=4, hidden_size=512, num_q_heads=8, num_kv_heads=2, head_dim=128, intermediate_size=0, vocab_size=512,
                      rope_theta=1e6, num_experts=16, experts_per_token=8, moe_intermediate_size=256, quant=QuantSpec("nvfp4", 4, 16))
    ids = list(range(300))

    def step(own):
        runner = DecoderRunner(cfg, random_decoder_weights(cfg, "cuda", seed=0), num_pages=40, max_tokens=4096)
        if own:
            for lw in runner.w.layers:
                lw.moe.scratch = None
        ex = GpuExecutor(runner, max_rows=2, max_prefill_tokens=4096, max_model_len=512, use_graphs=False)
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        ex.execute([Segment(0, ids, 0, list(range(20)), True)])
        return runner.h[:300].clone(), torch.cuda.memory_allocated() - before
    shared, grown = step(False)
    own, set_each = step(True)
    assert torch.equal(shared, own)
    assert set_each > 4 * 4096 * 8 * (512 + 512 + 256 + 512) * 2 and grown < set_each // 8
