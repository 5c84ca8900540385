"""Steps whose row blocks are cut between the attention forms: runner, executor and draft head against the general kernel over all of them."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from cubic_serve_b200.models.config import ModelConfig, QuantSpec
from cubic_serve_b200.models.decoder import DecoderRunner

from test_gpu_paged_forms import _cache, _close, _run

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("group,hkv", [(4, 2), (16, 1), (1, 3)])
def test_attend_of_a_mixed_step(group, hkv):
    """Decode rows before, between and after portions of prompts, over cuts of the row blocks as lanes of a pipeline stage make them."""
    from cubic_serve_b200.ops import kernels as K
    qb = 16 // group
    portions = [(40, 1), (17, 1), (0, 90), (33, 70), (200, 1), (3, 4 * qb), (99, 2), (64, 1)]      # (context, tokens); the prompts are 2 and 3
    cache, table = _cache([s + n for s, n in portions], hkv, 8, 8, group)
    T = sum(n for _, n in portions)
    q = torch.randn(T, group * hkv, 128, device=DEV, generator=torch.Generator(device=DEV).manual_seed(6)).bfloat16()
    blocks, t, at = [], 0, []
    for r, (s, n) in enumerate(portions):
        at.append(len(blocks))
        blocks += [(r, t + i, min(qb, n - i), s + i + 1) for i in range(0, n, qb)]
        t += n
    want = _run("", q, cache, table, blocks, group * hkv, hkv, 8, 8, 1)
    rb = [torch.tensor(c, dtype=torch.int32, device=DEV) for c in zip(*blocks)]
    ws = K.workspace(torch.device(DEV, 0))
    runner = SimpleNamespace(hq=group * hkv, hkv=hkv, D=128, k_bits=8, v_bits=8, cfg=SimpleNamespace(attention_scale=0.05), ws=ws)
    b = SimpleNamespace(page_table=table, rb_req=rb[0], rb_qstart=rb[1], rb_qcount=rb[2], rb_ctx=rb[3], attn_splits=3, attn_decode=False, attn_prompts=(at[2], at[4]))
    n = len(blocks)
    for cut in (0, 1, at[2], at[2] + 3, at[3], at[4] - 1, at[4], n - 1):
        out = torch.full_like(q, 7.0)
        for lo, hi in ((0, cut), (cut, n)):
            DecoderRunner._attend(runner, b, q, out, cache, lo, hi)
        ws.check_status()
        assert _close(out, want)


def test_prompt_steps_of_a_speculative_executor():
    """Target and draft head take prompts through the prompt kernel, alone and beside a decoding request, with no more scratch than before."""
    from cubic_serve_b200.executor.gpu_executor import Segment
    from cubic_serve_b200.executor.spec_executor import SpeculativeGpuExecutor
    from cubic_serve_b200.models.decoder import random_decoder_weights
    from cubic_serve_b200.models.mtp import MtpRunner, random_mtp_weights
    from cubic_serve_b200.ops import kernels as K
    dev = torch.device("cuda")
    cfg = ModelConfig(name="routes", num_layers=2, hidden_size=512, num_q_heads=16, num_kv_heads=4, head_dim=128, intermediate_size=1024, vocab_size=2048,
                      rope_theta=1e6, quant=QuantSpec("cubic", 4, 128))
    n, pages = 1024, 66
    runner = DecoderRunner(cfg, random_decoder_weights(cfg, dev, seed=0, std=0.05), num_pages=8 * pages, max_tokens=8192)
    runner.ws = K.Workspace(dev)
    scratch = runner.ws.attn.numel()
    ex = SpeculativeGpuExecutor(runner, MtpRunner(runner, random_mtp_weights(cfg, dev, std=0.05)), 2, max_rows=8, max_prefill_tokens=8192, max_model_len=16 * pages)
    rng = np.random.default_rng(0)
    table = [list(range(r * pages, (r + 1) * pages)) for r in range(8)]
    prompts = [Segment(r, rng.integers(0, 2048, n).tolist(), 0, table[r], True, uid=r) for r in range(8)]
    mixed = [Segment(0, [5], n, table[0], True, uid=0)] + [Segment(r, rng.integers(0, 2048, n).tolist(), 0, table[r], True, uid=r) for r in range(1, 8)]
    made, attend = [], K.paged_attention

    def attention(*a, form="", **k):
        made.append(form)
        return attend(*a, form=form, **k)
    heads, forward = [], ex.mtp.forward
    ex.mtp.forward = lambda *a: heads.append(forward(*a).float()) or heads[-1]
    hidden, chosen = [], ex.builder._prompts
    try:
        K.paged_attention = attention
        for rule in (chosen, lambda blocks: (0, 0)):
            ex.builder._prompts = rule
            ex.last_hidden.zero_()
            for segs in (prompts, mixed):
                ex.execute(segs)
                hidden.append(ex.last_hidden.float())
    finally:
        K.paged_attention = attend
    runner.ws.check_status()
    layers = cfg.num_layers + 1
    assert made == ["prefill"] * layers + ["", "prefill"] * layers + [""] * 2 * layers
    assert runner.ws.attn.numel() == scratch
    for got, want in zip(hidden[:2] + heads[:2], hidden[2:] + heads[2:]):
        # a flipped rounding of an activation or a cache code moves what follows by parts of a bf16 step, layer after layer
        assert ((got - want).norm() / want.norm()).item() < 2e-2


@pytest.mark.parametrize("graphs", [True, False])
def test_review_passes_take_the_general_kernel(graphs):
    """16 query heads a key / value head: the rows of a review fill four row blocks a request, which portions of prompts of that length
    would leave to the prompt kernel behind short contexts."""
    from cubic_serve_b200.executor.gpu_executor import Segment
    from cubic_serve_b200.executor.spec_executor import SpeculativeGpuExecutor
    from cubic_serve_b200.models.decoder import random_decoder_weights
    from cubic_serve_b200.models.mtp import MtpRunner, random_mtp_weights
    from cubic_serve_b200.ops import kernels as K
    dev = torch.device("cuda")
    cfg = ModelConfig(name="review", num_layers=1, hidden_size=512, num_q_heads=64, num_kv_heads=4, head_dim=128, intermediate_size=512, vocab_size=512,
                      rope_theta=1e6, quant=QuantSpec("cubic", 4, 128))
    requests, pages = 64, 4
    runner = DecoderRunner(cfg, random_decoder_weights(cfg, dev, seed=0), num_pages=requests * pages, max_tokens=1024)
    ex = SpeculativeGpuExecutor(runner, MtpRunner(runner, random_mtp_weights(cfg, dev)), 3, max_rows=requests, max_prefill_tokens=1024, max_model_len=16 * pages,
                                round_graphs=graphs)
    table = [list(range(r * pages, (r + 1) * pages)) for r in range(requests)]
    ex.execute([Segment(r, list(range(16)), 0, table[r], True, uid=r) for r in range(requests)])
    made, attend = [], K.paged_attention

    def attention(*a, form="", **k):
        made.append(form)
        return attend(*a, form=form, **k)
    try:
        K.paged_attention = attention
        ex.execute_speculative([Segment(r, [5], 16, table[r], True, uid=r) for r in range(requests)])
    finally:
        K.paged_attention = attend
    runner.ws.check_status()
    assert made and set(made) == {""}
    assert ex.stats["graphed_rounds"] == int(graphs)
    ex._round_graph.clear()
