"""Which attention form serves a step's row blocks, and with how many KV splits (host side)."""
from types import SimpleNamespace

import pytest
import torch

from cubic_serve_b200.executor.gpu_executor import BatchBuilder, Segment
from cubic_serve_b200.models.decoder import DecoderRunner
from cubic_serve_b200.models.mtp import MtpRunner
from cubic_serve_b200.ops import kernels as K
from cubic_serve_b200.ops.strategies import active


def _fill(portions, hq=32, hkv=8, pad=None):
    """A step of ``(context, tokens)`` portions."""
    bb = BatchBuilder(max_rows=max(len(portions), pad or 0), max_tokens=8192, max_model_len=9000, group=hq // hkv, kv_heads=hkv, device="cpu")
    segs, page = [], 0
    for r, (start, n) in enumerate(portions):
        per = -(-(start + n) // 16)
        segs.append(Segment(r, [1] * n, start, list(range(page, page + per)), uid=r))
        page += per
    return bb.fill(segs, pad_rows_to=pad)[0]


@pytest.fixture
def launches(monkeypatch):
    """What a runner asks of paged attention: (row blocks, query rows of the first block, form, splits)."""
    made = []

    def attention(q, out, cache, table, req, qstart, qcount, ctx, hq, hkv, *_, scale=None, splits=1, ws=None, form=""):
        made.append((req.numel(), int(qstart[0]), form, splits))
        return out
    monkeypatch.setattr(K, "paged_attention", attention)
    return made


def _runner(hq=32, hkv=8):
    return SimpleNamespace(hq=hq, hkv=hkv, D=128, k_bits=8, v_bits=8, cfg=SimpleNamespace(attention_scale=None), ws=None)


def _draft_head(monkeypatch, hq, hkv, rows):
    for name in ("embedding", "rmsnorm", "wq_gemm"):
        monkeypatch.setattr(K, name, lambda x, *a, out=None, **k: x if out is None else out)
    monkeypatch.setattr(K, "rope_kv_write", lambda *a, **k: None)
    monkeypatch.setattr(K, "gate_up_act", lambda *a, **k: 1)
    cfg = SimpleNamespace(hidden_size=8, rms_eps=1e-6, rotary_dim=128, attention_scale=None)
    buf = lambda n: torch.zeros(rows, n)  # noqa: E731
    t = SimpleNamespace(cfg=cfg, tp=None, hq=hq, hkv=hkv, D=128, k_bits=8, v_bits=8, kv_rotation=False, ws=None, inv_freq=None,
                        w=SimpleNamespace(embed=buf(8), vocab_start=0), x=buf(8), qkv=buf(8), q=buf(hq * 128), attn=buf(hq * 128), gu=buf(8), act=buf(8))
    t._attend = lambda *a: DecoderRunner._attend(t, *a)
    head = MtpRunner.__new__(MtpRunner)
    head.t, head.kv, head.cat, head.emb, head.h, head.part = t, None, buf(16), buf(8), buf(8), None
    lw = SimpleNamespace(ln1=None, ln2=None, qkv=None, o=None, gate_up=None, down=None, q_norm=None, k_norm=None)
    head.w = SimpleNamespace(enorm=None, hnorm=None, fc=None, layer=lw)
    return head


@pytest.mark.parametrize("portions", [[(0, 1024)] * 8, [(0, 512)] * 4, [(0, 1200)], [(700, 1)] * 40 + [(0, 2000), (0, 2000)], [(100, 1)] * 7, [(2048, 256)] * 4])
@pytest.mark.parametrize("hq,hkv", [(32, 8), (64, 4), (8, 8)])
def test_partial_sums_of_target_and_draft_head_stay_small(monkeypatch, launches, portions, hq, hkv):
    b = _fill(portions, hq, hkv)
    if b.num_tokens > 2048 and len(portions) == 8 and hq == 32:
        assert b.attn_prompts == (0, 2048)
    q = torch.zeros(b.num_tokens, hq, 128)
    DecoderRunner._attend(_runner(hq, hkv), b, q, q, None, 0, b.num_row_blocks)
    target = list(launches)
    head = _draft_head(monkeypatch, hq, hkv, b.num_tokens)
    head.forward(b, torch.zeros(b.num_tokens, 8))
    assert launches == target * 2 and head.launches == 15 + len(target) - 1
    assert sum(n for n, *_ in target) == b.num_row_blocks
    # splits that fill the machine once (twice for the decode form, whose splits are rounded up from half as many blocks)
    assert all(s == 1 or n * hkv * s <= 4 * active().attention.target_ctas for n, _, _, s in target)
