"""Which attention form serves a step's row blocks, and with how many KV splits (host side)."""
from types import SimpleNamespace

import pytest
import torch

from cubic_serve_b200.executor.gpu_executor import BatchBuilder, Segment
from cubic_serve_b200.models.decoder import DecoderRunner
from cubic_serve_b200.models.mtp import MtpRunner
from cubic_serve_b200.ops import kernels as K
from cubic_serve_b200.ops.strategies import active


def _fill(portions, hq=32, hkv=8, pad=None, review=False):
    """A step of ``(context, tokens)`` portions."""
    bb = BatchBuilder(max_rows=max(len(portions), pad or 0), max_tokens=9000, max_model_len=9000, group=hq // hkv, kv_heads=hkv, device="cpu")
    segs, page = [], 0
    for r, (start, n) in enumerate(portions):
        per = -(-(start + n) // 16)
        segs.append(Segment(r, [1] * n, start, list(range(page, page + per)), uid=r))
        page += per
    b = bb.fill(segs, pad_rows_to=pad, review=review)[0]
    bb.stage.upload()
    return b


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


@pytest.mark.parametrize("hq,hkv,portions,prompt", [
    (32, 8, [(0, 1024)] * 8, True), (32, 8, [(2048, 256)] * 4, True), (32, 8, [(0, 2048)], True), (32, 8, [(0, 64)] * 16, True), (32, 8, [(0, 331)], False),
    (32, 8, [(240, 104)] * 7, False), (32, 8, [(300, 20)] * 40, False), (32, 8, [(4000, 64)], False), (32, 32, [(240, 104)] * 7, False), (32, 32, [(0, 2048)], True),
    (64, 4, [(1000, 128)] * 2, True), (64, 4, [(4000, 64)], False), (16, 2, [(0, 2048)], True), (16, 2, [(0, 700)], False), (16, 1, [(0, 2048)], True),
    (8, 1, [(0, 1100)], False), (8, 8, [(0, 200)] * 30, False), (8, 8, [(3000, 1000)], False)])
def test_prompts_take_the_kernel_that_was_measured_faster(hq, hkv, portions, prompt):
    b = _fill(portions, hq, hkv)
    assert b.attn_prompts == ((0, b.num_row_blocks) if prompt else (0, 0)) and not b.attn_decode


@pytest.mark.parametrize("hq,hkv,portions,prompt", [
    (32, 32, [(0, 64)] * 5, False), (32, 32, [(0, 64), (0, 40), (0, 33), (0, 64), (0, 51)], False), (16, 1, [(0, 26 - i % 19) for i in range(40)], False),
    (32, 8, [(0, 64)] * 8, True)])
def test_short_prompts_take_the_kernel_that_was_measured_faster(hq, hkv, portions, prompt):
    b = _fill(portions, hq, hkv)
    assert b.attn_prompts == ((0, b.num_row_blocks) if prompt else (0, 0))


@pytest.mark.parametrize("hq,hkv,portions,prompts", [
    (32, 8, [(1000, 1)] * 64 + [(0, 512)] * 2, (64, 320)), (32, 4, [(700, 1)] * 20 + [(0, 512)] * 2 + [(700, 1)] * 20, (0, 0)),
    (16, 1, [(1000, 4)] * 32 + [(0, 1024)] * 4, (0, 0)),               # the long review CTAs would start last
    (8, 8, [(1000, 4)] * 32 + [(0, 1024)] * 4, (0, 0)), (32, 8, [(1000, 4)] * 32 + [(0, 1024)] * 4, (32, 1056)), (8, 8, [(1000, 1)] * 64 + [(0, 1024)] * 7, (0, 0))])
def test_prompts_beside_other_rows(hq, hkv, portions, prompts):
    assert _fill(portions, hq, hkv).attn_prompts == prompts


@pytest.mark.parametrize("hq,hkv,depth,requests", [(64, 4, 3, 64), (32, 4, 7, 64), (16, 2, 7, 128), (32, 2, 3, 128), (32, 8, 3, 8)])
def test_review_rows_are_launched_alike_behind_any_context(hq, hkv, depth, requests):
    """A captured review pass serves later rounds, whose contexts are longer."""
    steps = [_fill([(c, depth + 1)] * requests, hq, hkv, review=True) for c in (20, 100, 1000, 4000)]
    assert all(b.attn_prompts == (0, 0) and not b.attn_decode and b.attn_splits == steps[0].attn_splits for b in steps)


DECODE, PROMPT = (900, 1), (0, 1024)


@pytest.mark.parametrize("hq,hkv", [(32, 8), (16, 1)])              # blocks of four positions and of one
@pytest.mark.parametrize("portions,first", [([PROMPT] * 8, 0), ([DECODE] * 5 + [PROMPT] * 8, 5), ([PROMPT] * 8 + [DECODE] * 5, 0), ([DECODE] * 3 + [PROMPT] * 8 + [(10, 2)] + [DECODE], 3),
                                            ([PROMPT] + [DECODE] + [PROMPT] * 6 + [(5, 3)] + [PROMPT], 2)])
def test_a_step_of_prompts_and_other_rows_is_cut_once(launches, portions, first, hq, hkv):
    """The longest run of prompts in one launch, what is before and after it in one each, with the splits of those alone."""
    b = _fill(portions, hq, hkv)
    qb = 16 // (hq // hkv)
    blocks = [-(-n // qb) for _, n in portions]
    run = 6 if PROMPT in portions[:1] and DECODE in portions[1:2] else 8
    lo, hi = sum(blocks[:first]), sum(blocks[:first + run])
    assert b.attn_prompts == (lo, hi)
    rest = b.num_row_blocks - (hi - lo)
    splits = min(active().attention.max_splits, max(1, -(-active().attention.target_ctas // max(1, rest * hkv))))
    q = torch.zeros(b.num_tokens, hq, 128)
    made = [(n, form, s) for n, form, s in ((lo, "", splits), (hi - lo, "prefill", 1), (b.num_row_blocks - hi, "", splits)) if n]
    assert DecoderRunner._attend(_runner(hq, hkv), b, q, q, None, 0, b.num_row_blocks) == len(made)
    assert [(n, form, s) for n, _, form, s in launches] == made
    # lanes of a pipeline stage: any cut gives every block to the same form
    form_of = ["prefill" if lo <= i < hi else "" for i in range(b.num_row_blocks)]
    for cut in (1, lo, lo + 9, hi - 1, hi, b.num_row_blocks - 1):
        launches.clear()
        for rb0, rb1 in ((0, cut), (cut, b.num_row_blocks)):
            DecoderRunner._attend(_runner(hq, hkv), b, q, q, None, rb0, rb1)
        got = [form for n, _, form, _ in launches for _ in range(n)]
        assert got == form_of
        at = 0
        for n, qstart, _, _ in launches:
            assert qstart == int(b.rb_qstart[at])
            at += n


def test_decode_steps_take_the_decode_form(launches):
    for hq, hkv, form in ((32, 8, "decode"), (8, 8, "decode"), (16, 1, "")):
        b = _fill([(100 + i, 1) for i in range(7)], hq, hkv, pad=8)
        q = torch.zeros(8, hq, 128)
        assert DecoderRunner._attend(_runner(hq, hkv), b, q, q, None, 0, 8) == 1
        assert launches.pop()[:3] == (8, 0, form)
