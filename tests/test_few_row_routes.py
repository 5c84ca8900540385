"""Which kernel a weight GEMM of few rows is given to (host side: the native library is a list of the calls made)."""
from types import SimpleNamespace

import pytest
import torch

from cubic_serve_b200.ops import autotune, kernels as K, native, strategies, wq_pack


class Calls:
    def __init__(self):
        self.made = []

    def __getattr__(self, name):
        def call(*args):
            if name.startswith("cb_wq_gemm_workspace"):
                return 1 << 20
            self.made.append((name, args))
            return 0
        return call


@pytest.fixture
def calls(monkeypatch):
    c = Calls()
    monkeypatch.setattr(native, "lib", lambda: c)
    monkeypatch.setattr(K, "_stream", lambda: 0)
    monkeypatch.setattr(K, "sm_count", lambda _: 148)
    return c


def _ws(gemm=64 << 20, counters=1 << 16):
    return SimpleNamespace(gemm=torch.empty(gemm, dtype=torch.uint8), gemm_counters=torch.zeros(counters, dtype=torch.int32), status=torch.zeros(1, dtype=torch.int32))


def _route(calls, m, w, act=False, **kw):
    x = torch.zeros(m, w.k, dtype=torch.bfloat16)
    kw.setdefault("ws", _ws())
    (K.wq_gemm_act if act else K.wq_gemm)(x, w, **kw)
    return calls.made.pop()[0]


def _weight(fmt=wq_pack.FMT_CUBIC4, n=512, k=1024, act=False):
    return autotune._random_weight(fmt, n, k, act, "cpu")


@pytest.mark.parametrize("m", [1, 8, 16])
@pytest.mark.parametrize("act", [False, True])
def test_an_installed_plan_comes_before_the_rule(calls, m, act):
    w = _weight(act=act)
    assert _route(calls, m, w, act) == "cb_wq_gemm_skinny"
    try:
        autotune.install({autotune.plan_key(w.fmt, m, w.n, w.k, act): {"use": True, "kernel": "tile", "splits": 3}})
        assert _route(calls, m, w, act) == ("cb_wq_gemm_act" if act else "cb_wq_gemm_tp")
        autotune.install({autotune.plan_key(w.fmt, m, w.n, w.k, act): {"use": True, "kernel": "stream_k", "splits": 0}})
        assert _route(calls, m, w, act) == ("cb_wq_gemm_act" if act else "cb_wq_gemm_sk")
        autotune.install({autotune.plan_key(w.fmt, m + 1, w.n, w.k, act): {"use": True, "kernel": "tile", "splits": 3}})
        assert _route(calls, m, w, act) == "cb_wq_gemm_skinny"
    finally:
        autotune.install(None)


def test_the_operator_configuration_sets_the_thresholds(calls):
    w, head, small = _weight(), _weight(wq_pack.FMT_BF16, 19072, 128), _weight(wq_pack.FMT_BF16, 512, 128)
    routes = lambda: [_route(calls, m, a) == "cb_wq_gemm_skinny" for a, m in ((w, 16), (w, 17), (head, 32), (head, 33), (small, 8), (small, 9))]  # noqa: E731
    assert routes() == [True, False] * 3
    old = strategies.active()
    try:
        strategies.install(strategies.operator_config_from_dict({"gemm": {"few_rows_quantized": 0, "few_rows_bf16": 9, "few_rows_bf16_streamed": 0},
                                                                 "moe": {"few_rows_per_expert": 3, "rows_per_item_by_load": False}}))
        assert routes() == [False, False, False, False, True, True]
        assert K.skinny_rows_per_expert() == 3 and K.rows_per_work_item(8192, 128, 64) == 64
    finally:
        strategies.install(old)
    for bad in ({"gemm": {"few_rows_quantized": 33}}, {"gemm": {"few_rows_bf16": -1}}, {"moe": {"few_rows_per_expert": -1}}):
        with pytest.raises(ValueError):
            strategies.operator_config_from_dict(bad)


@pytest.mark.parametrize("m,need", [(1, 2424832), (8, 2424832), (9, 4849664), (16, 4849664)])
def test_a_workspace_too_small_for_the_parts_takes_the_other_kernels(calls, m, need):
    w = _weight()
    assert _route(calls, m, w, ws=_ws(gemm=need)) == "cb_wq_gemm_skinny" and _route(calls, m, w, ws=_ws(gemm=need - 1)) == "cb_wq_gemm_tp"
    assert _route(calls, m, w, ws=_ws(counters=4)) == "cb_wq_gemm_skinny" and _route(calls, m, w, ws=_ws(counters=3)) == "cb_wq_gemm_tp"
    act = _weight(act=True)
    assert _route(calls, m, act, True, ws=_ws(gemm=need - 1)) == "cb_wq_gemm_act"


@pytest.mark.parametrize("stride,at,takes", [(512, 0, True), (516, 4, True), (516, 1, False), (516, 2, False), (514, 1, True), (513, 3, True)])
def test_results_that_start_anywhere(calls, stride, at, takes):
    """Only rows a multiple of four elements apart are written four elements at a time."""
    w = _weight()
    out = torch.empty(at + 8 * stride, dtype=torch.bfloat16)[at:].view(8, stride)[:, :512]
    even = torch.empty(8 * stride, dtype=torch.bfloat16).view(8, stride)[:, :512]
    assert _route(calls, 8, w, out=out) == ("cb_wq_gemm_skinny" if takes else "cb_wq_gemm_tp")
    assert _route(calls, 8, w, out=even, residual=out) == ("cb_wq_gemm_skinny" if takes else "cb_wq_gemm_tp")


@pytest.mark.parametrize("ranks", [1, 2, 8])
@pytest.mark.parametrize("tokens,entry", [(16, "cb_wq_gemm_skinny_grouped"), (64, "cb_wq_gemm_skinny_grouped"), (65, "cb_wq_gemm_grouped"), (200, "cb_wq_gemm_grouped")])
def test_rows_of_an_expert_count_over_all_ranks(calls, ranks, tokens, entry):
    """32 experts, 8 a token: 16 rows an expert at 64 tokens, whichever rank owns them."""
    local, rows = 32 // ranks, tokens * 8
    w = wq_pack.PackedWeight(wq_pack.FMT_NVFP4, 128, 256, 16, torch.zeros(local, 16), torch.zeros(local, 16), 1.0)
    sc = K.MoeScratch(tokens, 8, 256, 128, local, 32, "cpu", experts=32)
    K.wq_gemm_grouped(torch.zeros(rows, 256, dtype=torch.bfloat16), w, torch.empty(rows, 128, dtype=torch.bfloat16), rows, sc, 16, 16, _ws())
    assert calls.made.pop()[0] == entry


@pytest.mark.parametrize("routes,mb,n,k,fmt,entry", [
    (24, 32, 1536, 2048, wq_pack.FMT_NVFP4, "cb_wq_gemm_skinny_grouped"), (25, 32, 1536, 2048, wq_pack.FMT_NVFP4, "cb_wq_gemm_ts_grouped"),
    (4096, 128, 1536, 2048, wq_pack.FMT_CUBIC4, "cb_wq_gemm_ts_grouped"), (4096, 144, 1536, 2048, wq_pack.FMT_CUBIC4, "cb_wq_gemm_grouped"),
    (4096, 128, 384, 2048 + 64, wq_pack.FMT_AFFINE4, "cb_wq_gemm_grouped"), (4096, 128, 384, 2048, wq_pack.FMT_BF16, "cb_wq_gemm_grouped")])
def test_experts_with_two_tiles_for_every_sm(calls, routes, mb, n, k, fmt, entry):
    w = wq_pack.PackedWeight(fmt, n, k, 128, torch.zeros(128, 16), torch.zeros(128, 16), 1.0)
    sc = SimpleNamespace(experts=128, local_experts=128, mb=mb, tiles=torch.zeros(1, dtype=torch.int32), items=lambda rows: rows)
    K.wq_gemm_grouped(torch.zeros(routes, k, dtype=torch.bfloat16), w, torch.empty(routes, n, dtype=torch.bfloat16), routes, sc, 16, 16, _ws())
    assert calls.made.pop()[0] == entry
    assert K.rows_per_work_item(4096, 64, 64, (w,), 128) == (128 if n * k == 1536 * 2048 and fmt != wq_pack.FMT_BF16 else 96)
    assert K.rows_per_work_item(1024, 64, 64, (w,), 128) == 64 and K.rows_per_work_item(4096, 64, 160, (w,), 128) == 160


@pytest.mark.parametrize("n,k,rows,others", [(24576, 4096, (129, 331, 512), (513, 8192)), (6144, 4096, (331, 512), (200, 600)), (4096, 4096, (129, 256), (331, 512)),
                                            (2048, 4096, (200, 512), (513, 768)), (512, 1024, (), (129, 512))])
def test_batches_of_more_rows_than_a_block(n, k, rows, others):
    """28 units an SM, or parts of a tile's own, up to 512 rows: on both sides of the lines."""
    w, ws = SimpleNamespace(fmt=wq_pack.FMT_NVFP4, n=n, k=k, group_k=16), _ws()
    takes = lambda m, ws=ws: K.use_ts(m, w, torch.empty(m, k, dtype=torch.bfloat16), ws=ws)  # noqa: E731
    assert all(takes(m) for m in rows) and not any(takes(m) for m in others)
    for m in rows[:1]:
        blocks = -(-m // 128)
        need, tiles = 2 * 148 * -(-(-(-m // blocks)) // 16) * 16 * 512, n // 128 * blocks
        assert takes(m, _ws(gemm=need, counters=tiles)) and not takes(m, _ws(gemm=need - 1)) and not takes(m, _ws(counters=tiles - 1))
    old = strategies.active()
    try:
        strategies.install(strategies.operator_config_from_dict({"gemm": {"tensor_memory_rows": 112}}))
        assert not any(takes(m) for m in rows)
    finally:
        strategies.install(old)


@pytest.mark.parametrize("n,k,takes,others", [
    (4096, 4096, (1, 8, 64, 128, 129, 256), (257,)), (6144, 4096, (1, 8, 96, 128), (129,)), (8192, 2048, (1, 64, 128), (129,)), (10240, 2048, (1, 64, 96), (97, 128)),
    (14336, 1024, (), (0, 1, 9, 64, 128)), (2560, 9728, (1, 128), ()), (3584, 5120, (9, 96, 128), ()), (2048, 8192, (1, 64, 88), (89, 128)),
    (1024, 16384, (1, 9, 64), (65, 128)), (1024, 8192, (129, 192, 257, 512), (64, 128, 256))])
def test_lines_of_the_kernel_with_tiles_in_tensor_memory(n, k, takes, others):
    w = SimpleNamespace(fmt=wq_pack.FMT_CUBIC4, n=n, k=k, group_k=128)
    use = {m: K.use_ts(m, w, torch.empty(m, k, dtype=torch.bfloat16), ws=_ws()) for m in takes + others}
    assert use == {m: m in takes for m in takes + others}


def test_blocks_of_rows_have_a_limit_of_their_own():
    w, ws, old = SimpleNamespace(fmt=wq_pack.FMT_CUBIC4, n=24576, k=4096, group_k=128), _ws(), strategies.active()
    takes = lambda m: K.use_ts(m, w, torch.empty(m, 4096, dtype=torch.bfloat16), ws=ws)  # noqa: E731
    try:
        for most, rows, others in ((0, (1, 128), (129, 512)), (300, (128, 129, 300), (301, 512)), (700, (128, 512, 700), (701,))):
            strategies.install(strategies.operator_config_from_dict({"gemm": {"tensor_memory_rows_in_blocks": most}}))
            assert all(takes(m) for m in rows) and not any(takes(m) for m in others)
        with pytest.raises(ValueError):
            strategies.install(strategies.operator_config_from_dict({"gemm": {"tensor_memory_rows_in_blocks": -1}}))
    finally:
        strategies.install(old)
