"""The decode and prompt forms of paged attention against the general kernel (itself tested against the dense oracle) and, for one
layout, against the oracle."""

import pytest
import torch

from cubic_serve_b200.ops import eager

pytestmark = pytest.mark.gpu
DEV = "cuda"
D = 128


def _cache(tokens, hkv, kb, vb, seed):
    """Pages of random codes; token slots past a request's length hold NaN scales.  Returns the cache and the page table."""
    g = torch.Generator().manual_seed(seed)
    lay = eager.blob_layout(D, kb, vb)
    per = [-(-n // 16) for n in tokens]
    order = torch.randperm(sum(per), generator=g).tolist()
    blob = torch.randint(0, 256, (sum(per), hkv, lay["bytes"]), dtype=torch.uint8, generator=g)
    table = torch.zeros(len(tokens), max(per), dtype=torch.int32)
    at = 0
    for r, n in enumerate(tokens):
        for j in range(per[r]):
            page = order[at]
            at += 1
            table[r, j] = page
            for name, end, s in (("k_scale", "v_code", 0.05), ("v_scale", "bytes", 0.02)):
                scale = (torch.rand(hkv, 16, D // 32, generator=g) + 0.5) * s * 127 / ((1 << ((kb if name == "k_scale" else vb) - 1)) - 1)
                scale[:, max(0, n - 16 * j):] = float("nan")
                blob[page, :, lay[name]:lay[end]] = scale.reshape(hkv, -1).contiguous().view(torch.uint8).reshape(hkv, -1)
    return blob.to(DEV), table.to(DEV)


def _run(form, q, cache, table, blocks, hq, hkv, kb, vb, splits):
    from cubic_serve_b200.ops import kernels as K
    rb = [torch.tensor(c, dtype=torch.int32, device=DEV) for c in zip(*blocks)]
    out = torch.full_like(q, 7.0)
    K.paged_attention(q, out, cache, table, *rb, hq, hkv, D, kb, vb, scale=0.05, splits=splits, form=form)
    ws = K.workspace(torch.device(DEV, 0))
    ws.check_status()
    assert not ws.attn_counters.any()
    return out


def _close(a, b):
    """Probabilities are rounded to f16 (2^-11) relative to another running maximum (up to four times lower), sums run in another order, results are rounded
    to bf16 (2^-8): two steps of the value, or of a small part of the row's scale."""
    a, b = a.float(), b.float()
    assert torch.isfinite(a).all()
    return ((a - b).abs() <= 2.0 ** -7 * b.abs() + 2.0 ** -8 * b.square().mean(-1, keepdim=True).sqrt()).all()


@pytest.mark.parametrize("kb,vb", [(8, 8), (4, 8), (6, 6), (4, 4), (8, 4), (6, 8), (8, 6), (4, 6), (6, 4)])
@pytest.mark.parametrize("group", [1, 4, 8])
def test_decode_form(kb, vb, group):
    hkv = 2
    tokens = [1, 15, 16, 17, 47, 129, 1000, 300]
    cache, table = _cache(tokens, hkv, kb, vb, kb * vb + group)
    q = torch.randn(len(tokens), group * hkv, D, device=DEV, generator=torch.Generator(device=DEV).manual_seed(1)).bfloat16()
    blocks = [(r, r, 0 if r == 5 else 1, n) for r, n in enumerate(tokens)]                # request 5 is padding
    want = _run("", q, cache, table, blocks, group * hkv, hkv, kb, vb, 1)
    for splits in (1, 2, 7, 32):
        got = _run("decode", q, cache, table, blocks, group * hkv, hkv, kb, vb, splits)
        assert (got[5] == 7).all() and _close(got[:5], want[:5]) and _close(got[6:], want[6:])


@pytest.mark.parametrize("kb,vb", [(8, 8), (4, 8), (6, 6), (4, 4), (8, 4), (6, 8), (8, 6), (4, 6), (6, 4)])
@pytest.mark.parametrize("group", [1, 4, 8, 16])
def test_prompt_form(kb, vb, group):
    hkv, qb = 2, 16 // group
    portions = [(0, 1), (0, 3 * qb + 1), (37, 5), (0, 64), (15, 50), (500, 70), (0, 129)]   # (start, tokens) of every request
    cache, table = _cache([s + n for s, n in portions], hkv, kb, vb, kb * vb + group)
    T = sum(n for _, n in portions)
    q = torch.randn(T, group * hkv, D, device=DEV, generator=torch.Generator(device=DEV).manual_seed(2)).bfloat16()
    blocks, t = [], 0
    for r, (s, n) in enumerate(portions):
        blocks += [(r, t + i, min(qb, n - i), s + i + 1) for i in range(0, n, qb)]
        if r == 2:
            blocks.append((0, 0, 0, 0))                                                    # a padding block in between
        t += n
    want = _run("", q, cache, table, blocks, group * hkv, hkv, kb, vb, 1)
    assert _close(_run("prefill", q, cache, table, blocks, group * hkv, hkv, kb, vb, 1), want)


@pytest.mark.parametrize("form", ["decode", "prefill"])
def test_forms_against_the_oracle(form):
    hkv, group, n = 2, 4, 333
    cache, table = _cache([n], hkv, 8, 8, 5)
    rows = 1 if form == "decode" else 40
    q = torch.randn(rows, group * hkv, D, device=DEV, generator=torch.Generator(device=DEV).manual_seed(3)).bfloat16()
    kv = [[eager.decode_cache_page(cache[p, h].cpu(), D, 8, 8) for h in range(hkv)] for p in table[0].tolist()]
    k, v = (torch.stack([torch.cat([page[h][i] for page in kv])[:n] for h in range(hkv)], 1) for i in (0, 1))
    first = n - rows
    ref = eager.attention_rows(q.cpu(), k, v, torch.arange(first + 1, n + 1), 0.05)
    blocks = [(0, 0, 1, n)] if form == "decode" else [(0, i, min(4, rows - i), first + i + 1) for i in range(0, rows, 4)]
    assert _close(_run(form, q, cache, table, blocks, group * hkv, hkv, 8, 8, 2 if form == "decode" else 1).cpu(), ref)


def test_decode_form_reports_too_many_rows():
    from cubic_serve_b200.ops import kernels as K
    from cubic_serve_b200.ops.native import NativeLibraryError
    cache, table = _cache([40], 1, 8, 8, 6)
    q = torch.randn(4, 4, D, device=DEV).bfloat16()
    with pytest.raises(NativeLibraryError):
        _run("decode", q, cache, table, [(0, 0, 4, 37)], 4, 1, 8, 8, 1)
    with pytest.raises(NativeLibraryError):
        K.paged_attention(q.view(1, 16, D), torch.empty(1, 16, D, device=DEV, dtype=torch.bfloat16), cache, table, *(torch.ones(1, dtype=torch.int32, device=DEV) for _ in range(4)),
                          16, 1, D, 8, 8, form="decode")


def _scales(cache, kb, vb):
    """V scales of the cache as floats [page][head][token of the page][group]."""
    lay = eager.blob_layout(D, kb, vb)
    return cache[:, :, lay["v_scale"]:lay["bytes"]].view(torch.float32).view(cache.shape[0], cache.shape[1], 16, D // 32)


@pytest.mark.parametrize("kb,vb", [(8, 8), (4, 8), (6, 6), (8, 4)])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_prompt_form_keeps_values_to_those_who_see_them(kb, vb, bad):
    """An infinite value of one request reaches neither the requests that share a CTA with it nor earlier positions of its own."""
    hkv, group, qb = 2, 4, 4
    portions = [(0, 30), (20, 21), (0, 17), (5, 70)]
    cache, table = _cache([s + n for s, n in portions], hkv, kb, vb, 11)
    T = sum(n for _, n in portions)
    q = torch.randn(T, group * hkv, D, device=DEV, generator=torch.Generator(device=DEV).manual_seed(3)).bfloat16()
    blocks, t, rows = [], 0, []
    for r, (s, n) in enumerate(portions):
        blocks += [(r, t + i, min(qb, n - i), s + i + 1) for i in range(0, n, qb)]
        rows += [(r, s + i) for i in range(n)]
        t += n
    want = _run("prefill", q, cache, table, blocks, group * hkv, hkv, kb, vb, 1)
    for req, tok in ((1, 33), (3, 0), (3, 74)):
        hit = cache.clone()
        _scales(hit, kb, vb)[int(table[req, tok // 16]), :, tok % 16] = bad
        got = _run("prefill", q, hit, table, blocks, group * hkv, hkv, kb, vb, 1)
        sees = torch.tensor([r == req and p >= tok for r, p in rows], device=DEV)
        assert torch.equal(got[~sees], want[~sees])
        assert not torch.isfinite(got[sees].float()).all(-1).any()


@pytest.mark.parametrize("kb,vb", [(8, 8), (6, 4), (4, 6)])
def test_prompt_form_with_values_that_are_infinite_in_a_channel_group(kb, vb):
    """Infinite V scales of one channel group, of one token, of a few far apart, of all from some on: that group of the rows that see them is what
    the codes say, the other groups and rows keep their results."""
    group, n = 4, 300
    cache, table = _cache([n], 1, kb, vb, 25)
    q = torch.randn(n, group, D, device=DEV, generator=torch.Generator(device=DEV).manual_seed(11)).bfloat16()
    blocks = [(0, i, min(4, n - i), i + 1) for i in range(0, n, 4)]
    want = _run("prefill", q, cache, table, blocks, group, 1, kb, vb, 1)
    for toks in ([77], [3, 130, 299], range(150, n)):
        hit = cache.clone()
        for t in toks:
            _scales(hit, kb, vb)[int(table[0, t // 16]), 0, t % 16, 2] = float("inf")
        got = _run("prefill", q, hit, table, blocks, group, 1, kb, vb, 1)
        sees = torch.arange(n, device=DEV) >= min(toks)
        one = _request(hit, table, 0, n, kb, vb) if len(toks) == 1 else None
        assert torch.equal(got[~sees], want[~sees]) and not torch.isfinite(got[sees][..., 64:96].float()).any()
        if one:                                              # infinities by the sign of the token's codes, NaN where those are zero
            codes = one[1][toks[0], 64:96].float()
            assert torch.equal(got[sees][..., 64:96].cpu().float().nan_to_num(nan=0), codes.nan_to_num(nan=0).expand(int(sees.sum()), group, 32).nan_to_num(nan=0))
        for cols in (slice(0, 64), slice(96, 128)):
            assert _close(got[..., cols], want[..., cols])


@pytest.mark.parametrize("kb,vb", [(8, 8), (8, 4)])
@pytest.mark.parametrize("top", [16000.0, 16400.0, 40000.0, 65000.0])
def test_prompt_form_has_the_range_of_f16_for_scales(kb, vb, top):
    """Scales up to the largest f16: probabilities are at most one where four times a scale would not fit."""
    hkv, group, n = 2, 4, 700
    cache, table = _cache([n], hkv, kb, vb, 12)
    s = _scales(cache, kb, vb)
    s.mul_(top / s.nan_to_num().max())
    q = torch.randn(n, group * hkv, D, device=DEV, generator=torch.Generator(device=DEV).manual_seed(4)).bfloat16()
    blocks = [(0, i, min(4, n - i), i + 1) for i in range(0, n, 4)]
    want = _run("", q, cache, table, blocks, group * hkv, hkv, kb, vb, 1)
    assert torch.isfinite(want.float()).all() and _close(_run("prefill", q, cache, table, blocks, group * hkv, hkv, kb, vb, 1), want)


@pytest.mark.parametrize("kb,vb,group,hkv", [(8, 8, 4, 8), (6, 6, 16, 4), (4, 8, 1, 16)])
@pytest.mark.parametrize("portions", [[(0, 700), (33, 1), (900, 301), (0, 64), (5, 300)], [(63, 9000)], [(64 * i, 65) for i in range(20)]])
def test_prompt_form_with_more_items_than_ctas(kb, vb, group, hkv, portions):
    """A CTA takes several items of 256 rows, of unequal length, one after the other; 9000 tokens make more groups than are sorted."""
    qb = 16 // group
    if group == 1:
        portions = [(s, 4 * n) for s, n in portions if n < 9000] or [(0, 2600)]
    cache, table = _cache([s + n for s, n in portions], hkv, kb, vb, kb + group)
    T = sum(n for _, n in portions)
    q = torch.randn(T, group * hkv, D, device=DEV, generator=torch.Generator(device=DEV).manual_seed(5)).bfloat16()
    blocks, t = [], 0
    for r, (s, n) in enumerate(portions):
        blocks += [(r, t + i, min(qb, n - i), s + i + 1) for i in range(0, n, qb)]
        t += n
    assert -(-len(blocks) // 16) * hkv > torch.cuda.get_device_properties(0).multi_processor_count
    want = _run("", q, cache, table, blocks, group * hkv, hkv, kb, vb, 1)
    assert _close(_run("prefill", q, cache, table, blocks, group * hkv, hkv, kb, vb, 1), want)


@pytest.mark.parametrize("kb,vb", [(8, 8), (4, 6)])
@pytest.mark.parametrize("low,high", [(-6, 6), (-20, 0), (0, 30), (60, 100), (-110, -98)])
def test_prompt_form_with_scales_of_any_size(kb, vb, low, high):
    """V scales of 2^low to 2^high, larger from page to page: the powers of two that keep the operands in the range of f16 change on the way.
    (Results below 2^-126 would not be normal numbers.)"""
    hkv, group, n = 1, 4, 200
    cache, table = _cache([n], hkv, kb, vb, 13)
    pages = table[0, :13].tolist()
    factor = torch.tensor([2.0 ** round(low + (high - low) * i / 12) for i in range(13)], dtype=torch.float64)
    for i, page in enumerate(pages):
        s = _scales(cache, kb, vb)[page]
        s.copy_((s.double() * factor[i].item()).float())
    q = torch.randn(n, group * hkv, D, device=DEV, generator=torch.Generator(device=DEV).manual_seed(6)).bfloat16()
    blocks = [(0, i, min(4, n - i), i + 1) for i in range(0, n, 4)]
    got = _run("prefill", q, cache, table, blocks, group * hkv, hkv, kb, vb, 1)
    k, v = (torch.cat([eager.decode_cache_page(cache[p, 0].cpu(), D, kb, vb)[i] for p in pages])[:n].double() for i in (0, 1))
    z = torch.einsum("thd,sd->ths", q.cpu().double(), k) * 0.05
    z.masked_fill_(torch.arange(n)[None, None] > torch.arange(n)[:, None, None], float("-inf"))
    ref = torch.einsum("ths,sd->thd", z.softmax(-1), v)
    # relative to a power of two near the row's scale, so that _close's own arithmetic stays in range
    unit = torch.exp2(ref.abs().amax(-1, keepdim=True).log2().floor())
    assert _close((got.cpu().double() / unit), ref / unit)


def _scale_views(cache, kb, vb):
    """K and V scales of the cache as floats [page][head][token of the page][group]."""
    lay = eager.blob_layout(D, kb, vb)
    return [cache[:, :, lay[a]:lay[b]].view(torch.float32).view(cache.shape[0], cache.shape[1], 16, D // 32)
            for a, b in (("k_scale", "v_code"), ("v_scale", "bytes"))]


def _request(cache, table, r, n, kb, vb):
    """K and V of the first ``n`` tokens of a request with one key / value head, in 64 bits."""
    pages = [eager.decode_cache_page(cache[p, 0].cpu(), D, kb, vb) for p in table[r, :-(-n // 16)].tolist()]
    return [torch.cat([page[i] for page in pages])[:n].double() for i in (0, 1)]


def _softmax_of(q, k, v, first):
    """Rows [T, G, D] of positions first, first + 1, .. against keys and values, in 64 bits."""
    z = torch.einsum("thd,sd->ths", q.cpu().double(), k) * 0.05
    z.masked_fill_(torch.arange(k.shape[0])[None, None] > (first + torch.arange(q.shape[0]))[:, None, None], float("-inf"))
    return torch.einsum("ths,sd->thd", z.softmax(-1), v)


def _close_in_groups(got, ref):
    """As ``_close`` in every row and channel group, whatever the size of its values."""
    got, ref = got.cpu().double().unflatten(-1, (-1, 32)), ref.unflatten(-1, (-1, 32))
    unit = torch.exp2(ref.abs().amax(-1, keepdim=True).clamp_min(1e-300).log2().floor())
    return torch.isfinite(got).all() and _close(got / unit, ref / unit)


def _sharp(k, rows, group, seed):
    """Queries that see next to nothing but the key of their own position."""
    g = torch.Generator().manual_seed(seed)
    unit = k[-rows:] / k[-rows:].norm(dim=-1, keepdim=True).clamp_min(1e-30)
    return (unit[:, None] * 6000 + torch.randn(rows, group, D, generator=g)).bfloat16().to(DEV)


@pytest.mark.parametrize("kb,vb", [(8, 8), (4, 6), (6, 4)])
@pytest.mark.parametrize("first,last", [(6, -6), (12, -2), (30, 0), (60, -2), (-10, -14), (0, 40)])
def test_prompt_form_with_v_scales_that_fall(kb, vb, first, last):
    """V scales that shrink (or grow) from page to page, seen by rows that attend to their own position: what was large before is no measure
    of what comes."""
    group, n = 4, 600
    cache, table = _cache([n], 1, kb, vb, 19)
    for i, page in enumerate(table[0].tolist()):
        _scale_views(cache, kb, vb)[1][page] *= 2.0 ** round(first + (last - first) * i / table.shape[1])
    k, v = _request(cache, table, 0, n, kb, vb)
    q = _sharp(k, n, group, 8)
    got = _run("prefill", q, cache, table, [(0, i, min(4, n - i), i + 1) for i in range(0, n, 4)], group, 1, kb, vb, 1)
    assert _close_in_groups(got, _softmax_of(q, k, v, 0))


@pytest.mark.parametrize("kb,vb", [(8, 8), (4, 6)])
@pytest.mark.parametrize("apart", [12, 24, 30, 60, -24, -60])
def test_prompt_form_with_requests_of_other_scales_in_an_item(kb, vb, apart):
    """Requests whose V scales are far from their neighbours' in the same item: each has the result that it has by itself."""
    group, portions = 4, [(0, 12), (20, 21), (0, 9), (130, 22), (3, 40), (64, 30)]
    cache, table = _cache([s + n for s, n in portions], 1, kb, vb, 20)
    for r, (s, n) in enumerate(portions):
        _scale_views(cache, kb, vb)[1][table[r, :-(-(s + n) // 16)].long()] *= 2.0 ** (apart * (r % 2))
    T = sum(n for _, n in portions)
    q = torch.randn(T, group, D, device=DEV, generator=torch.Generator(device=DEV).manual_seed(9)).bfloat16()
    blocks, t = [], 0
    for r, (s, n) in enumerate(portions):
        blocks += [(r, t + i, min(4, n - i), s + i + 1) for i in range(0, n, 4)]
        t += n
    got = _run("prefill", q, cache, table, blocks, group, 1, kb, vb, 1)
    t = 0
    for r, (s, n) in enumerate(portions):
        assert _close_in_groups(got[t:t + n], _softmax_of(q[t:t + n], *_request(cache, table, r, s + n, kb, vb), s))
        t += n


@pytest.mark.parametrize("kb,vb", [(8, 8), (8, 6), (8, 4)])
@pytest.mark.parametrize("up,down", [(0, 6), (0, 11), (12, 11), (12, 20), (40, 20), (100, 60)])
def test_prompt_form_with_v_scales_apart_in_a_step(kb, vb, up, down):
    """Tokens, and channel groups of a token, far below others of the same step, alone or before them.  (2^-28 of scales of ordinary size is
    nothing to a product of a probability and a scale in f16 either.)"""
    group, n = 4, 150
    cache, table = _cache([n], 1, kb, vb, 21)
    g = torch.Generator().manual_seed(down)
    for at in range(n):
        factor = 2.0 ** up * torch.where(torch.rand(D // 32, generator=g) < (0.5 if at >= 10 else 1.1), 2.0 ** -down, 1.0)
        _scale_views(cache, kb, vb)[1][int(table[0, at // 16]), 0, at % 16] *= factor.to(DEV)
    k, v = _request(cache, table, 0, n, kb, vb)
    q = torch.cat([_sharp(k, n, 2, 10), torch.randn(n, 2, D, generator=g).bfloat16().to(DEV)], 1).contiguous()
    got = _run("prefill", q, cache, table, [(0, i, min(4, n - i), i + 1) for i in range(0, n, 4)], group, 1, kb, vb, 1)
    assert _close_in_groups(got, _softmax_of(q, k, v, 0))


@pytest.mark.parametrize("kb,vb", [(8, 8), (6, 8), (4, 8)])
@pytest.mark.parametrize("up,at", [(9, 40), (24, 40), (40, 63), (100, 0), (100, 100)])
def test_prompt_form_with_a_key_far_above_the_others(kb, vb, up, at):
    """One token's K scales far above those of its step: rows before it, and rows that it is nothing to, have the scores of the others."""
    group, n = 4, 130
    cache, table = _cache([n], 1, kb, vb, 22)
    _scale_views(cache, kb, vb)[0][int(table[0, at // 16]), 0, at % 16] *= 2.0 ** up
    k, v = _request(cache, table, 0, n, kb, vb)
    g = torch.Generator().manual_seed(up)
    q = torch.randn(n, group, D, generator=g).bfloat16()
    # half of the rows look away from it
    q[:, 2:] = torch.where(((q[:, 2:].double() * k[at]).sum(-1, keepdim=True) > 0), -q[:, 2:], q[:, 2:])
    q = q.to(DEV)
    got = _run("prefill", q, cache, table, [(0, i, min(4, n - i), i + 1) for i in range(0, n, 4)], group, 1, kb, vb, 1)
    assert _close_in_groups(got, _softmax_of(q, k, v, 0))


@pytest.mark.parametrize("kb,vb", [(8, 8), (4, 6)])
def test_prompt_form_with_k_scales_apart(kb, vb):
    """K scales of the tokens of a step 2^-40 to 1 of each other."""
    group, n = 4, 200
    cache, table = _cache([n], 1, kb, vb, 23)
    ks, g = _scale_views(cache, kb, vb)[0], torch.Generator().manual_seed(1)
    for at in range(n):
        ks[int(table[0, at // 16]), 0, at % 16] *= 2.0 ** -int(torch.randint(0, 41, (1,), generator=g))
    k, v = _request(cache, table, 0, n, kb, vb)
    q = torch.randn(n, group, D, generator=g).bfloat16().to(DEV)
    got = _run("prefill", q, cache, table, [(0, i, min(4, n - i), i + 1) for i in range(0, n, 4)], group, 1, kb, vb, 1)
    assert _close_in_groups(got, _softmax_of(q, k, v, 0))


@pytest.mark.parametrize("kb,vb,hkv", [(8, 8, 8), (4, 6, 16)])
def test_prompt_form_with_one_tile_ahead_of_the_other(kb, vb, hkv):
    """Items whose first tile sees one step and whose second sees many, the other way round, and with padding for a tile; several of a CTA."""
    group, qb = 4, 4
    kinds = [[(0, 32), (2000, 32)], [(700, 32), None], [(1500, 32), (3, 32)], [None, (64, 32)], [(0, 7), (129, 25), (900, 32)]]
    portions, blocks, t = [], [], 0
    for i in range(30):
        for portion in kinds[i % 5]:
            if portion is None:
                blocks += [(0, 0, 0, 0)] * 8
                continue
            s, n = portion
            blocks += [(len(portions), t + o, min(qb, n - o), s + o + 1) for o in range(0, n, qb)]
            portions.append(portion)
            t += n
        blocks += [(0, 0, 0, 0)] * (-len(blocks) % 16)
    assert len(blocks) // 16 * hkv > torch.cuda.get_device_properties(0).multi_processor_count
    cache, table = _cache([s + n for s, n in portions], hkv, kb, vb, 17)
    q = torch.randn(t, group * hkv, D, device=DEV, generator=torch.Generator(device=DEV).manual_seed(7)).bfloat16()
    want = _run("", q, cache, table, blocks, group * hkv, hkv, kb, vb, 1)
    assert _close(_run("prefill", q, cache, table, blocks, group * hkv, hkv, kb, vb, 1), want)


@pytest.mark.parametrize("form,splits", [("", 1), ("decode", 1), ("decode", 4), ("prefill", 1)])
def test_rows_that_see_no_token_are_zero(form, splits):
    """Alone in their CTA and beside rows that see something."""
    cache, table = _cache([70, 70], 1, 8, 8, 7)
    q = torch.randn(12, 4, D, device=DEV).bfloat16()
    for blocks in ([(0, 0, 1, 0)], [(0, 0, 1, 0), (1, 1, 1, 50)], [(0, 4 * i, 1, 0) for i in range(3)]):
        out = _run(form, q, cache, table, blocks, 4, 1, 8, 8, splits)
        assert all((out[t] == 0).all() for _, t, _, ctx in blocks if ctx == 0)
        assert all((out[t] != 0).any() and torch.isfinite(out[t].float()).all() for _, t, _, ctx in blocks if ctx)
