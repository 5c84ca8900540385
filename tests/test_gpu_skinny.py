"""The weight GEMM for few batch rows (csrc/wq_gemm_skinny.cu) against the dense matrix and against the per-tile kernel."""
import pytest
import torch

from cubic_serve_b200.ops import wq_pack

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _weight(fmt, n, k, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    rand = lambda *s: torch.rand(*s, device=DEV, generator=g)  # noqa: E731
    if fmt == "cubic":
        codes = torch.randint(-7, 8, (n, k), device=DEV, generator=g, dtype=torch.int8)
        return wq_pack.pack_cubic4(codes, rand(n, k // 128) * 0.05, 0.5 + rand(n, k // 128), rand(n, k // 128) - 0.5, 128)
    if fmt == "affine":
        q = torch.randint(0, 16, (n, k), device=DEV, generator=g, dtype=torch.uint8)
        return wq_pack.pack_affine4(q, rand(n, k // 32) * 0.02, -rand(n, k // 32) * 0.2, 32)
    if fmt == "nvfp4":
        q = torch.randint(0, 256, (n, k // 2), device=DEV, generator=g, dtype=torch.uint8)
        return wq_pack.pack_nvfp4(q, (rand(n, k // 16) * 8).to(torch.float8_e4m3fn), 0.01)
    return wq_pack.pack_bf16((rand(n, k) - 0.5) * 0.1)


def _close(y, y0, k):
    """Both kernels multiply the same bf16 operands into fp32 sums of another order (2^-24 of the sum of magnitudes for each of K
    terms, well below a bf16 step of the largest results) and round once: a step of bf16 apart at most, near zero that of the scale."""
    y, y0 = y.float(), y0.float()
    return ((y - y0).abs() <= 2.0 ** -7 * y0.abs() + 2.0 ** -9 * y0.square().mean().sqrt()).all()


@pytest.mark.parametrize("fmt", ["cubic", "affine", "nvfp4", "bf16"])
@pytest.mark.parametrize("n,k", [
    (128, 256),            # one tile, one iteration (two for bf16)
    (200, 768),            # a tile with 72 rows of padding, three parts
    (1000, 1280),          # five parts of a tile, the last tile short
    (4096, 2048),          # aligned runs
    (24576, 1024),         # runs that straddle tiles
])
def test_skinny_gemm(fmt, n, k):
    from cubic_serve_b200.ops import kernels as K
    w = _weight(fmt, n, k, n + k)
    dense = wq_pack.unpack_to_dense(w)[:n]
    g = torch.Generator(device=DEV).manual_seed(1)
    for m in (1, 2, 7, 8, 9, 15, 16) + ((17, 31, 32) if fmt == "bf16" and n > 148 * 128 else ()):
        wide = torch.randn(m, k + 64, device=DEV, generator=g).bfloat16()
        x, res = wide[:, :k], torch.randn(m, n, device=DEV, generator=g).bfloat16()
        assert m <= 8 or fmt != "bf16" or n > 148 * 128 or not K.use_skinny(m, w, x)
        ref = x.float() @ dense.t()
        out = torch.full((m, n + 8), 7.0, device=DEV, dtype=torch.bfloat16)
        K.wq_gemm(x, w, out=out[:, :n])
        assert (out[:, n:] == 7).all()
        assert _close(out[:, :n], K.wq_gemm(x, w, splits=1), k)
        assert ((out[:, :n].float() - ref).norm() / ref.norm()).item() < 6e-3        # rounding of decode arithmetic and result
        got = K.wq_gemm(x, w, residual=res)
        assert _close(got, K.wq_gemm(x, w, residual=res, splits=1), k)
        assert torch.equal(got, K.wq_gemm(x, w, residual=res))                       # parts are summed in their order
    K.workspace(torch.device(DEV, 0)).check_status()
    assert not K.workspace(torch.device(DEV, 0)).gemm_counters.any()


@pytest.mark.parametrize("fmt", ["cubic", "affine", "nvfp4"])
@pytest.mark.parametrize("m,inter,k", [(1, 128, 512), (8, 192, 256), (16, 12288, 512)])
def test_skinny_gemm_gated_epilogue(fmt, m, inter, k):
    from cubic_serve_b200.ops import kernels as K
    w = wq_pack.swiglu_interleave(_weight(fmt, 2 * inter, k, inter))
    x = torch.randn(m, k, device=DEV, generator=torch.Generator(device=DEV).manual_seed(2)).bfloat16()
    plain = wq_pack.PackedWeight(w.fmt, w.n, w.k, w.group_k, w.codes, w.meta, w.alpha)
    gu = torch.empty(m, 2 * inter, device=DEV, dtype=torch.bfloat16)
    gu[:, wq_pack.swiglu_row_order(inter).to(DEV)] = K.wq_gemm(x, plain)
    assert torch.equal(K.wq_gemm_act(x, w), K.swiglu(gu))


@pytest.mark.parametrize("tokens", [1, 5, 40, 90])
@pytest.mark.parametrize("skew", [False, True])
def test_skinny_grouped_gemm(tokens, skew):
    """Few rows an expert; with ``skew`` every token goes to the same eight experts, whose items take several passes."""
    from cubic_serve_b200.models.moe import MoeLayer, stack_experts
    from cubic_serve_b200.ops import kernels as K
    E, H, I = 64, 512, 256
    gu, c0, m0 = stack_experts([_weight("nvfp4", 2 * I, H, e) for e in range(E)])
    dn, c1, m1 = stack_experts([_weight("nvfp4", H, I, 100 + e) for e in range(E)])
    router = torch.randn(E, H, device=DEV, generator=torch.Generator(device=DEV).manual_seed(3)) * 0.1
    x = torch.randn(tokens, H, device=DEV, generator=torch.Generator(device=DEV).manual_seed(4)).bfloat16()
    if skew:
        x[:, 0] = 8.0
        router[:8, 0] += 10.0
    layer = MoeLayer(wq_pack.pack_bf16(router), gu, dn, (c0, m0, c1, m1), E, 8, 0, E, True)
    layer.fuse_activation()
    got = layer.forward(x).clone()
    limit, K.SKINNY_ROWS_PER_EXPERT = K.SKINNY_ROWS_PER_EXPERT, 0
    try:
        want = layer.forward(x)
    finally:
        K.SKINNY_ROWS_PER_EXPERT = limit
    # two chained products: a flipped rounding of an activation moves a result by a part of a bf16 step
    assert ((got.float() - want.float()).norm() / want.float().norm()).item() < 2e-3


@pytest.mark.parametrize("n,k", [(128, 256), (200, 768), (1000, 1280), (9216, 1024)])
def test_skinny_gemm_of_block_scaled_fp8(n, k):
    from cubic_serve_b200.ops import kernels as K
    g = torch.Generator(device=DEV).manual_seed(n)
    w = wq_pack.pack_fp8_block((torch.randn(n, k, device=DEV, generator=g) * 100).clamp_(-448, 448).to(torch.float8_e4m3fn),
                               torch.rand(-(-n // 128), -(-k // 128), device=DEV, generator=g) + 0.5)
    dense = w.codes.view(torch.float8_e4m3fn).double() * w.meta.double().repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)[:, :k]
    for m in (1, 8, 9, 16):
        x, res = torch.randn(m, k, device=DEV, generator=g).bfloat16(), torch.randn(m, n, device=DEV, generator=g).bfloat16()
        a = K.fp8_quantize(x, out=K.Fp8Act(torch.empty(m, k, dtype=torch.uint8, device=DEV), torch.empty(m, device=DEV)))
        ref = (a.q.view(torch.float8_e4m3fn).double() * a.scale.double()[:, None]) @ dense.t()
        out = torch.full((m, n + 8), 7.0, device=DEV, dtype=torch.bfloat16)
        assert K.use_skinny(m, w, a.q)
        K.wq_gemm(a, w, out=out[:, :n])
        assert (out[:, n:] == 7).all()
        assert ((out[:, :n].double() - ref).norm() / ref.norm()).item() < 2.0 ** -9       # one rounding to bf16
        assert _close(out[:, :n], K.wq_gemm(a, w, splits=1), k)
        assert _close(K.wq_gemm(a, w, residual=res), K.wq_gemm(a, w, residual=res, splits=1), k)
    K.workspace(torch.device(DEV, 0)).check_status()
    assert not K.workspace(torch.device(DEV, 0)).gemm_counters.any()


@pytest.mark.parametrize("counts", [[1], [0, 5, 16, 17, 0, 40, 3], [16] * 9])
def test_skinny_grouped_block_scaled_fp8(counts):
    """Experts with no, few and more rows than a pass takes, rows behind the last untouched."""
    from cubic_serve_b200.ops import kernels as K, native
    E, n, k, T = len(counts), 256, 512, sum(counts)
    g = torch.Generator(device=DEV).manual_seed(E)
    codes = (torch.randn(E * n, k, device=DEV, generator=g) * 100).clamp_(-448, 448).to(torch.float8_e4m3fn)
    scale = torch.rand(E * n // 128, k // 128, device=DEV, generator=g) + 0.5
    a = K.fp8_quantize(torch.randn(T, k, device=DEV, generator=g).bfloat16())
    items, at = [], 0
    for e, c in enumerate(counts):
        items += [(e, at, c)] if c else []
        at += c
    tiles = torch.tensor([len(items)] + [v for i in items for v in i], dtype=torch.int32, device=DEV)
    ws = K.workspace(torch.device(DEV, 0))
    dense = codes.double() * scale.double().repeat_interleave(128, 0).repeat_interleave(128, 1)
    x = a.q.view(torch.float8_e4m3fn).double() * a.scale.double()[:, None]
    for rows in (8, 16, 32):
        out = torch.full((T + 4, n), 7.0, device=DEV, dtype=torch.bfloat16)
        native.check(native.lib().cb_wq_gemm_skinny_fp8_grouped(a.q.data_ptr(), k, a.scale.data_ptr(), codes.data_ptr(), scale.data_ptr(), out.data_ptr(), n, T, n, k,
                                                                tiles.data_ptr(), rows, E, ws.status.data_ptr(), K._stream()), "grouped")
        assert (out[T:] == 7).all()
        for e, first, c in items:
            ref = x[first:first + c] @ dense[e * n:(e + 1) * n].t()
            assert ((out[first:first + c].double() - ref).norm() / ref.norm()).item() < 2.0 ** -9
    ws.check_status()


@pytest.mark.parametrize("fmt", ["cubic", "affine", "nvfp4"])
@pytest.mark.parametrize("n,k", [
    (128, 128),            # one tile, one unit
    (200, 1152),           # nine parts of a tile with 72 rows of padding
    (5120, 2048),          # parts of uneven length
    (10000, 1024),         # runs that straddle tiles
    (24576, 512),          # whole tiles between parts
])
def test_gemm_with_decoded_tiles_in_tensor_memory(fmt, n, k):
    from cubic_serve_b200.ops import kernels as K
    w = _weight(fmt, n, k, n + k)
    dense = wq_pack.unpack_to_dense(w)[:n]
    g = torch.Generator(device=DEV).manual_seed(2)
    ws = K.workspace(torch.device(DEV, 0))
    for m in (1, 16, 17, 33, 128):
        wide = torch.randn(m, k + 64, device=DEV, generator=g).bfloat16()
        x, res = wide[:, :k], torch.randn(m, n, device=DEV, generator=g).bfloat16()
        ref = x.float() @ dense.t()
        out = torch.full((m, n + 8), 7.0, device=DEV, dtype=torch.bfloat16)
        K._wq_gemm_skinny(x, w, out[:, :n], None, ws, False, "cb_wq_gemm_ts")
        assert (out[:, n:] == 7).all()
        assert _close(out[:, :n], K.wq_gemm(x, w, splits=1), k)
        assert ((out[:, :n].float() - ref).norm() / ref.norm()).item() < 6e-3        # rounding of decode arithmetic and result
        got = [K._wq_gemm_skinny(x, w, torch.empty(m, n, device=DEV, dtype=torch.bfloat16), res, ws, False, "cb_wq_gemm_ts") for _ in range(2)]
        assert _close(got[0], K.wq_gemm(x, w, residual=res, splits=1), k) and torch.equal(*got)      # parts are summed in their order
        if n % 128 == 0:
            act = wq_pack.swiglu_interleave(w)
            plain = wq_pack.PackedWeight(act.fmt, act.n, act.k, act.group_k, act.codes, act.meta, act.alpha)
            gu = torch.empty(m, n, device=DEV, dtype=torch.bfloat16)
            gu[:, wq_pack.swiglu_row_order(n // 2).to(DEV)] = K._wq_gemm_skinny(x, plain, torch.empty_like(gu), None, ws, False, "cb_wq_gemm_ts")
            assert torch.equal(K._wq_gemm_skinny(x, act, torch.empty(m, n // 2, device=DEV, dtype=torch.bfloat16), None, ws, True, "cb_wq_gemm_ts"), K.swiglu(gu))
    ws.check_status()
    assert not ws.gemm_counters.any()


@pytest.mark.parametrize("n,k", [
    (200, 1152),           # parts of a block's tile of their own, 72 rows of padding
    (3000, 640),           # whole tiles and parts
    (128, 128),            # a unit a tile
])
@pytest.mark.parametrize("fmt", ["cubic", "affine", "nvfp4"])
def test_gemm_with_decoded_tiles_in_tensor_memory_in_blocks_of_rows(fmt, n, k):
    """The smallest second block, blocks of one size and a shorter last one, many blocks."""
    from cubic_serve_b200.ops import kernels as K
    w = _weight(fmt, n, k, n + k)
    g = torch.Generator(device=DEV).manual_seed(3)
    ws = K.workspace(torch.device(DEV, 0))
    for m in (129, 256, 331, 1030):
        x, res = torch.randn(m, k, device=DEV, generator=g).bfloat16(), torch.randn(m, n, device=DEV, generator=g).bfloat16()
        out = torch.full((m + 2, n + 8), 7.0, device=DEV, dtype=torch.bfloat16)
        K._wq_gemm_skinny(x, w, out[:m, :n], None, ws, False, "cb_wq_gemm_ts")
        assert (out[:, n:] == 7).all() and (out[m:] == 7).all()
        assert _close(out[:m, :n], K.wq_gemm(x, w, splits=1), k)
        got = [K._wq_gemm_skinny(x, w, torch.empty(m, n, device=DEV, dtype=torch.bfloat16), res, ws, False, "cb_wq_gemm_ts") for _ in range(2)]
        assert _close(got[0], K.wq_gemm(x, w, residual=res, splits=1), k) and torch.equal(*got)
        if n % 128 == 0:
            act = wq_pack.swiglu_interleave(w)
            plain = wq_pack.PackedWeight(act.fmt, act.n, act.k, act.group_k, act.codes, act.meta, act.alpha)
            gu = torch.empty(m, n, device=DEV, dtype=torch.bfloat16)
            gu[:, wq_pack.swiglu_row_order(n // 2).to(DEV)] = K._wq_gemm_skinny(x, plain, torch.empty_like(gu), None, ws, False, "cb_wq_gemm_ts")
            assert torch.equal(K._wq_gemm_skinny(x, act, torch.empty(m, n // 2, device=DEV, dtype=torch.bfloat16), None, ws, True, "cb_wq_gemm_ts"), K.swiglu(gu))
    ws.check_status()
    assert not ws.gemm_counters.any()


@pytest.mark.parametrize("mb", [16, 48, 128])
@pytest.mark.parametrize("fmt", ["cubic", "affine", "nvfp4"])
def test_grouped_gemm_with_decoded_tiles_in_tensor_memory(fmt, mb):
    """Experts with no, few and many rows (an item full, one row over, several items, a short last tile), fewer and more tiles than SMs."""
    from cubic_serve_b200.models.moe import stack_experts
    from cubic_serve_b200.ops import kernels as K, native
    ws = K.workspace(torch.device(DEV, 0))
    for counts, n, k in (([1], 128, 128), ([0, 5, 16, 17, 0, 129, 3, 300], 320, 640), ([40] * 30, 1280, 256)):
        T, g = sum(counts), torch.Generator(device=DEV).manual_seed(mb)
        each = [_weight(fmt, n, k, e) for e in range(len(counts))]
        w, cs, ms = stack_experts(each)
        x = torch.randn(T, k + 64, device=DEV, generator=g).bfloat16()[:, :k]
        items, at = [], 0
        for e, c in enumerate(counts):
            items += [(e, at + o, min(mb, c - o)) for o in range(0, c, mb)]
            at += c
        tiles = torch.tensor([len(items)] + [v for i in items for v in i], dtype=torch.int32, device=DEV)

        def run(w, out, act):
            native.check(native.lib().cb_wq_gemm_ts_grouped(w.fmt, x.data_ptr(), x.stride(0), w.codes.data_ptr(), K._ptr(w.meta), out.data_ptr(), out.stride(0), w.alpha,
                                                            T, n, k, w.group_k, act, tiles.data_ptr(), len(items) + 2, mb, cs, ms, ws.status.data_ptr(), K._stream()), "grouped")
            return out
        out = run(w, torch.full((T + 4, n + 3), 7.0, device=DEV, dtype=torch.bfloat16), 0)
        assert (out[T:] == 7).all() and (out[:, n:] == 7).all()
        at = 0
        for e, c in enumerate(counts):
            if c:
                assert _close(out[at:at + c, :n], K.wq_gemm(x[at:at + c], each[e], splits=1), k)
            at += c
        if n % 128 == 0:
            act = wq_pack.swiglu_interleave(w, stacked=True)
            gu = torch.empty(T, n, device=DEV, dtype=torch.bfloat16)
            gu[:, wq_pack.swiglu_row_order(n // 2).to(DEV)] = run(act, torch.empty_like(gu), 0)
            assert torch.equal(run(act, torch.empty(T, n // 2, device=DEV, dtype=torch.bfloat16), 1), K.swiglu(gu))
    ws.check_status()


def test_gemm_with_decoded_tiles_in_tensor_memory_refuses_what_it_does_not_take():
    from cubic_serve_b200.ops import kernels as K
    from cubic_serve_b200.ops.native import NativeLibraryError
    ws = K.workspace(torch.device(DEV, 0))
    w = _weight("affine", 128, 128, 0)
    for m, weight in ((0, w), (8, _weight("affine", 128, 192, 0)), (8, _weight("bf16", 128, 128, 0))):
        x = torch.zeros(m, weight.k, device=DEV, dtype=torch.bfloat16)
        assert not K.use_ts(m, weight, x)
        with pytest.raises(NativeLibraryError):
            K._wq_gemm_skinny(x, weight, torch.empty(m, 128, device=DEV, dtype=torch.bfloat16), None, ws, False, "cb_wq_gemm_ts")


def _moe_layer(weight, E, H, I, skew, tokens):
    """A layer of experts with eight routes a token, and rows for it; with ``skew`` every token goes to the same eight experts."""
    from cubic_serve_b200.models.moe import MoeLayer, stack_experts
    gu, c0, m0 = stack_experts([weight(2 * I, H, e) for e in range(E)])
    dn, c1, m1 = stack_experts([weight(H, I, 100 + e) for e in range(E)])
    router = torch.randn(E, H, device=DEV, generator=torch.Generator(device=DEV).manual_seed(3)) * 0.1
    x = torch.randn(tokens, H, device=DEV, generator=torch.Generator(device=DEV).manual_seed(4)).bfloat16()
    if skew:
        x[:, 0] = 8.0
        router[:8, 0] += 10.0
    return MoeLayer(wq_pack.pack_bf16(router), gu, dn, (c0, m0, c1, m1), E, 8, 0, E, True), x


def _same_by_other_kernels(layer, x, monkeypatch, change, entries):
    """``layer.forward(x)`` calls the first of ``entries``, under ``change`` the second, with the same results."""
    from cubic_serve_b200.ops import kernels as K, native
    called, lib = [], native.lib()

    class Spy:
        def __getattr__(self, name):
            if "grouped" in name:
                called.append(name)
            return getattr(lib, name)
    monkeypatch.setattr(K.native, "lib", lambda spy=Spy(): spy)
    got = layer.forward(x).clone()
    change()
    want = layer.forward(x).clone()
    K.workspace(torch.device(DEV, 0)).check_status()
    assert called == [entries[0]] * 2 + [entries[1]] * 2
    # two chained products: a flipped rounding of an activation moves a result by a part of a bf16 step
    assert torch.isfinite(got).all() and ((got.float() - want.float()).norm() / want.float().norm()).item() < 2e-3


@pytest.mark.parametrize("skew", [False, True])
@pytest.mark.parametrize("tokens", [1, 60, 120])
def test_layer_of_block_scaled_experts(tokens, skew, monkeypatch):
    """Few rows an expert on average, with ``skew`` many of eight that take several passes."""
    from cubic_serve_b200.ops import kernels as K
    g = torch.Generator(device=DEV).manual_seed(5)

    def weight(n, k, seed):
        return wq_pack.pack_fp8_block((torch.randn(n, k, device=DEV, generator=g) * 100).clamp_(-448, 448).to(torch.float8_e4m3fn),
                                      (torch.rand(-(-n // 128), -(-k // 128), device=DEV, generator=g) + 0.5) * 2e-4)
    layer, x = _moe_layer(weight, 64, 512, 256, skew, tokens)
    _same_by_other_kernels(layer, x, monkeypatch, lambda: monkeypatch.setattr(K, "SKINNY_ROWS_PER_EXPERT", 0),
                           ("cb_wq_gemm_skinny_fp8_grouped", "cb_wq_gemm_fp8_grouped"))


@pytest.mark.parametrize("skew", [False, True])
@pytest.mark.parametrize("fmt", ["cubic", "nvfp4"])
@pytest.mark.parametrize("tokens", [30, 512, 1100])
def test_layer_of_4_bit_experts_in_tensor_memory(fmt, tokens, skew, monkeypatch):
    """Small work items, and items of 128 rows: the load of an expert is above the least ones."""
    from cubic_serve_b200.ops import kernels as K, strategies
    layer, x = _moe_layer(lambda n, k, seed: _weight(fmt, n, k, seed), 64, 640, 384, skew, tokens)
    old = strategies.active()
    try:
        _same_by_other_kernels(layer, x, monkeypatch, lambda: strategies.install(strategies.operator_config_from_dict({"gemm": {"tensor_memory_rows": 0}})),
                               ("cb_wq_gemm_ts_grouped", "cb_wq_gemm_skinny_grouped" if tokens == 30 and K.skinny_fits(layer.down, x, x) else "cb_wq_gemm_grouped"))
        strategies.install(old)
        layer.forward(x)
        assert layer.scratch.mb == (32 if tokens == 30 else 128)
    finally:
        strategies.install(old)
