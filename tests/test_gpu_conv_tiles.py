"""The convolution of Gated DeltaNet layers cut into tiles of rows, against the oracle one request at a time."""
import pytest
import torch

from cubic_serve_b200.ops import eager

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("lengths", [[1], [2, 3], [31, 32, 33], [1, 64, 65, 100, 2]])
@pytest.mark.parametrize("channels,wide", [(256, 256), (384, 400), (131, 131)])        # even and odd row strides, a ragged last block
@pytest.mark.parametrize("commit", [True, False])
def test_conv_tiles(lengths, channels, wide, commit):
    from cubic_serve_b200.ops import kernels as K
    g = torch.Generator().manual_seed(sum(lengths) + channels)
    T, n = sum(lengths), len(lengths)
    x = torch.randn(T, wide, generator=g).bfloat16()
    w = torch.randn(channels, 4, generator=g) * 0.5
    state = torch.randn(n + 2, 3, channels, generator=g).bfloat16()
    slots, pos0 = torch.randperm(n + 2, generator=g)[:n], [0 if i % 3 == 1 else 40 for i in range(n)]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    row0 = [sum(lengths[:i]) for i in range(n)]
    seg = K.GdnSegments(i32(row0), i32(lengths), i32(slots.tolist()), i32(pos0), n)
    out = torch.zeros(T, channels, dtype=torch.bfloat16, device=DEV)
    got_state = state.to(DEV)
    K.gdn_conv(x.to(DEV), w.to(DEV), got_state, seg, out, commit=commit)
    want_state = state.clone()
    for i, m in enumerate(lengths):
        rows = slice(row0[i], row0[i] + m)
        y, st = eager.gdn_conv(x[rows, :channels], w, state[slots[i]] if pos0[i] else None)
        # fp32 sums of four products in both, the exponential of the activation approximated: a step of bf16, or of the small values' scale
        assert ((out[rows].cpu().float() - y.float()).abs() <= 2.0 ** -7 * y.float().abs() + 2.0 ** -14).all()
        if commit:
            want_state[slots[i]] = st
    assert torch.equal(got_state.cpu(), want_state)


@pytest.mark.parametrize("channels,longest", [(4096, 20000), (131, 100000)])
def test_conv_over_its_input(channels, longest):
    """``out`` is ``x``: rows that later tiles look back at have been overwritten when there are more tiles than the GPU runs at once."""
    from cubic_serve_b200.ops import kernels as K
    g = torch.Generator(device=DEV).manual_seed(channels)
    lengths = [longest, 1, 300, 90]
    T, n = sum(lengths), len(lengths)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    seg = K.GdnSegments(i32([sum(lengths[:i]) for i in range(n)]), i32(lengths), i32([2, 0, 3, 1]), i32([0, 7, 0, 9]), n)
    wide = torch.randn(T, 2 * channels, device=DEV, generator=g).bfloat16()
    w = torch.randn(channels, 4, device=DEV, generator=g) * 0.5
    state = torch.randn(n, 3, channels, device=DEV, generator=g).bfloat16()
    x = wide[:, :channels]
    want, want_state = torch.empty(T, channels, dtype=torch.bfloat16, device=DEV), state.clone()
    K.gdn_conv(x, w, want_state, seg, want)
    beside, beside_state = wide.clone(), state.clone()           # neighbouring columns of one buffer share no element
    K.gdn_conv(beside[:, :channels], w, beside_state, seg, beside[:, channels:])
    assert torch.equal(beside[:, channels:], want) and torch.equal(beside[:, :channels], x) and torch.equal(beside_state, want_state)
    K.gdn_conv(x, w, state, seg, x)
    assert torch.equal(x, want) and torch.equal(state, want_state)
