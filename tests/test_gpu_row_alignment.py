"""Rows that start anywhere: the kernels that read and write several channels at once give the same bytes as for aligned rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("offset,stride", [(0, 256), (1, 259), (2, 258), (4, 260), (4, 262), (3, 264)])
def test_hadamard_of_views(offset, stride):
    from cubic_serve_b200.ops import kernels as K
    x = torch.randn(7, 256, device=DEV, generator=torch.Generator(device=DEV).manual_seed(stride)).bfloat16()
    want = K.hadamard(x.clone())
    buf = torch.full((offset + 7 * stride,), 5.0, device=DEV, dtype=torch.bfloat16)
    view = buf[offset:].view(7, stride)[:, :256]
    view.copy_(x)
    out = torch.full_like(buf, 5.0)[offset:].view(7, stride)
    assert torch.equal(K.hadamard(view, out=out[:, :256]), want) and (out[:, 256:] == 5).all()
    assert torch.equal(K.hadamard(view[:1]), want[:1]) and torch.equal(view[1:], x[1:])
    assert torch.equal(K.hadamard(view[1:]), want[1:])


@pytest.mark.parametrize("bits", [(8, 8), (6, 4)])
@pytest.mark.parametrize("at_in,at_out", [(1, 0), (0, 1), (2, 2), (4, 4), (3, 5)])
def test_rotary_and_cache_write_of_views(bits, at_in, at_out):
    from cubic_serve_b200.ops import eager, kernels as K
    hq, hkv, d, t = 4, 2, 128, 21
    wide = (hq + 2 * hkv) * d
    g = torch.Generator(device=DEV).manual_seed(8)
    qkv = torch.randn(t, wide, device=DEV, generator=g).bfloat16()
    pos = torch.arange(30, 30 + t, dtype=torch.int32, device=DEV)
    slots = torch.arange(t, dtype=torch.int32, device=DEV)
    inv = eager.rope_inv_freq(d, 1e6, DEV)

    def run(src, dst):
        cache = torch.zeros(2, hkv, K.kv_blob_bytes(d, *bits), dtype=torch.uint8, device=DEV)
        K.rope_kv_write(src, dst, cache, pos, slots, inv, hq, hkv, d, *bits)
        return dst.clone(), cache
    want = run(qkv, torch.empty(t, hq * d, dtype=torch.bfloat16, device=DEV))
    src = torch.empty(at_in + t * wide, dtype=torch.bfloat16, device=DEV)[at_in:].view(t, wide)
    src.copy_(qkv)
    got = run(src, torch.empty(at_out + t * hq * d, dtype=torch.bfloat16, device=DEV)[at_out:].view(t, hq * d))
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
