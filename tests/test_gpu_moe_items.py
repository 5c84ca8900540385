"""Work items of the grouped expert GEMMs that follow a step's load."""
import pytest
import torch

from cubic_serve_b200.ops import kernels as K, wq_pack


@pytest.mark.parametrize("rows,experts,least,want", [(0, 8, 64, 64), (8, 128, 64, 64), (4096, 128, 64, 64), (8192, 128, 64, 96), (16384, 128, 32, 176),
                                                     (32768, 128, 64, 160), (65536, 128, 64, 208), (10 ** 6, 8, 64, 256)])
def test_rows_of_a_work_item(rows, experts, least, want):
    mb = K.rows_per_work_item(rows, experts, least)
    assert mb == want and mb % 16 == 0 and least <= mb <= 256


@pytest.mark.gpu
@pytest.mark.parametrize("tokens", [130, 301, 700])
def test_layer_with_large_work_items(tokens):
    from cubic_serve_b200.models.moe import MoeLayer, stack_experts
    E, H, I = 8, 256, 128
    g = torch.Generator(device="cuda").manual_seed(tokens)
    rand = lambda *s: torch.rand(*s, device="cuda", generator=g)  # noqa: E731

    def nv(n, k):
        q = torch.randint(0, 256, (n, k // 2), device="cuda", generator=g, dtype=torch.uint8)
        return wq_pack.pack_nvfp4(q, (rand(n, k // 16) * 8).to(torch.float8_e4m3fn), 0.01)
    gu, c0, m0 = stack_experts([nv(2 * I, H) for _ in range(E)])
    dn, c1, m1 = stack_experts([nv(H, I) for _ in range(E)])
    router = wq_pack.pack_bf16(rand(E, H) - 0.5)
    x = (rand(tokens, H) - 0.5).bfloat16()
    layer = MoeLayer(router, gu, dn, (c0, m0, c1, m1), E, 2, 0, E, True)
    layer.fuse_activation()
    got = layer.forward(x).clone()
    sc = layer.scratch
    counts = sc.counts.long()
    n = int(sc.tiles[0])
    assert n == int(((counts + sc.mb - 1) // sc.mb).sum()) <= sc.items(2 * tokens)
    rule, K.rows_per_work_item = K.rows_per_work_item, lambda *_: 64
    try:
        want = layer.forward(x)
    finally:
        K.rows_per_work_item = rule
    assert sc.mb == 64 and torch.equal(got, want)        # the rows of an item do not meet: the same sums
