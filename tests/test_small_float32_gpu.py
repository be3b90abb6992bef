"""What a small float32 model runs on: the product's small tiles and the general attention at the head sizes where its build changes."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from llm_b200.csrc import ops
    return ops


@pytest.mark.parametrize("K", [4, 96, 128, 132, 256, 388, 1000])
@pytest.mark.parametrize("M,N", [(1, 1), (15, 33), (17, 96), (64, 384)])
def test_small_tiles_have_the_bits_of_the_large_ones(ops, M, N, K):
    """A product of few tiles and the same rows inside one of many tiles: one chain of multiply-adds over k in both."""
    g = torch.Generator(device=DEV).manual_seed(K + M)
    a, w = torch.randn(10000, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV)
    small = torch.full((M + 1, N + 2), 7.0, device=DEV)
    ops.gemm_simt(a, w, small[:, :N], M)
    large = torch.empty(10000, N, device=DEV)
    ops.gemm_simt(a, w, large, 10000)                                  # 157 rows of tiles: the large ones
    assert torch.equal(small[:M, :N], large[:M])
    assert bool((small[M] == 7).all()) and bool((small[:, N:] == 7).all())


@pytest.mark.parametrize("HS", [32, 64, 72, 128, 136, 264])
@pytest.mark.parametrize("n,window", [(1, 0), (32, 0), (33, 0), (161, 0), (161, 40)])
def test_general_attention_over_head_sizes(ops, HS, n, window):
    page, NH, NKV = 8, 3, 1
    g = torch.Generator(device=DEV).manual_seed(HS + n)
    pages = -(-n // page)
    kp, vp = (torch.randn(pages + 2, NKV, page, HS, generator=g, device=DEV) for _ in range(2))
    bt = torch.randperm(pages + 2, generator=torch.Generator().manual_seed(n))[:pages].to(torch.int32)[None].contiguous()
    q = torch.randn(n, NH * HS, generator=g, device=DEV)
    k, v = (p[bt[0].long().to(DEV)].permute(1, 0, 2, 3).reshape(NKV, -1, HS)[0, :n].double() for p in (kp, vp))
    i = torch.arange(n, device=DEV)
    dist = i[:, None] - i[None]
    seen = (dist >= 0) & ((dist < window) if window else torch.ones_like(dist, dtype=torch.bool))
    s = torch.einsum("thd,jd->htj", q.view(n, NH, HS).double(), k) / math.sqrt(HS)
    ref = torch.einsum("htj,jd->thd", torch.softmax(s.masked_fill(~seen, -math.inf), -1), v).reshape(n, NH * HS)
    out = torch.empty(n, NH * HS, device=DEV)
    ops.paged_attention_generic(out, q, kp, vp, bt.to(DEV), torch.zeros(n, dtype=torch.int32, device=DEV), i.to(torch.int32), n, NH, NKV, HS,
                                window, 1.0 / math.sqrt(HS))
    # float32 sums of n weights and HS products
    assert float((out.double() - ref).norm() / ref.norm()) < 2e-6
    if window:                                     # a page that has gone back keeps no number
        last = torch.empty(1, NH * HS, device=DEV)
        bt[0, :max(0, (n - window)) // page] = -1
        ops.paged_attention_generic(last, q[-1:], kp, vp, bt.to(DEV), torch.zeros(1, dtype=torch.int32, device=DEV),
                                    i[-1:].to(torch.int32).contiguous(), 1, NH, NKV, HS, window, 1.0 / math.sqrt(HS))
        assert torch.equal(last[0], out[-1])
