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


def attend(q, k, v, seen, scale, sink=None, gate=None):
    """One query a row in 64 bits: q [t, h, d], k [j, d], v [j, e], seen [t, j]; sink: score per head without a value; gate: sigmoid weights."""
    s = torch.einsum("thd,jd->htj", q, k) * scale
    s = s.masked_fill(~seen, -math.inf)
    if gate is not None:
        p = torch.sigmoid(s + gate[:, None, None])
    else:
        p = torch.softmax(s if sink is None else torch.cat([s, sink[:, None, None].expand(-1, s.shape[1], 1)], -1), -1)[..., :k.shape[0]]
    return torch.einsum("htj,je->the", p, torch.where(seen.any(0)[:, None], v, 0.0)).flatten(1)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("HS", [32, 64, 128])
@pytest.mark.parametrize("n,option", [(33, ""), (161, ""), (161, "sink"), (161, "learned"), (161, "keep"), (300, "keep"), (161, "chunk"), (300, "chunk"),
                                      (161, "sigmoid"), (300, "sigmoid")])
@pytest.mark.parametrize("lowest", ["none", "last key", "a tile", "first tile"])
def test_general_attention_with_options_and_scores_of_minus_infinity(ops, dtype, HS, n, option, lowest):
    """Up to 64 channels four warps take a head's tiles of 32 keys in turn: options that leave tiles out, and keys whose product with the query is
    -inf, which weigh nothing wherever they lie (in tiles that hold no other, too); in every form the weights' sums are over what is left."""
    if lowest == "first tile" and option in ("chunk", "sigmoid"):
        pytest.skip("the last queries see no key of it")
    page, NH = 8, 3
    g = torch.Generator(device=DEV).manual_seed(HS + n)
    rand = lambda *s: torch.randn(*s, generator=g, device=DEV)
    pages = -(-n // page)
    kp, vp = (rand(pages, 1, page, HS).to(dtype) for _ in range(2))
    q = rand(n, NH * HS).abs().to(dtype)
    rows = {"none": [], "last key": [n - 1], "a tile": list(range(64, 96)) if n > 96 else [32], "first tile": list(range(32))}[lowest]
    for j in rows:
        kp[j // page, 0, j % page, 5] = -math.inf
    i = torch.arange(n, device=DEV)
    dist = i[:, None] - i[None]
    seen = dist >= 0
    kw, window, sink, gate = {}, 0, None, None
    if option == "sink":
        kw, sink = dict(sink=True), torch.zeros(NH, device=DEV).double()
    if option == "learned":
        kw = dict(sink=True, sink_values=rand(NH) * 2)
        sink = kw["sink_values"].double()
    if option == "keep":
        window, kw = 40, dict(keep_first=6)
        seen = seen & ((dist < 40) | (i[None] < 6))
    if option in ("chunk", "sigmoid"):
        kw = dict(chunk=150)
        seen = seen & (i[:, None] // 150 == i[None] // 150)
    if option == "sigmoid":
        kw["sigmoid_bias"] = rand(NH) - 2
        gate = kw["sigmoid_bias"].double()
    k, v = (p.reshape(-1, HS)[:n].double() for p in (kp, vp))
    k = torch.where(torch.isinf(k), 0.0, k)
    low = torch.zeros(n, dtype=torch.bool, device=DEV)
    low[rows] = True
    seen = seen & ~low[None]
    some = seen.any(1) | (option in ("sink", "learned", "sigmoid"))      # the other queries see scores of -inf alone
    ref = attend(q.double().view(n, NH, HS), k, v, seen, HS ** -0.5, sink, gate)
    out = torch.empty(n, NH * HS, device=DEV, dtype=dtype)
    ops.paged_attention_generic(out, q, kp, vp, torch.arange(pages, dtype=torch.int32, device=DEV)[None].contiguous(),
                                torch.zeros(n, dtype=torch.int32, device=DEV), i.to(torch.int32), n, NH, 1, HS, window, HS ** -0.5, **kw)
    # float32 sums of n weights and HS products; bfloat16 results are rounded once more
    assert float((out.double() - ref)[some].norm() / ref[some].norm()) < (2e-6 if dtype == torch.float32 else 2.0 ** -8)


@pytest.mark.parametrize("HS", [32, 64, 128])
def test_infinite_values_of_keys_that_weigh_nothing(ops, HS):
    """A key 400 below the largest score has the weight exp(-400) = 0 in float32, and its value counts nothing, whichever tile it lies in."""
    n, page = 161, 8
    q = torch.zeros(1, HS, device=DEV)
    q[0, 0] = 1.0
    kp = torch.zeros(-(-n // page), 1, page, HS, device=DEV)
    vp = torch.randn_like(kp)
    for j in (40, 160):
        kp[j // page, 0, j % page, 0] = -400.0
        vp[j // page, 0, j % page, 3] = math.inf
    # a tile of such keys alone, and no other for its warp
    for j in range(96, 128):
        kp[j // page, 0, j % page, 0], vp[j // page, 0, j % page, 7] = -400.0, math.inf
    v = vp.reshape(-1, HS)[:n].double()
    keep = [j for j in range(n) if j not in (40, 160) and not 96 <= j < 128]
    out = torch.empty(1, HS, device=DEV)
    ops.paged_attention_generic(out, q, kp, vp, torch.arange(kp.shape[0], dtype=torch.int32, device=DEV)[None].contiguous(),
                                torch.zeros(1, dtype=torch.int32, device=DEV), torch.tensor([n - 1], dtype=torch.int32, device=DEV), 1, 1, 1, HS, 0, 1.0)
    ref = v[keep].mean(0)
    assert float((out[0].double() - ref).norm() / ref.norm()) < 2e-6


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("HS", [20, 32, 64])
@pytest.mark.parametrize("window,kw", [(0, {}), (0, dict(sink=True)), (40, dict(keep_first=6)), (0, dict(chunk=150))])
def test_general_attention_has_the_same_bits_in_launches_of_few_and_many(ops, dtype, HS, window, kw):
    """Four warps to a head in a launch of few pairs, one warp to a head in a launch of many: the sums are the same ones in the same order."""
    page, NH, n = 8, 3, 300
    g = torch.Generator(device=DEV).manual_seed(HS)
    rand = lambda *s: torch.randn(*s, generator=g, device=DEV).to(dtype)
    kp, vp, q = rand(-(-n // page), 1, page, HS), rand(-(-n // page), 1, page, HS), rand(n, NH * HS)
    table = torch.arange(kp.shape[0], dtype=torch.int32, device=DEV)[None].contiguous()

    def run(rows, pos):
        out = torch.empty(rows.shape[0], NH * HS, device=DEV, dtype=dtype)
        ops.paged_attention_generic(out, rows.contiguous(), kp, vp, table, torch.zeros(len(pos), dtype=torch.int32, device=DEV), pos, len(pos), NH, 1, HS,
                                    window, HS ** -0.5, **kw)
        return out

    at = torch.tensor([0, 31, 32, 63, 64, 95, 96, 127, 128, 299], dtype=torch.int32, device=DEV)
    few = run(q[at.long()], at)
    times = 40 * ops.sm_count() // (n * NH) + 1                          # 40 pairs an SM
    many = run(q.repeat(times, 1), torch.arange(n, dtype=torch.int32, device=DEV).repeat(times)).view(times, n, -1)
    assert bool((many == many[:1]).all()) and torch.equal(few, many[0][at.long()])
