"""Single tokens with the attention options on the warp-level tensor cores, against the general kernel on the same numbers in
float32 (which the designs' own tests compare with plain implementations)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

CASES = [   # heads, key heads, head size, page, longest, options
    (16, 4, 128, 16, 1500, dict(window=1024, keep_first=8, softcap=40.0, sink=True)),
    (16, 4, 128, 16, 700, dict(window=300, keep_first=33, softcap=30.0, sink="learned", dist=True)),
    (16, 4, 64, 16, 1025, dict(chunk=256, sigmoid=True)),
    (16, 4, 128, 8, 257, dict(chunk=256, sigmoid=True)),
    (3, 3, 64, 32, 97, dict(sigmoid=True, softcap=5.0)),
    (16, 1, 128, 16, 1100, dict(window=1024, sink="learned", latent=True)),
    (24, 1, 64, 16, 300, dict(window=100, sink="learned", latent=True)),
    (20, 1, 64, 8, 260, dict(softcap=10.0)),
    (16, 4, 128, 16, 640, dict(v_share=2)),
    (6, 6, 64, 16, 130, dict(v_share=3, dist=True)),
    (1, 1, 64, 1, 40, dict(window=1, keep_first=3, sink=True)),
    (8, 2, 64, 64, 2500, dict(window=31, keep_first=64, sink=True)),
    (4, 2, 128, 16, 33, dict(chunk=32)),
]


@pytest.mark.parametrize("splits,parts", [(None, 1), (1, 1), (2, 2), (6, 1), (11, 1)])
@pytest.mark.parametrize("case", CASES)
def test_single_tokens_with_options_match_the_general_kernel_in_float32(case, splits, parts):
    from llm_b200.csrc import ops
    H, G, D, page, longest, o = case
    if parts > 1 and not o.get("latent"):
        parts = 1
    g = torch.Generator(device=DEV).manual_seed(longest + H)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    share, w = o.get("v_share", 1), o.get("window", 0)
    lens = [longest, 1, 2, 31, 32, 33, max(1, longest // 2), w + o.get("keep_first", 0) + 1, max(1, o.get("chunk", 1) - 1), o.get("chunk", 1) + 1]
    lens = [min(n, longest) for n in lens]
    B = len(lens)
    width = -(-longest // page) + 1
    pages = sum(-(-n // page) for n in lens) + 2
    order = torch.randperm(pages, generator=torch.Generator().manual_seed(1)).tolist()
    table = torch.zeros(B, width, dtype=torch.int32)
    for b, n in enumerate(lens):
        k = -(-n // page)
        table[b, :k] = torch.tensor([order.pop() for _ in range(k)], dtype=torch.int32)
    table = table.to(DEV)
    kp = rand(pages, G, page, D).bfloat16()
    vp = kp if o.get("latent") else rand(pages, G // share, page, D).bfloat16()
    q = (rand(B, H * D + 8) * 1.5).bfloat16()
    kv_lens = torch.tensor(lens, dtype=torch.int32, device=DEV)
    kw = dict(softcap=o.get("softcap", 0.0), sink=bool(o.get("sink")), keep_first=o.get("keep_first", 0), v_share=share, chunk=o.get("chunk", 0),
              sink_values=rand(H) * 2 if o.get("sink") == "learned" else None, sigmoid_bias=rand(H) - 3 if o.get("sigmoid") else None,
              dist_bias=(rand(H).abs(), rand(H).abs()) if o.get("dist") else None)
    scale = 1.0 / math.sqrt(D)
    out = torch.full((B, H * D), float("nan"), device=DEV, dtype=torch.bfloat16)
    ops.paged_attention_decode(out, q, kp, vp, table, kv_lens, B, H, G, D, w, scale, splits=splits, head_parts=parts, **kw)
    ref = torch.zeros(B, H * D, device=DEV)
    kf = kp.float()
    ops.paged_attention_generic(ref, q.float(), kf, kf if o.get("latent") else vp.float(), table, torch.arange(B, dtype=torch.int32, device=DEV),
                                kv_lens - 1, B, H, G, D, w, scale, **kw)
    # the scores and weights are float32 sums in another order, P keeps 16 bits and more: what is left is the rounding of the
    # output to bfloat16, 2^-9 of a value; the error is that of the rounded reference but for values that round the other way
    norm = ref.double().norm()
    err, floor = (out.double() - ref.double()).norm() / norm, (ref.bfloat16().double() - ref.double()).norm() / norm
    assert err <= 1.05 * floor + 2e-6, (float(err), float(floor))
    assert ((out.float() - ref).abs() <= ref.abs() * 2 ** -8 + 2e-5).all()


def test_chunks_and_sigmoid_weights_are_refused_where_only_the_cuda_core_kernel_runs():
    from llm_b200.csrc import ops
    q, kp = torch.zeros(1, 96, device=DEV, dtype=torch.bfloat16), torch.zeros(2, 1, 16, 96, device=DEV, dtype=torch.bfloat16)
    with pytest.raises(ops.KernelError):
        ops.paged_attention_decode(torch.zeros_like(q), q, kp, kp, torch.zeros(1, 1, dtype=torch.int32, device=DEV),
                                   torch.ones(1, dtype=torch.int32, device=DEV), 1, 1, 1, 96, 0, 0.1, chunk=4)


@pytest.mark.parametrize("sigmoid", [False, True])
def test_more_single_tokens_than_arrival_counters(sigmoid):
    """512 requests of 16 key heads are 8,192 pairs, twice the counters: chunks and sigmoid weights take the general kernel then."""
    import types

    from llm_b200.csrc import ops
    B, G, D, page, chunk = 512, 16, 64, 16, 24
    g = torch.Generator(device=DEV).manual_seed(2)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    lens = torch.randint(1, 3 * page, (B,), device=DEV, dtype=torch.int32, generator=g)
    table = torch.arange(3 * B, dtype=torch.int32, device=DEV).view(B, 3)
    kp, vp, q = rand(3 * B, G, page, D).bfloat16(), rand(3 * B, G, page, D).bfloat16(), rand(B, G * D).bfloat16()
    kw = dict(chunk=chunk, sigmoid_bias=rand(G) - 1 if sigmoid else None)
    ctx = types.SimpleNamespace(decode_only=True, kv_bucket=3 * page, n_entries=B, n_tokens=B, kv_lens=lens, positions=lens - 1,
                                token_entry=torch.arange(B, dtype=torch.int32, device=DEV))
    out = torch.full((B, G * D), float("nan"), device=DEV, dtype=torch.bfloat16)
    ops.paged_attention(out, q, kp, vp, types.SimpleNamespace(block_table=table), ctx, G, G, D, 0, 0.125, **kw)
    ref = torch.zeros(B, G * D, device=DEV)
    ops.paged_attention_generic(ref, q.float(), kp.float(), vp.float(), table, ctx.token_entry, ctx.positions, B, G, G, D, 0, 0.125, **kw)
    # float32 sums of at most 24 terms of size one, then the output's rounding
    assert ((out.float() - ref).abs() <= ref.abs() * 2 ** -8 + 2e-5).all()


def exact(q, kp, vp, table, lens, H, G, D, window, scale, o):
    """The attention of single tokens in 64 bits."""
    ref = torch.zeros(len(lens), H, D, dtype=torch.float64, device=DEV)
    column = lambda t: t.double()[:, None]
    for b, n in enumerate(lens):
        at = table[b].long()
        K, V = ([t[at].permute(1, 0, 2, 3).flatten(1, 2)[:, :n].double().repeat_interleave(H // t.shape[1], 0) for t in (kp, vp)])
        s, away = (q[b].view(H, 1, D).double() * K).sum(-1) * scale, n - 1 - torch.arange(n, device=DEV)
        seen = (away < window) | (torch.arange(n, device=DEV) < o["keep_first"]) if window else away >= 0
        if o["chunk"]:
            seen = torch.arange(n, device=DEV) // o["chunk"] == (n - 1) // o["chunk"]
        if o["softcap"]:
            s = o["softcap"] * torch.tanh(s / o["softcap"])
        if o["dist_bias"]:
            s = s - column(o["dist_bias"][0]) * torch.log1p(column(o["dist_bias"][1]) * away.double())
        if o["sigmoid_bias"] is not None:
            p = torch.sigmoid(s + column(o["sigmoid_bias"])) * seen
        else:
            sink = s[:, :0] if not o["sink"] else torch.zeros_like(s[:, :1]) if o["sink_values"] is None else column(o["sink_values"])
            p = torch.softmax(torch.cat([s.masked_fill(~seen, -math.inf), sink], 1), -1)[:, :n]
        ref[b] = torch.einsum("hk,hkd->hd", p, V)
    return ref.flatten(1)


@pytest.mark.parametrize("case", [(16, 4, 128, dict(window=1024, softcap=40.0, sink=True, keep_first=8)), (16, 4, 128, dict(softcap=8.0)),
                                  (16, 4, 128, dict(softcap=500.0)), (20, 4, 128, dict(softcap=30.0, dist=True, v_share=2)), (16, 4, 64, dict(dist=True)),
                                  (16, 4, 64, dict(chunk=256, sigmoid=True)), (16, 4, 128, dict(sigmoid=True)), (16, 1, 128, dict(window=1024, sink="learned"))])
def test_scores_and_weights_keep_the_precision_of_float32(case):
    """How many outputs are not the exact value rounded once to bfloat16: no more than twice as many (and a dozen) as those of the general
    kernel, whose scores, weights and sums are float32 numbers.  Weights of sixteen bits, or functions with an absolute error under a large cap,
    give several times as many (five to fifty)."""
    from llm_b200.csrc import ops
    H, G, D, o = case
    g = torch.Generator(device=DEV).manual_seed(H + D)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    lens, page, share, w = [1900, 1500, 1024, 700, 1, 33] * 4, 16, o.get("v_share", 1), o.get("window", 0)
    B, width = len(lens), -(-max(lens) // page)
    kp, vp = rand(B * width, G, page, D).bfloat16(), rand(B * width, G // share, page, D).bfloat16()
    table = torch.randperm(B * width, device=DEV, generator=g).to(torch.int32).view(B, width)
    q, kv_lens = (rand(B, H * D) * 1.5).bfloat16(), torch.tensor(lens, dtype=torch.int32, device=DEV)
    kw = dict(softcap=o.get("softcap", 0.0), sink=bool(o.get("sink")), keep_first=o.get("keep_first", 0), v_share=share, chunk=o.get("chunk", 0),
              sink_values=rand(H) * 2 if o.get("sink") == "learned" else None, sigmoid_bias=rand(H) - 3 if o.get("sigmoid") else None,
              dist_bias=(rand(H).abs(), rand(H).abs()) if o.get("dist") else None)
    best = exact(q, kp, vp, table, lens, H, G, D, w, D ** -0.5, kw).bfloat16()
    out, general = torch.zeros_like(q), torch.zeros_like(q)
    ops.paged_attention_decode(out, q, kp, vp, table, kv_lens, B, H, G, D, w, D ** -0.5, splits=6, **kw)
    ops.paged_attention_generic(general, q, kp, vp, table, torch.arange(B, dtype=torch.int32, device=DEV), kv_lens - 1, B, H, G, D, w, D ** -0.5, **kw)
    off = lambda t: int((t != best).sum())
    assert off(out) <= 2 * off(general) + 12, (off(out), off(general), best.numel())
