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
