"""Long contexts whose ranges are handed out by the requests' lengths: a document beside short requests, equal lengths, single keys,
windows, chunks, latents, and the kernel that rotates and stores too, against the general kernel on the same numbers in float32."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def pages_of(lens, page, width):
    """A table of `width` pages an entry, in shuffled order, and the number of pages."""
    pages = sum(-(-n // page) for n in lens) + 1
    order = torch.randperm(pages, generator=torch.Generator().manual_seed(1)).tolist()
    table = torch.zeros(len(lens), width, dtype=torch.int32)
    for b, n in enumerate(lens):
        k = -(-n // page)
        table[b, :k] = torch.tensor([order.pop() for _ in range(k)], dtype=torch.int32)
    return table.to(DEV), pages


@pytest.mark.parametrize("lens", [[6000, 400, 1, 33, 700], [5000] * 3, [1, 1, 4100], [2049], [31, 32, 64, 65, 9000, 127, 128, 1, 2, 3]])
@pytest.mark.parametrize("H,G,D,window,options", [(8, 2, 128, 0, False), (4, 4, 64, 0, False), (8, 1, 64, 1500, False), (8, 2, 128, 1024, True)])
def test_ranges_by_length_match_the_general_kernel_in_float32(lens, H, G, D, window, options):
    from llm_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(sum(lens) + D)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    page, B, longest = 16, len(lens), 8192 + 2048
    table, pages = pages_of(lens, page, -(-longest // page))
    kp, vp, q = rand(pages, G, page, D).bfloat16(), rand(pages, G, page, D).bfloat16(), rand(B, H * D).bfloat16()
    kv_lens = torch.tensor(lens, dtype=torch.int32, device=DEV)
    kw = dict(softcap=30.0, sink=True, keep_first=5) if options else {}
    scale = 1.0 / math.sqrt(D)
    def exact(values):
        ref = torch.zeros(B, H * D, device=DEV)
        ops.paged_attention_generic(ref, q.float(), kp.float(), values, table, torch.arange(B, dtype=torch.int32, device=DEV), kv_lens - 1,
                                    B, H, G, D, window, scale, **kw)
        return ref
    ref = exact(vp.float())
    # the output's rounding to bfloat16 is 2^-9 of a value; with options the weights keep 16 bits and more, without they too are rounded
    # to bfloat16, which moves a sum by at most 2^-9 of the sum of its terms' sizes (twice both, for what else rounds)
    bound = ref.abs() * 2 ** -8 + 2e-5 + (0 if options else exact(vp.float().abs()) * 2 ** -8)
    for splits in (1, 3, ops.decode_places(B, G, longest), 64):
        out = torch.full((B, H * D), float("nan"), device=DEV, dtype=torch.bfloat16)
        ops.paged_attention_decode(out, q, kp, vp, table, kv_lens, B, H, G, D, window, scale, splits=splits, max_keys=longest, **kw)
        assert ((out.float() - ref).abs() <= bound).all(), splits


@pytest.mark.parametrize("lens", [[9000, 5000, 8191, 8192, 8193, 1, 4097], [12000 + 300 * i for i in range(8)]])
@pytest.mark.parametrize("G,D,chunk", [(2, 128, 4096), (4, 64, 3000)])
def test_ranges_of_chunks_match_the_general_kernel_in_float32(lens, G, D, chunk):
    """A chunk of more than 2,048 keys: an entry's ranges are those of the keys that it sees, not of its whole length."""
    from llm_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(sum(lens) + D)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    H, page, B = 2 * G, 16, len(lens)
    table, pages = pages_of(lens, page, -(-max(lens) // page))
    kp, vp, q = rand(pages, G, page, D).bfloat16(), rand(pages, G, page, D).bfloat16(), rand(B, H * D).bfloat16()
    kv_lens = torch.tensor(lens, dtype=torch.int32, device=DEV)
    kw = dict(chunk=chunk, sigmoid_bias=rand(H) - 3)
    ref = torch.zeros(B, H * D, device=DEV)
    ops.paged_attention_generic(ref, q.float(), kp.float(), vp.float(), table, torch.arange(B, dtype=torch.int32, device=DEV), kv_lens - 1,
                                B, H, G, D, 0, D ** -0.5, **kw)
    for splits in (1, ops.decode_places(B, G, chunk), 64):
        out = torch.full((B, H * D), float("nan"), device=DEV, dtype=torch.bfloat16)
        ops.paged_attention_decode(out, q, kp, vp, table, kv_lens, B, H, G, D, 0, D ** -0.5, splits=splits, max_keys=chunk, **kw)
        # weights in float32 and up to 4,096 terms of size one: the output's rounding, and float32 sums in another order
        assert ((out.float() - ref).abs() <= ref.abs() * 2 ** -8 + 1e-4).all(), splits


@pytest.mark.parametrize("lens", [[6000, 400, 1, 33, 700], [5000] * 3, [300, 9000]])
@pytest.mark.parametrize("H,G,D,latent", [(8, 2, 128, False), (8, 4, 64, False), (16, 1, 128, True)])
def test_other_routes_by_length_match_the_planned_ranges(lens, H, G, D, latent):
    """The kernel that rotates and stores (which a Llama decode step runs), and latents with their heads over several CTAs, with ranges by
    length beside one range a request, which no length changes."""
    from llm_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(sum(lens) + D)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    page, B, longest = 16, len(lens), 10240
    table, pages = pages_of(lens, page, longest // page)
    kp = rand(pages, G, page, D).bfloat16()
    vp = kp if latent else rand(pages, G, page, D).bfloat16()
    kv_lens = torch.tensor(lens, dtype=torch.int32, device=DEV)
    q = rand(B, (H if latent else H + 2 * G) * D).bfloat16()
    angle = rand(longest, D // 2)

    def run(splits, max_keys, parts=1):
        out, k, v = torch.full((B, H * D), float("nan"), device=DEV, dtype=torch.bfloat16), kp.clone(), vp.clone()
        if latent:
            ops.paged_attention_decode(out, q, kp, kp, table, kv_lens, B, H, G, D, 0, D ** -0.5, splits=splits, max_keys=max_keys, head_parts=parts)
        else:
            ops.decode_attention_fused(out, q, angle.cos(), angle.sin(), k, v, table, kv_lens, B, H, G, D, 0, D ** -0.5, splits=splits,
                                       max_keys=max_keys)
        return out, k, v
    want, k1, v1 = run(1, 0)
    for splits, parts in ((1, 1), (5, 2), (ops.decode_places(B, G, longest), 4), (64, 1)):
        got, k2, v2 = run(splits, longest, parts)
        assert torch.equal(k1, k2) and torch.equal(v1, v2)
        # weights rounded to bfloat16 below another maximum, and the output's rounding: 2^-8 of values up to a few units
        assert float((got.float() - want.float()).abs().max()) <= 2 ** -6 * float(want.float().abs().max()), splits
