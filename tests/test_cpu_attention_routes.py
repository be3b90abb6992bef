"""Which kernels the parts of a decode step are sent to, on the CPU (attention with the kernels' entry points replaced)."""
import types

import pytest
import torch


@pytest.mark.parametrize("entries,options,want", [
    (256, dict(chunk=32), "decode"), (257, dict(chunk=32), "general"), (512, dict(sigmoid=True), "general"), (4, dict(sigmoid=True, chunk=8), "decode"),
    (4, dict(chunk=32, page=24), "general"), (4, dict(chunk=32, dtype=torch.float32), "general"), (257, dict(softcap=3.0), "decode")])
def test_chunks_and_sigmoid_weights_beyond_the_counters_take_the_general_kernel(entries, options, want, monkeypatch):
    """16 key heads: 256 requests are as many (request, key head) pairs as the decode kernel has arrival counters."""
    from llm_b200.csrc import ops
    sent = []
    monkeypatch.setattr(ops, "sm_count", lambda: 148)
    monkeypatch.setattr(ops, "paged_attention_decode", lambda *a, **k: sent.append("decode"))
    monkeypatch.setattr(ops, "paged_attention_generic", lambda *a, **k: sent.append("general"))
    o = dict(options)
    page, dtype, G, D = o.pop("page", 16), o.pop("dtype", torch.bfloat16), 16, 64
    if o.pop("sigmoid", False):
        o["sigmoid_bias"] = torch.zeros(G)
    pages = torch.zeros(1, G, page, D, dtype=dtype)
    ctx = types.SimpleNamespace(decode_only=True, kv_bucket=64, n_entries=entries, n_tokens=entries, kv_lens=None, positions=None, token_entry=None)
    q = torch.zeros(entries, G * D, dtype=dtype)
    group = types.SimpleNamespace(block_table=torch.zeros(entries, 4, dtype=torch.int32))
    ops.paged_attention(q, q, pages, pages, group, ctx, G, G, D, 0, 0.1, **o)
    assert sent == [want]


@pytest.mark.parametrize("tokens,top,experts,want", [(8, 4, 16, True), (32, 4, 16, True), (18, 8, 32, True), (19, 8, 32, False), (32, 8, 16, False), (32, 5, 64, False),
                                                     (20, 8, 128, True), (33, 1, 16, False), (32, 1, 128, False)])
def test_routing_of_few_tokens_takes_one_launch_while_its_ctas_have_an_sm_each(tokens, top, experts, want):
    """The last two are more than the launch takes: tokens, or scores in shared memory."""
    from llm_b200.csrc import ops
    assert ops.moe_route_few_pays(tokens, top, experts, sms=148) == want
