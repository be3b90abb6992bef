"""Which kernel a decode step's attention with options is sent to, on the CPU with the kernels' entry points replaced."""
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
