"""Which products of few rows go to the kernel of their own (gemm_few), on the CPU (operands that only say where they lie)."""
import types

import pytest
import torch


def weights(n, k):
    """A bfloat16 matrix on a device, as far as the choice looks at it."""
    return types.SimpleNamespace(dtype=torch.bfloat16, shape=(n, k), stride=lambda d: (k, 1)[d], data_ptr=lambda: 0, is_cuda=True)


def at(offset, *shape):
    """A float32 tensor whose first number lies `offset` bytes behind a 16-byte boundary."""
    n = torch.Size(shape).numel()
    buf = torch.zeros(n + 8)
    first = (-buf.data_ptr() % 16 + offset) // 4
    return buf[first:first + n].view(*shape)


@pytest.mark.parametrize("resid,gain,want", [(0, 0, True), (0, 4, False), (0, 8, False), (4, 0, False), (8, 8, False)])
def test_rows_before_their_norm_lie_on_16_bytes(resid, gain, want, monkeypatch):
    """A gain may be a view that a caller gave among the model's tensors: the kernel copies it 16 bytes at a time, the norm's own kernel takes any."""
    from llm_b200.csrc import ops
    monkeypatch.setattr(ops, "sm_count", lambda: 148)
    rows = ops.NormedRows(at(resid, 4, 64), at(gain, 64), 1e-5, 4, torch.bfloat16)
    assert ops.gemm_few_available(rows, weights(192, 64), 4) == want


@pytest.mark.parametrize("rows,n,unsummed", [(8, 1 << 21, True), (8, (1 << 21) + 8, False), (1, 1 << 24, True), (1, (1 << 24) + 8, False)])
def test_results_beyond_the_scratch_buffer_are_written_out(rows, n, unsummed, monkeypatch):
    """64 MB of float32 sums are what the buffer holds."""
    from llm_b200.csrc import ops
    from llm_b200.parts.linear import linear
    out = types.SimpleNamespace(dtype=torch.bfloat16, shape=(rows, n))
    monkeypatch.setattr(ops, "gemm_few_available", lambda a, w, rows: True)
    monkeypatch.setattr(ops, "gemm_few", lambda a, w, out, rows, **k: out)
    monkeypatch.setattr(ops, "gemm_few_sums_pay", lambda a, rows: True)
    monkeypatch.setattr(ops, "_partials", lambda device: torch.empty(ops._PARTIAL_BYTES // 4, device="meta"))
    w = types.SimpleNamespace(shape=(n, 64), device="meta")
    got = linear(None, w, out, rows, allow_partial=True)
    assert isinstance(got, ops.PartialSum) if unsummed else got is out


@pytest.mark.parametrize("n,k,plain,normed,gated", [
    (2368, 64, True, True, True), (2369, 64, False, True, True), (7104, 64, False, True, True), (7105, 64, False, False, True),
    (11840, 64, False, False, True), (11841, 64, False, False, False), (4736, 256, True, True, True), (4737, 256, False, True, True),
    (11840, 512, True, True, True), (16576, 512, False, True, True), (16577, 512, False, False, True), (21313, 512, False, False, False),
    (32000, 768, False, True, True), (32000, 1024, True, True, True), (128256, 1024, True, True, True), (128256, 4096, True, True, True)])
def test_short_rows_on_many_tiles_take_the_other_kernel(n, k, plain, normed, gated, monkeypatch):
    from llm_b200.csrc import ops
    monkeypatch.setattr(ops, "sm_count", lambda: 148)
    rows = torch.zeros(4, k, dtype=torch.bfloat16)
    a = types.SimpleNamespace(dtype=torch.bfloat16, is_cuda=True, stride=rows.stride, data_ptr=lambda: 0)
    rows_under = ops.NormedRows(at(0, 4, k), at(0, k), 1e-5, 4, torch.bfloat16)
    assert ops.gemm_few_available(a, weights(n, k), 4) == plain
    assert ops.gemm_few_available(rows_under, weights(n, k), 4) == normed
    assert ops.gemm_few_available(a, weights(n, k), 4, gated=True) == ops.gemm_few_available(rows_under, weights(n, k), 4, gated=True) == gated


@pytest.mark.parametrize("rows,k,want", [(8, 4032, "few"), (8, 4096, "split"), (5, 6528, "few"), (5, 6592, "split"), (1, 14336, "few")])
@pytest.mark.parametrize("kind", ["unsummed", "whole", "biased", "normed"])
def test_unsummed_products_of_long_rows_are_split(rows, k, want, kind, monkeypatch):
    """Only where the next kernel takes several terms, and the rows are there as they are multiplied."""
    from llm_b200.csrc import ops
    from llm_b200.parts.linear import linear
    sent = []
    monkeypatch.setattr(ops, "gemm_few_available", lambda a, w, rows: True)
    monkeypatch.setattr(ops, "gemm_fast_available", lambda *a: True)
    monkeypatch.setattr(ops, "gemm_fast", lambda *a, **k: sent.append("split"))
    monkeypatch.setattr(ops, "gemm_few", lambda *a, **k: sent.append("few"))
    monkeypatch.setattr(ops, "gemm_few_sums", lambda *a, **k: sent.append("few"))
    x = torch.zeros(rows, k, dtype=torch.bfloat16)
    if kind == "normed":
        x = ops.NormedRows(x.float(), torch.zeros(k), 1e-5, rows, torch.bfloat16)
    linear(x, torch.zeros(96, k, dtype=torch.bfloat16), torch.zeros(rows, 96, dtype=torch.bfloat16), rows, allow_partial=kind != "whole",
           bias=torch.zeros(96) if kind == "biased" else None)
    assert sent == [want if kind == "unsummed" else "few"]
