"""The norm over several streams for few rows, which runs over clusters of CTAs, at the edges of its range of rows and widths."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def partials(ops, y, splits):
    """y as a sum of `splits` float32 terms."""
    if splits == 0:
        return y.to(torch.bfloat16).contiguous()
    parts = torch.randn(splits, *y.shape, device=DEV)
    parts[-1] += y - parts.sum(0)
    return ops.PartialSum(parts.contiguous(), splits, y.shape[0], y.shape[1], torch.bfloat16)


@pytest.mark.parametrize("streams,hidden", [(1, 1024), (2, 1032), (3, 2040), (4, 2048), (4, 2056), (5, 1024)])
@pytest.mark.parametrize("rows", [1, 8, 37, 38, 74, 75])
@pytest.mark.parametrize("splits", [None, 0, 1, 5])
def test_hc_norm(rows, streams, hidden, splits):
    from llm_b200.csrc import ops
    torch.manual_seed(rows + hidden)
    x, y = torch.randn(rows, streams * hidden, device=DEV), torch.randn(rows, hidden, device=DEV)
    mix, wout, win = torch.randn(streams, streams, device=DEV), torch.randn(streams, device=DEV), torch.randn(streams, device=DEV)
    gain = torch.tensor([1.3], device=DEV)
    delta = None if splits is None else partials(ops, y, splits)
    new = x.double().view(rows, streams, hidden)
    if splits is not None:
        term = delta.double() if splits == 0 else delta.buf.double().sum(0)
        new = torch.einsum("sr,tsw->trw", mix.double(), new) + wout.double()[:, None] * term[:, None]
    out = torch.empty(rows, hidden, device=DEV, dtype=torch.bfloat16)
    ops.hc_norm(x, delta, mix if delta is not None else None, wout if delta is not None else None, win, gain, out, rows, hidden, streams, 1e-5,
                torch.bfloat16)
    assert float((x.double().view(rows, streams, hidden) - new).abs().max()) < 5e-5
    u = torch.einsum("s,tsw->tw", win.double(), new)
    ref = u / torch.sqrt((u * u).mean(-1, keepdim=True) + 1e-5) * 1.3
    assert bool(((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all())
