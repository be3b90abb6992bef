"""Blocks of several arrangements on one residual stream: who reads the stream's rows in the compute dtype reads them as they are."""
import types

import pytest
import torch

BF16, F64 = torch.bfloat16, torch.float64
W, FF, EPS, ALPHA = 64, 128, 1e-5, 1.25


def plain_kernels(monkeypatch):
    """The kernels that these blocks reach, in plain torch (their arithmetic on the CPU; which of them run is the package's choice)."""
    from llm_b200.csrc import ops
    put = lambda name, f: monkeypatch.setattr(ops, name, f)
    whole = lambda y: y.float()
    rms = lambda x, gain, eps: x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * gain

    def add_rmsnorm(resid, delta, gamma, out, rows, eps):
        if delta is not None:
            resid[:rows] += whole(delta[:rows])
        if out is not None:
            out[:rows] = rms(resid[:rows], gamma, eps).to(out.dtype)

    def sum_rmsnorm(resid, alpha, y, gain, out, rows, eps, dtype):
        resid[:rows] = rms(alpha * resid[:rows] + whole(y[:rows]), gain, eps)
        if out is not None:
            out[:rows] = resid[:rows].to(out.dtype)

    def add_layernorm(resid, delta, post, mult, pre, out, rows, eps):
        assert post is None and out is None
        resid[:rows] += mult * whole(delta[:rows])

    def gemm_few(a, w, out, rows, kind=None, bias=None, limit=0.0, alpha=0.0):
        x = rms(a.resid[:rows], a.gain, a.eps).to(BF16) if isinstance(a, ops.NormedRows) else a[:rows]
        z = x.float() @ w.float().T
        if kind == "add":
            out[:rows] += z
        elif kind == "silu":
            g, u = z.chunk(2, -1)
            out[:rows] = (torch.nn.functional.silu(g) * u).to(out.dtype)
        else:
            out[:rows] = (z if bias is None else z + bias).to(out.dtype)
        return out

    def silu_mul(out, gate_up, rows, act="silu"):
        g, u = gate_up[:rows].float().chunk(2, -1)
        out[:rows] = (torch.nn.functional.silu(g) * u).to(out.dtype)

    def concat_embedding(out, resid, table, ids, n):
        out[:n] = torch.cat([resid[:n], table[ids[:n].long()].float()], -1).to(out.dtype)

    put("add_rmsnorm", add_rmsnorm), put("sum_rmsnorm", sum_rmsnorm), put("add_layernorm", add_layernorm), put("gemm_few", gemm_few)
    put("silu_mul", silu_mul), put("concat_embedding", concat_embedding)
    put("gemm_few_available", lambda a, w, rows, gated=False: rows <= 8)
    put("gemm_few_sums", lambda a, w, rows, dtype: gemm_few(a, w, torch.empty(rows, w.shape[0], dtype=dtype), rows))
    put("gemm_simt", lambda a, w, out, rows: out[:rows].copy_(a[:rows].float() @ w.float().T))
    put("add_bias", lambda x, bias, rows: x[:rows].add_(bias.to(x.dtype)))
    put("cast_rows", lambda out, rows_f32, n: out[:n].copy_(rows_f32[:n]))


class Scaled:
    """A mixer that returns what it reads, times a number."""

    def __init__(self, prefix, dtype, device):
        self.dtype = dtype

    def forward(self, x, ctx, view):
        return (x * 0.75).to(self.dtype).contiguous()

    def state_need(self):
        return None


def layers(device, tensors, offset=0):
    """offset: the gains are views that begin so many numbers into a buffer."""
    from llm_b200.models.spec import PartSpec
    from llm_b200.parts.base import part_class, register_part
    from llm_b200.parts.block import PostNormBlock, PreNormBlock, StreamBlock
    try:
        part_class("mixer", "scaled_rows")
    except KeyError:
        register_part("mixer", "scaled_rows", Scaled)
    norm = lambda p: PartSpec("rmsnorm", {"size": W, "eps": EPS}, p)
    mixer = PartSpec("scaled_rows", {}, "m")
    post = [PostNormBlock({"mixer": mixer, "norm1": norm(f"post{i}")}, BF16, device, alpha=ALPHA) for i in (0, 1)]
    pre = PreNormBlock({"norm1": norm("n1"), "mixer": mixer, "norm2": norm("n2"),
                        "ffn": PartSpec("swiglu", {"hidden_size": W, "intermediate_size": FF}, "ff")}, BF16, device)
    again = StreamBlock({"stream": PartSpec("embedding_reinjection", {"hidden_size": W, "vocab_size": 32, "passes": 1, "pass_index": 0,
                                                                      "table_name": "table"}, "loop")}, BF16, device)
    for part in [p for b in post + [pre, again] for p in b.parts.values() if hasattr(p, "bind")]:
        for name, info in part.parameters().items():
            g = torch.Generator().manual_seed(len(tensors))
            t = torch.randn(info.shape, generator=g) * (0.12 if info.kind == "matrix" else 0.1)      # sublayers as large as the stream
            t = (t.to(BF16) if info.kind == "matrix" else t + 1.0 if name.endswith("weight") else t).to(device)
            tensors[name] = torch.cat([t[:offset], t])[offset:] if offset and info.shape == (W,) else t
        part.bind(tensors)
    return post, pre, again


def check(device, rows, middle, offset=0):
    """A post-norm layer, then `middle`, then a post-norm layer, against 64 bits."""
    from llm_b200.parts.base import ResidualStream
    tensors = {}
    post, pre, again = layers(device, tensors, offset)
    t = {n: v.to(F64) for n, v in tensors.items()}
    rms = lambda x, n: x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * t[n + ".weight"]
    x0 = torch.randn(rows, W, generator=torch.Generator().manual_seed(rows)).to(device)
    ids = (torch.arange(rows, dtype=torch.int32, device=device) * 5) % 32
    ctx = types.SimpleNamespace(n_tokens=rows, token_ids=ids,
                                workspace=types.SimpleNamespace(get=lambda tag, n, cols, dtype: torch.empty(n, cols, dtype=dtype, device=device)))
    stream = ResidualStream(x0.clone(), rows)
    post[0].forward(stream, ctx, None)
    x = rms((ALPHA + 0.75) * x0.to(F64), "post0")
    if "prenorm" in middle:
        pre.forward(stream, ctx, None)
        x = x + 0.75 * rms(x, "n1")
        h = rms(x, "n2")
        x = x + (torch.nn.functional.silu(h @ t["ff.gate_proj.weight"].T) * (h @ t["ff.up_proj.weight"].T)) @ t["ff.down_proj.weight"].T
    if "stream" in middle:
        again.forward(stream, ctx, None)
        x = torch.cat([x, t["table"][ids.long()]], -1) @ t["loop.in"].T + t["loop.step"][0]
    post[1].forward(stream, ctx, None)
    x = rms((ALPHA + 0.75) * x, "post1")
    assert stream.pending is None
    # a dozen roundings to bfloat16 (2^-9 each) on the way, some of them of sums that partly cancel; rows from before `middle` differ by 0.1 and more
    assert float((stream.resid.to(F64) - x).norm() / x.norm()) < 0.03


@pytest.mark.parametrize("middle", ["prenorm", "stream", "prenorm stream"])
@pytest.mark.parametrize("rows", [4, 8, 9, 12])
def test_rows_after_other_arrangements(rows, middle, monkeypatch):
    plain_kernels(monkeypatch)
    check(torch.device("cpu"), rows, middle)


@pytest.mark.gpu
@pytest.mark.parametrize("middle", ["prenorm", "stream", "prenorm stream"])
@pytest.mark.parametrize("rows", [4, 8, 9, 12])
def test_rows_after_other_arrangements_on_the_kernels(rows, middle):
    check(torch.device("cuda"), rows, middle)


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [4, 9])
@pytest.mark.parametrize("offset", [1, 2])
def test_gains_off_the_16_byte_grid(rows, offset):
    check(torch.device("cuda"), rows, "prenorm", offset)
