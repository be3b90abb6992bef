"""What arrangements hand to the parts they call, and what the parts may hand back."""
import types

import pytest
import torch

BF16 = torch.bfloat16


class Norm:
    def __init__(self, prefix="", dtype=None, device=None):
        pass

    def forward(self, stream, ctx):
        stream.fold(ctx)
        return stream.resid[:stream.rows].clone()

    def unformed(self, stream):
        return "rows before their norm" if stream.pending is None else None


class Plain:
    """A mixer of a caller's own whose forward has parameters named like the options, with meanings of their own."""

    def __init__(self, prefix="", dtype=None, device=None):
        self.got = []

    cache_need = state_need = lambda self: None

    def forward(self, x, ctx, view=None, into="a place", whole="a number", **more):
        self.got.append((x if isinstance(x, str) else "rows", into, whole))
        return x

    def reads_unformed(self, rows, ctx):
        return True


def marked():
    from llm_b200.parts.base import takes

    class Marked(Plain):
        @takes("into", "whole")
        def forward(self, x, ctx, view=None, into=None, whole=False):
            Plain.forward(self, x, ctx, view, into, whole)
            if into is None:
                return torch.ones(ctx.n_tokens, 4)
            into.resid[:into.rows] += 1.0
            return None

    class Own(Marked):
        def forward(self, x, ctx, view=None):
            return Plain.forward(self, x, ctx, view)

    return Marked, Own


def register(kind, cls, role="mixer"):
    from llm_b200.parts.base import register_part
    register_part(role, kind, cls)


def prenorm(mixer):
    from llm_b200.models.spec import PartSpec
    from llm_b200.parts.block import PreNormBlock
    register("option_norm", Norm, "norm"), register("option_mixer", mixer)
    return PreNormBlock({"norm1": PartSpec("option_norm"), "mixer": PartSpec("option_mixer")}, torch.float32, torch.device("cpu"))


def test_only_marked_parts_get_the_stream():
    from llm_b200.parts.base import ResidualStream
    Marked, Own = marked()
    ctx = types.SimpleNamespace(n_tokens=2)
    for cls, want in ((Plain, ("rows", "a place", "a number")), (Own, ("rows", "a place", "a number"))):
        block, stream = prenorm(cls), ResidualStream(torch.zeros(2, 4), 2)
        block.forward(stream, ctx, None)
        assert block.mixer.got == [want] and stream.pending is not None
    block, stream = prenorm(Marked), ResidualStream(torch.zeros(2, 4), 2)
    block.forward(stream, ctx, None)
    block.forward(stream, ctx, None)
    assert block.mixer.got == [("rows before their norm", stream, False)] * 2
    assert stream.pending is None and bool((stream.resid == 2).all())      # None: the part has added its result


@pytest.mark.parametrize("rows,want", [(1, True), (8, True), (9, False)])
def test_the_left_of_two_mixers_is_asked_for_a_whole_result_of_few_rows(rows, want, monkeypatch):
    from llm_b200.csrc import ops
    from llm_b200.models.spec import PartSpec
    from llm_b200.parts.recurrent import ParallelMixers
    Marked, Own = marked()
    monkeypatch.setattr(ops, "scaled_sum", lambda out, a, b, sa, sb, n: out.copy_(sa * a + sb * b))
    ctx = types.SimpleNamespace(n_tokens=rows, workspace=types.SimpleNamespace(get=lambda tag, n, cols, dtype: torch.empty(n, cols)))
    view = types.SimpleNamespace(state=torch.zeros(1, 0))
    monkeypatch.setattr("llm_b200.parts.recurrent._sub_view", lambda view, state: view)
    for cls, whole in ((Marked, want), (Own, "a number"), (Plain, "a number")):
        register("option_left", cls), register("option_right", Own)
        two = ParallelMixers(4, PartSpec("option_left"), PartSpec("option_right"), combine="scaled_sum", dtype=torch.float32, device="cpu")
        x = torch.ones(rows, 4)
        got = two.forward(x, ctx, view)
        assert two.left.got[0][2] == whole and bool((got == 2).all())
