"""Grouped products of prompts, whose tiles get their width on the device from the number of row tiles in use."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("used", [1, 2, 8])
@pytest.mark.parametrize("N,E,pairs", [(264, 8, 9000), (300, 8, 9000), (1408, 8, 1500), (2048, 16, 2048)])
def test_every_width_gives_the_same_products(used, N, E, pairs):
    """The pairs go to `used` of the experts, so that few or all of the row tiles that were planned for are in use: other widths, the same
    numbers up to float32 sums in one order (K of two blocks), against float64."""
    from llm_b200.csrc import ops
    K, tile = 128, ops.MOE_TC_TILE
    g = torch.Generator(device=DEV).manual_seed(N + used)
    ids = (torch.arange(pairs, device=DEV, dtype=torch.int32) * 7 % used).contiguous()
    max_tiles = ops.moe_max_tiles(pairs, E, tile)
    width = 256 if N % 256 == 0 or N % 256 > 128 else 128
    assert max_tiles * -(-N // width) > ops.sm_count()                   # the kernel of persistent CTAs
    z = lambda n: torch.zeros(n, dtype=torch.int32, device=DEV)
    meta, tile_expert, slot_src, pair_slot = z(4), z(max_tiles), z(max_tiles * tile), z(pairs)
    ops.moe_group(ids, pairs, E, meta, tile_expert, slot_src, pair_slot, max_tiles, tile)
    x = torch.randn(pairs, K, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(E, N, K, generator=g, device=DEV) * 0.1).to(torch.bfloat16)
    rows = torch.zeros(max_tiles * tile, K, device=DEV, dtype=torch.bfloat16)
    ops.moe_gather(rows, x, slot_src, meta, 1, tile, max_tiles)
    y = torch.full((max_tiles * tile, N), 7.0, device=DEV)
    ops.moe_gemm_tc(rows, tile_expert, meta, w, y, max_tiles, tile=tile)
    half = torch.full((max_tiles * tile, N), 7.0, device=DEV, dtype=torch.bfloat16)
    ops.moe_gemm_tc(rows, tile_expert, meta, w, half, max_tiles, tile=tile, act="relu2")
    assert ops.gemm_tc_take_error() == 0
    slots = pair_slot.long()
    ref = torch.einsum("pk,pnk->pn", x.double(), w[ids.long()].double()) if pairs <= 2048 else torch.cat(
        [torch.einsum("pk,pnk->pn", x[i:i + 1000].double(), w[ids[i:i + 1000].long()].double()) for i in range(0, pairs, 1000)])
    assert float((y[slots].double() - ref).norm() / ref.norm()) < 1e-6
    relu2 = torch.relu(ref) ** 2
    assert float((half[slots].double() - relu2).norm() / relu2.norm()) < 2.0 ** -8
    in_use = int(meta[0]) * tile
    assert bool((y[in_use:] == 7).all())                                 # tiles that are not in use are left alone
