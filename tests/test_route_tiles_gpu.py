"""The row-tile list that the routing kernels write themselves, against the list made from the offsets, at
the edges of the three routing forms (one CTA up to 1024 assignments, up to 8192, chunks beyond).
"""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile_rows", [128, 32, 1])
@pytest.mark.parametrize("tokens,top_k,experts", [
    (1, 1, 1), (1, 8, 128), (512, 2, 33), (1024, 1, 1024), (129, 8, 511), (1024, 8, 512), (1025, 8, 8),
    (8192, 1, 511), (8193, 1, 511), (4000, 6, 1500)])
def test_list_written_with_the_routing(tokens, top_k, experts, tile_rows):
    from grain_gemm_b200 import moe
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    # A few experts get most rows, many get none; some ids are out of range, some tokens masked.
    ids = (experts * torch.rand((tokens, top_k), device="cuda", generator=gen) ** 3).long()
    ids[torch.rand((tokens, top_k), device="cuda", generator=gen) < 0.05] = experts + 7
    mask = torch.rand((tokens,), device="cuda", generator=gen) < 0.9
    for dtype in (torch.int64, torch.int32):
        together = moe.prepare_routes(ids.to(dtype), experts, mask, tile_rows=tile_rows)
        apart = moe.prepare_tiles(moe.prepare_routes(ids.to(dtype), experts, mask, tile_rows=0), tile_rows)
        for field in ("order", "counts", "offsets", "inverse", "effective_ids", "statistics", "tile_expert",
                      "tile_row"):
            assert torch.equal(getattr(together, field), getattr(apart, field)), field


@pytest.mark.parametrize("tokens,top_k,experts", [(128, 8, 64), (129, 8, 64), (3000, 4, 256)])
def test_selection_and_routing_of_any_size(tokens, top_k, experts):
    """The native call for sizes on either side of the one-launch form."""
    from grain_gemm_b200 import moe, route_topk
    from grain_gemm_b200.quantize import route_topk_routes
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    logits = torch.randn((tokens, experts), device="cuda", generator=gen)
    mask = torch.rand((tokens,), device="cuda", generator=gen) < 0.9
    for dtype in (torch.int64, torch.int32):
        weights, ids, routes = route_topk_routes(logits, top_k, token_mask=mask, ids_dtype=dtype)
        expected_weights, expected_ids = route_topk(logits, top_k, ids_dtype=dtype)
        assert torch.equal(weights, expected_weights) and torch.equal(ids, expected_ids) and ids.dtype == dtype
        expected = moe.prepare_routes(expected_ids, experts, mask)
        assert routes.tile_rows == 128
        assert (routes.tokens, routes.top_k, routes.experts) == (tokens, top_k, experts)
        for field in ("order", "counts", "offsets", "inverse", "effective_ids", "statistics", "tile_expert",
                      "tile_row"):
            assert torch.equal(getattr(routes, field).reshape(-1), getattr(expected, field).reshape(-1)), field
