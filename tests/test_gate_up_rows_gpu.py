"""Gate/Up with weight rows on the tensor core's M side, at the edges of its token blocks and row tiles.

Calls with few work items take that form.  Codes and scales are compared bit for bit with the unfused
CUDA-core kernels, for experts whose rows end on, before and behind a block of 32 and a tile of 128.
"""

import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS = [1, 16, 31, 32, 33, 0, 64, 65, 96, 97, 127, 128, 129, 300]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("layout", ["split", "interleaved"])
@pytest.mark.parametrize("hidden,inter,offset", [(256, 256, 0), (512, 512, 1), (1280, 256, 2)])
def test_ragged_rows_equal_unfused_bits(hidden, inter, offset, layout, dtype):
    """``offset``: elements by which the weight scales' start lies off a 16-byte boundary."""
    from grain_gemm_b200 import _loader, moe
    gen = torch.Generator(device="cuda").manual_seed(hidden + inter)
    experts, tokens = len(ROWS), sum(ROWS)

    def codes(*shape):
        return torch.randint(-127, 128, shape, dtype=torch.int8, device="cuda", generator=gen)

    ids = torch.cat([torch.full((rows,), e) for e, rows in enumerate(ROWS)])[torch.randperm(tokens)].cuda()[:, None]
    x, w1 = codes(tokens, hidden), codes(experts, 2 * inter, hidden)
    scale_x = torch.exp(3 * torch.randn((tokens, hidden // 256), device="cuda", generator=gen)) / 127
    scale_x[0:5] = 0.0              # gate = up = 0
    scale_x[5:10] *= 3.0e3          # exp(-gate) overflows, infinities in the 16-bit type
    scale_x[10:15] *= 1.0e-30       # tiny numerators
    scale_x[15:20] *= 1.0e30        # beyond the FMA sequence's range: infinity and NaN
    count = experts * (hidden // 256) * 2 * inter
    memory = (0.5 + torch.rand((count + 4,), device="cuda", generator=gen)) / 3000
    scale_w = memory[offset:offset + count].view(experts, hidden // 256, 2 * inter)
    results = []
    for tile_rows in (128, 32):
        routes = moe.prepare_routes(ids, experts, None, tile_rows=tile_rows)
        qh, sh = moe.gate_up_swiglu_quantize(x, scale_x, w1, scale_w, routes, output_dtype=dtype,
                                             gate_up_layout=layout)
        results.append((qh, sh.view(torch.int32)))
    assert torch.equal(results[0][0], results[1][0])
    assert torch.equal(results[0][1], results[1][1])
    assert _loader.device_status() == 0
