"""Codes of the branch-free requantisation against plain division and rounding, where they could differ.

The kernels divide by a sequence of fused multiply-adds and round by adding 1.5 * 2^23; rows whose
range that sequence does not cover take the library division.  Both have to give the codes of
``nearbyint(v / scale)`` clamped to [-127, 127], bit for bit, and NaN the code -127.
"""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _expected(x, group):
    grouped = x.reshape(-1, group)
    amax = torch.where(grouped.isnan(), 0.0, grouped.abs()).amax(dim=1, keepdim=True)
    scale = amax.clamp_min(1.0e-12) / 127.0
    codes = torch.round(grouped / scale).clamp(-127, 127)
    codes = torch.where(grouped.isnan(), -127.0, codes).to(torch.int8)
    return codes.reshape(x.shape), scale.reshape(x.shape[0], -1)


@pytest.mark.parametrize("group", [32, 256])
def test_codes_next_to_the_rounding_boundaries(group):
    from grain_gemm_b200 import quantize_rows
    gen = torch.Generator().manual_seed(group)
    rows = 512
    # Row maxima over the whole range of the sequence, a value exactly half way between two codes in
    # real arithmetic, and its neighbours in FP32 on either side.
    amax = torch.exp(torch.empty((rows, 1)).uniform_(-27.0, 68.0, generator=gen))
    halves = torch.randint(-127, 127, (rows, 1024), generator=gen) + 0.5
    x = (halves.double() * (amax.double() / 127)).float()
    direction = torch.randint(-1, 2, x.shape, generator=gen)
    x = torch.where(direction == 0, x, torch.nextafter(x, direction.float() * torch.inf))
    x[:, ::group] = amax
    codes, scale = quantize_rows(x.cuda(), group)
    expected, expected_scale = _expected(x, group)
    assert torch.equal(scale.cpu(), expected_scale)
    assert torch.equal(codes.cpu(), expected)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_nan_zeros_and_rows_out_of_range(dtype):
    from grain_gemm_b200 import quantize_rows
    gen = torch.Generator().manual_seed(3)
    x = torch.randn((8, 512), generator=gen).to(dtype)
    x[0, 3], x[1, 300] = float("nan"), float("nan")
    x[2, :256] = 0.0
    x[3, 5] = -0.0
    if dtype != torch.float16:
        x[4, 7], x[4, 8] = 2.0e30, -3.0e38        # beyond the sequence: library division
        x[5, :256] = x[5, :256] * 1.0e-37          # below the smallest scale: all codes 0
        x[6, 9], x[6, 10] = 9.9e29, float("nan")
    codes, scale = quantize_rows(x.cuda())
    expected, expected_scale = _expected(x.float(), 256)
    assert torch.equal(scale.cpu(), expected_scale)
    assert torch.equal(codes.cpu(), expected)
