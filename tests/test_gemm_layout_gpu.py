"""Edges of the tensor-core kernels' weight order, scale ring and launch forms, bit for bit
against the oracle.

* Widths that are a multiple of 32 get their weight rows in fragment order, others in their own.
* Column scales move 16 bytes at a time where rows and base allow it, 4 bytes otherwise.
* Scales change hands four K groups at a time: groups around the chunk's and the ring's length.
* Quantised rows: one or four 256-value chunks per warp, guarded or library division.
"""

import pytest
import torch

from oracle import cpu as oracle

pytestmark = pytest.mark.gpu

VARIANTS = ["tc_n256", "tc_n128", "tc_n64", "tc_pair_n256", "tc_pair_n128"]


def _case(m, n, k, g, seed):
    gen = torch.Generator().manual_seed(seed)
    a = torch.randint(-127, 128, (m, k), dtype=torch.int8, generator=gen)
    w = torch.randint(-127, 128, (n, k), dtype=torch.int8, generator=gen)
    q = (k + g - 1) // g
    return (a, w.t(), (0.5 + torch.rand((m, q), generator=gen)) / 127,
            (0.5 + torch.rand((q, n), generator=gen)) / 127)


def _run(tensors, g, dtype, variant):
    from grain_gemm_b200 import int8_gemm
    return int8_gemm(*tensors, group_size=g, output_dtype=dtype, variant=variant)


@pytest.mark.parametrize("variant", VARIANTS)
@pytest.mark.parametrize("n", [31, 32, 33, 96, 130, 288, 520, 544])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_widths_in_both_weight_orders(variant, n, dtype):
    case = _case(140, n, 528, 256, n)
    actual = _run([t.cuda() for t in case], 256, dtype, variant)
    assert torch.equal(actual.cpu(), oracle.int8_gemm(*case, 256, dtype))


@pytest.mark.parametrize("variant", VARIANTS)
@pytest.mark.parametrize("group", [32, 256])
@pytest.mark.parametrize("groups", [1, 3, 4, 5, 8, 9])
def test_group_counts_around_the_scale_chunks(variant, group, groups):
    # One tile per CTA (pair): the ring's chunks and slots within a tile.
    case = _case(300, 320, group * groups, group, groups)
    actual = _run([t.cuda() for t in case], group, torch.float32, variant)
    assert torch.equal(actual.cpu(), oracle.int8_gemm(*case, group, torch.float32))


@pytest.mark.parametrize("variant", VARIANTS)
@pytest.mark.parametrize("groups", [1, 3, 5, 9])
def test_many_tiles_per_cta_carry_the_ring(variant, groups):
    # More than two tiles for every CTA (pair), so that a chunk that was only partly used and the
    # ring's position are carried from tile to tile.
    rows, columns, ctas = {"tc_n256": (128, 256, 1), "tc_n128": (128, 128, 1), "tc_n64": (128, 64, 1),
                           "tc_pair_n256": (256, 256, 2), "tc_pair_n128": (256, 128, 2)}[variant]
    m, n = 2600, 19 * columns + 32
    tiles = -(-m // rows) * -(-n // columns)
    workers = torch.cuda.get_device_properties(0).multi_processor_count // ctas
    assert tiles > 2 * workers
    case = _case(m, n, 32 * groups, 32, 7 + groups)
    actual = _run([t.cuda() for t in case], 32, torch.bfloat16, variant)
    take = torch.arange(0, m, 37)
    expected = oracle.int8_gemm(case[0][take], case[1], case[2][take], case[3], 32, torch.bfloat16)
    assert torch.equal(actual.cpu()[take], expected)


@pytest.mark.parametrize("form", ["offset", "odd_pitch", "strided", "transposed"])
def test_column_scales_that_cannot_move_as_vectors(form):
    case = _case(70, 256, 1280, 256, 3)
    a, b, sa, sb = [t.cuda() for t in case]
    q, n = sb.shape
    if form == "offset":
        sb = torch.cat((sb.new_zeros(1), sb.flatten()))[1:].view(q, n)
    elif form == "odd_pitch":
        sb = torch.nn.functional.pad(sb, (0, 1))[:, :n]
    elif form == "strided":
        sb = sb.repeat_interleave(2, dim=1)[:, ::2]
    else:
        sb = sb.t().contiguous().t()
    actual = _run([a, b, sa, sb], 256, torch.float32, "tc_n64")
    assert torch.equal(actual.cpu(), oracle.int8_gemm(*case, 256, torch.float32))


@pytest.mark.parametrize("rows,width", [(1, 256), (3, 512), (4737, 2048), (4738, 2304)])
@pytest.mark.parametrize("group", [32, 256])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_quantised_rows_of_both_launch_forms(rows, width, group, dtype):
    from grain_gemm_b200 import quantize_rows
    gen = torch.Generator().manual_seed(rows)
    x = torch.randn((rows, width), generator=gen).to(dtype)
    x[0, :4] = torch.tensor([0.0, float("inf"), -float("inf"), float("nan")]).to(dtype)
    x[rows // 2] = 0
    x[-1] *= 1e-4
    q, scales = quantize_rows(x.cuda(), group)
    take = torch.unique(torch.cat((torch.arange(0, rows, 61), torch.tensor([0, rows // 2, rows - 1]))))
    blocks = x[take].float().reshape(len(take), width // group, group)
    finite = blocks.isfinite().all(-1)
    amax = blocks.abs().amax(-1)
    expected_scale = amax.clamp_min(1e-12) / 127
    expected = (blocks / expected_scale[..., None]).round().clamp(-127, 127)
    got = q.cpu()[take].reshape(blocks.shape).float()
    assert torch.equal(scales.cpu()[take][finite], expected_scale[finite])
    assert torch.equal(got[finite], expected[finite])
