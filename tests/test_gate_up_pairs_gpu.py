"""The exchange of row maxima between the two CTAs of a Gate/Up item, where it could race.

A pair that walks many items with one or two K groups each reaches its next item while its partner
still reads the maxima of the last one; the two alternating sets of maxima and barriers have to
keep them apart.  Codes and scales are compared bit for bit with the form that fetches rows by
index, which always runs on single CTAs, and with the unfused CUDA-core kernels.
"""

import pytest
import torch

pytestmark = pytest.mark.gpu

EXPERTS, INTER = 8, 14336


def _kernels(call):
    """Names of the kernels that ``call`` launches."""
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as recorded:
        call()
        torch.cuda.synchronize()
    return [event.key for event in recorded.key_averages()]


def _items_of_a_pair(tokens, top_k):
    """Items the busiest pair walks, by the rule in ``gate_up_pairs`` (one row tile per expert here)."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    items = min(tokens * top_k, EXPERTS) * (INTER // 256)
    single, pairs = -(-items // sms), -(-items // (sms // 2))
    assert pairs * 52 < single * 100, "this size no longer goes to pairs"
    return pairs


@pytest.mark.parametrize("hidden", [256, 512, 1280])
@pytest.mark.parametrize("layout", ["split", "interleaved"])
@pytest.mark.parametrize("tokens,top_k", [(4, 2), (33, 2), (60, 8)])
def test_many_short_items_per_pair(hidden, layout, tokens, top_k):
    from grain_gemm_b200 import _loader, moe
    generator = torch.Generator(device="cuda").manual_seed(hidden + tokens)

    def codes(*shape):
        return torch.randint(-127, 128, shape, dtype=torch.int8, device="cuda", generator=generator)

    w1 = codes(EXPERTS, 2 * INTER, hidden)
    s1 = (0.5 + torch.rand((EXPERTS, hidden // 256, 2 * INTER), device="cuda", generator=generator)) / 3000
    # Every expert gets rows, in a ragged way.
    ids = torch.stack([torch.randperm(EXPERTS, device="cuda", generator=generator)[:top_k]
                       for _ in range(tokens)])
    ids[:4, 0], ids[:4, 1] = torch.arange(0, 8, 2), torch.arange(1, 8, 2)
    assert _items_of_a_pair(tokens, top_k) >= 3

    def stage(x, scale_x, tile_rows, row_gather):
        routes = moe.prepare_routes(ids, EXPERTS, tile_rows=tile_rows)
        qh, sh = moe.gate_up_swiglu_quantize(x, scale_x, w1, s1, routes, gate_up_layout=layout,
                                             row_gather=row_gather)
        return qh, sh

    for repeat in range(6):
        x = codes(tokens, hidden)
        # Row maxima that differ by orders of magnitude from row to row and from call to call.
        scale_x = torch.exp(4 * torch.randn((tokens, hidden // 256), device="cuda", generator=generator)) / 127
        pairs = stage(x, scale_x, 128, False)
        single = stage(x, scale_x, 128, True)
        assert torch.equal(pairs[0], single[0]) and torch.equal(pairs[1], single[1]), repeat
        if repeat == 0:
            unfused = stage(x, scale_x, 32, False)
            assert torch.equal(pairs[0], unfused[0]) and torch.equal(pairs[1], unfused[1])
    assert _loader.device_status() == 0

    def launched(row_gather):
        names = _kernels(lambda: stage(x, scale_x, 128, row_gather))
        return [name for name in names if "moe_gate_up_tc_kernel" in name]

    # Template arguments: output type, rows by index, CTA pairs.
    assert [name.split("<")[1].split(">")[0].split(",")[1:] for name in launched(False)] == [[" false", " true"]]
    assert [name.split("<")[1].split(">")[0].split(",")[1:] for name in launched(True)] == [[" true", " false"]]
