"""Calls that follow one another without a synchronisation, on inputs that change from call to call
and in buffers that are used again.

The kernels of a call start before their predecessor has finished (programmatic launches).  One that
read an operand too early would see the previous call's bytes in the same buffer, which a
repeated input hides; here every call has its own input, and every result is compared bit for bit
with the same call made on its own between two synchronisations.
"""

import pytest
import torch

pytestmark = pytest.mark.gpu

ROUNDS = 24


def _chained(inputs, call):
    """``call(slot)`` on every input in turn: the input is copied into the same buffers, the results
    are copied out, nothing waits for the GPU in between."""
    slot = [torch.empty_like(t) for t in inputs[0]]
    results = []
    torch.cuda.synchronize()
    for values in inputs:
        for held, value in zip(slot, values):
            held.copy_(value)
        results.append([t.clone() for t in call(*slot)])
    torch.cuda.synchronize()
    return results


def _alone(inputs, call):
    results = []
    for values in inputs:
        fresh = [t.clone() for t in values]
        torch.cuda.synchronize()
        results.append([t.clone() for t in call(*fresh)])
        torch.cuda.synchronize()
    return results


def _compare(chained, alone):
    for step, (got, expected) in enumerate(zip(chained, alone)):
        for index, (one, other) in enumerate(zip(got, expected)):
            assert torch.equal(one, other), f"call {step}, output {index}"


def _weights(shape, generator):
    return torch.randint(-127, 128, shape, dtype=torch.int8, device="cuda", generator=generator)


# Rows that take the weight-streaming kernel, split-K with its fold, one wave of narrow tiles, CTA
# pairs; widths outside the measured table, so that the library's own rule chooses.
@pytest.mark.parametrize("rows", [1, 2, 17, 200, 700])
@pytest.mark.parametrize("group", [32, 256])
def test_linear_layers(rows, group):
    from grain_gemm_b200 import int8_gemm, quantize_rows
    n, k = 3104, 2304
    generator = torch.Generator(device="cuda").manual_seed(rows + group)
    b = _weights((n, k), generator).t()
    scale_b = torch.rand((k // group, n), device="cuda", generator=generator)
    inputs = [(torch.randn((rows, k), device="cuda", generator=generator).to(torch.bfloat16) * (1 + i),)
              for i in range(ROUNDS)]

    def call(x):
        q, scale = quantize_rows(x, group)
        return q, scale, int8_gemm(q, b, scale, scale_b, group_size=group)

    _compare(_chained(inputs, call), _alone(inputs, call))


# The GEMM's weights and scales are a predecessor's output, too.
@pytest.mark.parametrize("rows", [1, 17, 200])
def test_weights_written_just_before(rows):
    from grain_gemm_b200 import int8_gemm, quantize_rows
    n, k = 3104, 2304
    generator = torch.Generator(device="cuda").manual_seed(rows)
    a = _weights((rows, k), generator)
    scale_a = torch.rand((rows, k // 256), device="cuda", generator=generator)
    inputs = [(torch.randn((n, k), device="cuda", generator=generator) * (1 + i),) for i in range(8)]

    def call(w):
        q, scale = quantize_rows(w)
        return (int8_gemm(a, q.t(), scale_a, scale.t(), output_dtype=torch.float32),)

    _compare(_chained(inputs, call), _alone(inputs, call))


# One CTA of routing with its 1024 assignments, one CTA with 8192, three kernels beyond that.
@pytest.mark.parametrize("tokens,experts,top_k", [(1, 32, 4), (24, 8, 2), (700, 32, 4), (3000, 16, 3)])
@pytest.mark.parametrize("layout", ["split", "interleaved"])
def test_moe_layers_with_a_workspace(tokens, experts, top_k, layout):
    from grain_gemm_b200 import moe_ffn, quantize_rows, route_topk_routes
    from grain_gemm_b200.moe import MoEWorkspace
    hidden, inter = 1024, 512
    generator = torch.Generator(device="cuda").manual_seed(tokens)
    w1 = _weights((experts, 2 * inter, hidden), generator).transpose(-2, -1)
    w2 = _weights((experts, hidden, inter), generator).transpose(-2, -1)
    s1 = torch.rand((experts, hidden // 256, 2 * inter), device="cuda", generator=generator) / 2000
    s2 = torch.rand((experts, inter // 256, hidden), device="cuda", generator=generator) / 2000
    inputs = [(torch.randn((tokens, hidden), device="cuda", generator=generator).to(torch.bfloat16) * (1 + i),
               torch.randn((tokens, experts), device="cuda", generator=generator),
               torch.rand((tokens,), device="cuda", generator=generator) > 0.2) for i in range(ROUNDS)]

    def layer(workspace):
        def call(x, logits, mask):
            q, scale_x = quantize_rows(x)
            weights, ids, routes = route_topk_routes(logits, top_k, token_mask=mask)
            given = moe_ffn(q, w1, w2, weights, ids, scale_x=scale_x, scale_gate_up=s1, scale_down=s2,
                            token_mask=mask, gate_up_layout=layout, routes=routes, workspace=workspace)
            routed = moe_ffn(q, w1, w2, weights, ids, scale_x=scale_x, scale_gate_up=s1, scale_down=s2,
                             token_mask=mask, gate_up_layout=layout, workspace=workspace)
            return weights, ids, given, routed
        return call

    alone = _alone(inputs, layer(None))
    for weights, ids, given, routed in alone:
        assert torch.equal(given, routed)
    _compare(_chained(inputs, layer(MoEWorkspace())), alone)


# The stages without moe_ffn's read-back, which waits for routing on every eager call.
@pytest.mark.parametrize("tokens,experts,top_k", [(1, 32, 4), (700, 32, 4), (3000, 16, 3)])
def test_moe_stages_without_any_wait(tokens, experts, top_k):
    from grain_gemm_b200 import moe, quantize_rows, route_topk
    hidden, inter = 1024, 512
    generator = torch.Generator(device="cuda").manual_seed(tokens)
    w1, w2 = _weights((experts, 2 * inter, hidden), generator), _weights((experts, hidden, inter), generator)
    s1 = torch.rand((experts, hidden // 256, 2 * inter), device="cuda", generator=generator) / 2000
    s2 = torch.rand((experts, inter // 256, hidden), device="cuda", generator=generator) / 2000
    inputs = [(torch.randn((tokens, hidden), device="cuda", generator=generator).to(torch.bfloat16) * (1 + i),
               torch.randn((tokens, experts), device="cuda", generator=generator)) for i in range(ROUNDS)]

    def stages(workspace):
        def call(x, logits):
            q, scale_x = quantize_rows(x)
            weights, ids = route_topk(logits, top_k)
            routes = moe.prepare_routes(ids, experts, workspace=workspace)
            qh, sh = moe.gate_up_swiglu_quantize(q, scale_x, w1, s1, routes, workspace=workspace)
            expert_out = moe.down_projection(qh, sh, w2, s2, routes, workspace=workspace)
            return (weights, ids, routes.order, routes.offsets, qh, sh, expert_out,
                    moe.combine(expert_out, weights, routes))
        return call

    _compare(_chained(inputs, stages(moe.MoEWorkspace())), _alone(inputs, stages(None)))


# The predecessor in time is on another stream: an event stands between the two, in eager calls and
# as a second dependency of the first captured kernel.
@pytest.mark.parametrize("captured", [False, True])
def test_operands_written_on_another_stream(captured):
    from grain_gemm_b200 import int8_gemm, quantize_rows
    rows, n, k = 200, 1056, 2304
    generator = torch.Generator(device="cuda").manual_seed(5)
    b = _weights((n, k), generator).t()
    scale_b = torch.rand((k // 256, n), device="cuda", generator=generator)
    inputs = [torch.randn((rows, k), device="cuda", generator=generator) * (1 + i) for i in range(8)]
    big = torch.randn((4096, 4096), device="cuda", generator=generator)
    x, source, early = torch.empty_like(inputs[0]), torch.empty_like(inputs[0]), torch.empty_like(inputs[0])
    main, side = torch.cuda.Stream(), torch.cuda.Stream()

    def step():
        side.wait_stream(main)
        quantize_rows(early)                       # a kernel of this package right before the join
        with torch.cuda.stream(side):
            product = big @ big                    # keeps the side stream busy for a while
            torch.add(source, product[0, 0] * 0, out=x)
        main.wait_stream(side)
        q, scale = quantize_rows(x)
        return q, scale, int8_gemm(q, b, scale, scale_b)

    expected = []
    for value in inputs:
        q, scale = quantize_rows(value)
        expected.append([q, scale, int8_gemm(q, b, scale, scale_b)])
    early.copy_(inputs[0])
    source.copy_(inputs[0])
    torch.cuda.synchronize()
    results = []
    with torch.cuda.stream(main):
        step()
        main.synchronize()
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=main):
                outputs = step()
        for value in inputs:
            source.copy_(value)
            if captured:
                graph.replay()
            results.append([t.clone() for t in (outputs if captured else step())])
    torch.cuda.synchronize()
    _compare(results, expected)
