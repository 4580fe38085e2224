"""A call that fails leaves nothing behind: the next good call succeeds.

The CUDA runtime keeps the error of a failed call for the thread until somebody asks for it.  Here a
launch is refused by the runtime, on the host, because its stream's capture has been invalidated
(a wait for the stream inside the capture does that); the same call on another stream must then
report its own success and not the old error.
"""

import ctypes
from contextlib import contextmanager

import pytest
import torch

pytestmark = pytest.mark.gpu

RELAXED = 2                       # cudaStreamCaptureModeRelaxed


@contextmanager
def refusing_stream():
    runtime = ctypes.CDLL("libcudart.so.12")
    stream = torch.cuda.Stream()
    raw = ctypes.c_void_p(stream.cuda_stream)
    torch.cuda.synchronize()
    assert runtime.cudaStreamBeginCapture(raw, RELAXED) == 0
    try:
        assert runtime.cudaStreamSynchronize(raw) != 0
        runtime.cudaGetLastError()       # of the runtime that torch uses; the library has its own
        yield stream
    finally:
        graph = ctypes.c_void_p()
        assert runtime.cudaStreamEndCapture(raw, ctypes.byref(graph)) != 0 and not graph.value
        runtime.cudaGetLastError()


def _gemm(m, n, k, variant):
    from grain_gemm_b200 import int8_gemm
    generator = torch.Generator(device="cuda").manual_seed(1)
    a = torch.randint(-127, 128, (m, k), dtype=torch.int8, device="cuda", generator=generator)
    b = torch.randint(-127, 128, (n, k), dtype=torch.int8, device="cuda", generator=generator).t()
    sa, sb = torch.rand((m, k // 256), device="cuda"), torch.rand((k // 256, n), device="cuda")
    return lambda: int8_gemm(a, b, sa, sb, variant=variant)


def _quantize():
    from grain_gemm_b200 import quantize_rows
    x = torch.randn((5, 512), device="cuda")
    return lambda: quantize_rows(x)[0]


def _topk(fused):
    from grain_gemm_b200 import route_topk, route_topk_routes
    logits = torch.randn((9, 16), device="cuda")
    return lambda: (route_topk_routes if fused else route_topk)(logits, 4)[0]


def _route(tokens, experts):
    from grain_gemm_b200 import moe
    ids = torch.randint(0, experts, (tokens, 2), device="cuda")
    return lambda: moe.prepare_routes(ids, experts).offsets


def _stage(name, tokens, experts, tile_rows=128, row_gather=False):
    from grain_gemm_b200 import moe, quantize_rows
    hidden, inter = 512, 256
    x, sx = quantize_rows(torch.randn((tokens, hidden), device="cuda"))
    w1 = torch.randint(-127, 128, (experts, 2 * inter, hidden), dtype=torch.int8, device="cuda")
    w2 = torch.randint(-127, 128, (experts, hidden, inter), dtype=torch.int8, device="cuda")
    s1 = torch.rand((experts, hidden // 256, 2 * inter), device="cuda") / 1000
    s2 = torch.rand((experts, inter // 256, hidden), device="cuda")
    ids = torch.randint(0, experts, (tokens, 2), device="cuda")
    weights = torch.rand((tokens, 2), device="cuda")
    routes = moe.prepare_routes(ids, experts, tile_rows=tile_rows)
    gate_up = lambda: moe.gate_up_swiglu_quantize(x, sx, w1, s1, routes, row_gather=row_gather)  # noqa: E731
    valid = tokens * 2
    if name == "gate_up":
        return lambda: gate_up()[0][:valid]
    qh, sh = gate_up()
    down = lambda: moe.down_projection(qh, sh, w2, s2, routes)   # noqa: E731
    if name == "down":
        return lambda: down()[:valid]
    rows = down()
    return lambda: moe.combine(rows, weights, routes)


CALLS = {
    "gemv": lambda: _gemm(1, 512, 512, "gemv"),
    "split_k": lambda: _gemm(9, 512, 512, "tc_splitk"),
    "single_ctas": lambda: _gemm(130, 512, 512, "tc_n64"),
    "cta_pairs": lambda: _gemm(300, 512, 512, "tc_pair_n256"),
    "cuda_cores": lambda: _gemm(9, 64, 512, "simt"),
    "quantize": _quantize,
    "topk": lambda: _topk(False),
    "topk_and_route": lambda: _topk(True),
    "route_one_cta": lambda: _route(100, 8),
    "route_medium": lambda: _route(1000, 8),
    "route_three_kernels": lambda: _route(6000, 8),
    "gate_up_pairs": lambda: _stage("gate_up", 8, 4),
    "gate_up_single": lambda: _stage("gate_up", 6272, 4),
    "gate_up_row_gather": lambda: _stage("gate_up", 8, 4, row_gather=True),
    "gate_up_cuda_cores": lambda: _stage("gate_up", 8, 4, tile_rows=32),
    "down": lambda: _stage("down", 8, 4),
    "combine": lambda: _stage("combine", 8, 4),
}


@pytest.mark.parametrize("name", CALLS)
def test_the_call_after_a_refused_launch_succeeds(name):
    call = CALLS[name]()
    expected = call()
    with refusing_stream() as stream:
        with torch.cuda.stream(stream), pytest.raises(RuntimeError, match=r"failed: .*\(status \d+\)"):
            call()
    assert torch.equal(call(), expected)
    torch.cuda.synchronize()


def test_the_status_is_not_handed_on_to_another_entry_point():
    call = _quantize()
    with refusing_stream() as stream:
        with torch.cuda.stream(stream), pytest.raises(RuntimeError):
            call()
    for name in ("topk", "split_k", "cta_pairs", "gate_up_pairs", "gate_up_cuda_cores", "route_three_kernels"):
        CALLS[name]()()
    torch.cuda.synchronize()
