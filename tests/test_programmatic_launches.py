"""Rules that kernels launched with programmatic stream serialisation have to keep, read from the
CUDA sources.

Such a kernel may be resident before its predecessor has written the operands.  So it waits
(``previous_kernel_done``) before the first access to global memory, and nothing it executes reads
through the read-only path (``__ldg``, ``ld.global.nc``, or plain loads that ``__restrict__`` lets
the compiler turn into them): that path is defined only for memory that stays constant from the
kernel's start to its end, and the wait does not order it.
"""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "grain_gemm_b200" / "csrc"
READ_ONLY = re.compile(r"__restrict__|__ldg\s*\(|__ldlu\s*\(|ld\.global(?:\.\w+)*\.nc")


def _without_comments(text):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def _functions(text):
    """``{name: declaration and body}`` of the device functions and kernels of a source file."""
    found = {}
    for match in re.finditer(r"__(?:global|device)__[^;{}]*?\b(\w+)\s*\(((?:[^()]|\([^()]*\))*)\)\s*\{", text):
        name = match.group(1)
        depth, end = 1, match.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        found[name] = text[match.start():end]
    return found


def _sources():
    return _without_comments("\n".join(path.read_text() for path in sorted(CSRC.glob("*.cu*"))))


TEXT = _sources()
FUNCTIONS = _functions(TEXT)
KERNELS = {name for name, code in FUNCTIONS.items() if code.startswith("__global__")}


def _programmatic():
    """Kernels handed to ``launch`` (directly or through a local variable) or launched with the
    attribute by ``launch_tc_kernel``, whose plain form takes it and whose grouped form does not."""
    names = set(re.findall(r"\blaunch\((?:gg::)?(\w+_kernel)\b", TEXT))
    return names | {"gemm_gemv_kernel", "gemm_tc_kernel"}


def _reached(name):
    seen, waiting = set(), [name]
    while waiting:
        current = waiting.pop()
        if current not in seen:
            seen.add(current)
            waiting += [other for other in FUNCTIONS if re.search(rf"\b{other}\b\s*[<(]", FUNCTIONS[current])]
    return seen


def test_sources_were_understood():
    assert {"quantize_rows_kernel", "combine_kernel", "gather_rows_kernel", "fold_partials_kernel",
            "moe_tiles_kernel", "route_medium_kernel", "gemm_tc_kernel", "gemm_gemv_kernel"} <= _programmatic()
    assert _programmatic() <= KERNELS
    assert "gemv_step" in _reached("gemm_gemv_kernel") and "router_topk_token" in _reached("router_topk_kernel")
    # Every kernel that waits is one of them, and the attribute is set nowhere else.
    waiting = {name for name in KERNELS if "previous_kernel_done();" in FUNCTIONS[name]}
    assert waiting == _programmatic()
    assert TEXT.count("cudaLaunchAttributeProgrammaticStreamSerialization") == 2


@pytest.mark.parametrize("name", sorted(_programmatic()))
def test_the_wait_stands_before_the_first_access(name):
    body = FUNCTIONS[name]
    before = body[body.index("{"):body.index("previous_kernel_done();")]
    before = re.sub(r"extern __shared__ [^;]*;", "", before)
    if name == "gemm_tc_kernel":
        assert "if constexpr (!kGrouped) previous_kernel_done();" in body
        # Before the wait: shared memory, barriers, tensor-map prefetch; the row-tile list only where
        # the launch is an ordinary one.
        before = re.sub(r"if constexpr \(kGrouped\) \{.*?\n  \}", "", before, flags=re.S)
        assert not re.search(r"\bp\.\w+\[|__ldg|tma_load|cp_async", before)
    else:
        assert not re.search(r"\[|\*\s*reinterpret_cast|__ldg|ldg_|ld_", before)


@pytest.mark.parametrize("name", sorted(_programmatic()))
def test_no_read_only_loads_behind_the_wait(name):
    for function in sorted(_reached(name)):
        code = FUNCTIONS[function]
        if function == "gemm_tc_kernel":
            # Destination addresses exist in the grouped form only, whose launch is an ordinary one.
            code = re.sub(r"__ldg\(p\.row_destination \+ \w+\)", "", code)
        assert not READ_ONLY.search(code), f"{function} reads through the read-only path"


def test_the_grouped_form_is_launched_without_the_attribute():
    assert re.search(r"config\.numAttrs = kGrouped \? 1 : 2;", TEXT)
    order = re.findall(r"attribute\[(\d)\]\.id = (\w+);", TEXT[TEXT.index("static int launch_tc_kernel"):])[:2]
    assert order == [("0", "cudaLaunchAttributeClusterDimension"),
                     ("1", "cudaLaunchAttributeProgrammaticStreamSerialization")]
