"""GrainGEMM's two hot paths on NVIDIA B200: ``int8_gemm`` and ``moe_ffn``.

The public names match the reference package (``src/grain_gemm/__init__.py:4`` there);
attributes are resolved lazily so that importing the package does not import torch.
"""

__version__ = "0.1.0"
__all__ = ["__version__", "get_kernel_config", "int8_gemm", "moe_ffn", "quantize_rows",
           "prepare_weight", "interleave_gate_up", "route_topk", "route_topk_routes"]


def __getattr__(name):
    if name in ("int8_gemm", "get_kernel_config"):
        from . import gemm as module
    elif name == "moe_ffn":
        from . import moe as module
    elif name in ("quantize_rows", "prepare_weight", "interleave_gate_up", "route_topk",
                  "route_topk_routes"):
        from . import quantize as module
    else:
        raise AttributeError(f"module 'grain_gemm_b200' has no attribute '{name}'")
    value = globals()[name] = getattr(module, name)   # found directly from the next use on
    return value
