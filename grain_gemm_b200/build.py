"""Build ``libgrain_b200.so`` (nvcc, sm_100a) and ``_host.so`` (g++, the native host path of the
public calls, against this interpreter's torch) and record what they were built from.

Both are built in-tree, next to this file, together with ``build.json`` (compiler
target, ABI version, the SHA-256 of every source file and, for the host path, the torch and
Python it was compiled against).  The loader refuses a library whose manifest does not match
the sources beside it, the same provenance rule as the reference's native bridges
(``src/grain_gemm/kernels/moe_gather.py:29-55`` there), and a host path built for another torch
or Python than the running one.

The library does not depend on the host path.  ``--library-only`` builds it alone, for a binding
of the C ABI or where torch's headers or a C++ compiler for them are missing; the public
Python functions then run all calls through their Python path.

    python -m grain_gemm_b200.build [--library-only] [--force] [--verbose]
"""

from __future__ import annotations

import hashlib
import json
import os
import shutil
import subprocess
import sys
import sysconfig
import tempfile
from pathlib import Path

PACKAGE = Path(__file__).resolve().parent
CSRC = PACKAGE / "csrc"
HEADER = PACKAGE.parent / "include" / "grain_gemm_b200.h"
LIBRARY = PACKAGE / "libgrain_b200.so"
HOST_MODULE = PACKAGE / "_host.so"
MANIFEST = PACKAGE / "build.json"
ABI_VERSION = 4
ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-O3", "-std=c++17", "-lineinfo", "--expt-relaxed-constexpr",
         "-Xcompiler", "-fPIC", "-shared"]
HOST_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared"]


def sources():
    return (sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.cpp"))
            + [HEADER])


def source_hashes():
    return {path.name: hashlib.sha256(path.read_bytes()).hexdigest() for path in sources()}


def find_nvcc():
    candidates = [os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"]
    for candidate in candidates:
        if candidate and Path(candidate).exists():
            return candidate
    raise RuntimeError("nvcc not found; set NVCC or add the CUDA toolkit to PATH")


def manifest():
    """What is recorded about the built files; empty when nothing readable is."""
    try:
        recorded = json.loads(MANIFEST.read_text())
    except (OSError, ValueError):
        return {}
    return recorded if isinstance(recorded, dict) else {}


def is_current():
    """Whether the library was built from the sources beside it."""
    recorded = manifest()
    return (LIBRARY.is_file() and recorded.get("abi_version") == ABI_VERSION
            and recorded.get("source_sha256") == source_hashes())


def host_environment():
    """What the host path's machine code depends on besides its source: it uses the layouts and
    inline functions of torch's headers and Python's C API."""
    import torch
    return {"torch": str(torch.__version__), "torch_git": torch.version.git_version,
            "cuda": torch.version.cuda, "python": sysconfig.get_config_var("SOABI"),
            "cxx11_abi": bool(torch._C._GLIBCXX_USE_CXX11_ABI), "flags": HOST_FLAGS}


def host_module_is_current():
    """Whether the host path was built from these sources, for this torch and this Python."""
    return (HOST_MODULE.is_file() and is_current()
            and manifest().get("host_module") == host_environment())


def library_only():
    """Whether the build was asked to leave the host path out."""
    return manifest().get("host_module") is False


def _build_host_module(output):
    """Compile the native host path against the torch of this interpreter."""
    import torch
    root = Path(torch.__file__).resolve().parent
    nvcc_root = Path(find_nvcc()).resolve().parents[1]
    include = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include",
               nvcc_root / "include", sysconfig.get_paths()["include"]]
    libraries = ["c10", "c10_cuda", "torch_cpu", "torch_cuda", "torch", "torch_python"]
    command = [os.environ.get("CXX", "g++"), *HOST_FLAGS, *(f"-I{path}" for path in include),
               f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
               "-o", str(output), str(CSRC / "host.cpp"), f"-L{root / 'lib'}",
               *(f"-l{name}" for name in libraries)]
    result = subprocess.run(command, capture_output=True, text=True)
    if result.returncode != 0:
        raise RuntimeError(f"{command[0]} failed:\n{result.stdout}\n{result.stderr}")


def _build_library(verbose):
    """Compile the library, put it in place and record it, without a host path so far."""
    nvcc = find_nvcc()
    with tempfile.TemporaryDirectory(dir=PACKAGE) as scratch:
        output = Path(scratch) / LIBRARY.name
        command = [nvcc, *ARCH_FLAGS, *FLAGS, "-o", str(output), str(CSRC / "abi.cu")]
        if verbose:
            command.insert(1, "-Xptxas=-v")
        result = subprocess.run(command, capture_output=True, text=True)
        if result.returncode != 0:
            raise RuntimeError(f"nvcc failed:\n{result.stdout}\n{result.stderr}")
        if verbose:
            print(result.stderr)
        os.replace(output, LIBRARY)
    _record({
        "architecture": "sm_100",
        "compiler_architecture": "sm_100a",
        "abi_version": ABI_VERSION,
        "flags": ARCH_FLAGS + FLAGS,
        "source_sha256": source_hashes(),
    })


def _record(values):
    MANIFEST.write_text(json.dumps(values, indent=1) + "\n")


def build_library(force=False, verbose=False, host_module=True):
    """Compile the library and the host path unless up-to-date ones are already in place.

    ``host_module=False`` leaves the host path out.  When only the host path cannot be built the
    library is in place all the same, and the error says so."""
    if force or not is_current():
        _build_library(verbose)
    if not host_module:
        if not library_only():
            _record({**manifest(), "host_module": False})
            HOST_MODULE.unlink(missing_ok=True)
        return LIBRARY
    if force or not host_module_is_current():
        with tempfile.TemporaryDirectory(dir=PACKAGE) as scratch:
            output = Path(scratch) / HOST_MODULE.name
            try:
                _build_host_module(output)
            except Exception as error:
                raise RuntimeError(
                    f"{LIBRARY.name} is built, the native host path is not ({error}); "
                    "`python -m grain_gemm_b200.build --library-only` does without it") from error
            os.replace(output, HOST_MODULE)
        _record({**manifest(), "host_module": host_environment()})
    return LIBRARY


if __name__ == "__main__":
    build_library(force="--force" in sys.argv, verbose="--verbose" in sys.argv,
                  host_module="--library-only" not in sys.argv)
    print(LIBRARY)
