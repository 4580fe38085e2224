"""What the build records and what the loader refuses: the library by its sources, the host path by
the torch and Python it was compiled against."""

import json
import subprocess

import pytest
import torch

from grain_gemm_b200 import _loader, build


@pytest.fixture
def loader():
    """Both parts built, and nothing cached from one state of the files to the next."""
    build.build_library()

    def clear():
        _loader.library.cache_clear()
        _loader.host.cache_clear()

    clear()
    yield clear
    clear()


@pytest.fixture
def elsewhere(tmp_path, monkeypatch, loader):
    """The built files' places in an empty folder."""
    for name in ("LIBRARY", "HOST_MODULE", "MANIFEST"):
        monkeypatch.setattr(build, name, tmp_path / getattr(build, name).name)
    monkeypatch.setattr(build, "PACKAGE", tmp_path)
    return tmp_path


def test_the_host_path_records_what_it_was_built_for(loader):
    recorded = json.loads(build.MANIFEST.read_text())["host_module"]
    assert recorded["torch"] == str(torch.__version__) and recorded["flags"] == build.HOST_FLAGS
    assert recorded == build.host_environment()
    assert build.is_current() and build.host_module_is_current()
    assert _loader.is_available()


@pytest.mark.parametrize("key,value", [("torch", "1.0.0"), ("cuda", "1.0"), ("python", "cpython-30"),
                                       ("cxx11_abi", None), ("flags", ["-O0"])])
def test_a_host_path_for_another_torch_or_python_is_refused(loader, tmp_path, monkeypatch, key, value):
    recorded = json.loads(build.MANIFEST.read_text())
    recorded["host_module"] = {**(recorded.get("host_module") or {}), key: value}
    altered = tmp_path / "build.json"
    altered.write_text(json.dumps(recorded))
    monkeypatch.setattr(build, "MANIFEST", altered)
    with pytest.raises(RuntimeError, match=f"{key} .*rebuild with `python -m grain_gemm_b200.build`"):
        _loader.host()
    assert not _loader.is_available()
    assert _loader.library().gg_abi_version() == build.ABI_VERSION    # the C ABI does not depend on it


def test_a_host_path_that_does_not_load_is_refused(loader, tmp_path, monkeypatch):
    broken = tmp_path / "_host.so"
    broken.write_bytes(b"not a shared object")
    monkeypatch.setattr(build, "HOST_MODULE", broken)
    with pytest.raises(RuntimeError, match="does not load .*rebuild"):
        _loader.host()
    assert not _loader.is_available()


def _fake_nvcc(monkeypatch):
    commands = []

    def run(command, **kwargs):
        commands.append(command)
        output = command[command.index("-o") + 1]
        open(output, "wb").close()
        return subprocess.CompletedProcess(command, 0, "", "")

    monkeypatch.setattr(build.subprocess, "run", run)
    monkeypatch.setattr(build, "find_nvcc", lambda: "/usr/local/cuda/bin/nvcc")
    return commands


def test_the_library_is_built_where_the_host_path_cannot_be(elsewhere, monkeypatch):
    commands = _fake_nvcc(monkeypatch)

    def without_headers(output):
        raise RuntimeError("no such file: ATen/ATen.h")

    monkeypatch.setattr(build, "_build_host_module", without_headers)
    with pytest.raises(RuntimeError, match="libgrain_b200.so is built.*ATen.h.*--library-only"):
        build.build_library()
    assert build.is_current() and not build.host_module_is_current() and not build.library_only()
    assert len(commands) == 1
    build.build_library(host_module=False)
    assert len(commands) == 1                      # the library was already there
    assert build.is_current() and build.library_only()


def test_only_the_part_that_is_out_of_date_is_built(elsewhere, monkeypatch):
    commands = _fake_nvcc(monkeypatch)
    build.build_library()
    assert len(commands) == 2 and build.host_module_is_current()
    build.build_library()
    assert len(commands) == 2
    recorded = build.manifest()
    recorded["host_module"]["torch"] = "1.0.0"
    build.MANIFEST.write_text(json.dumps(recorded))
    build.build_library()
    assert len(commands) == 3 and commands[2][-1] == "-ltorch_python"
    assert build.host_module_is_current()


def test_without_the_host_path_every_call_takes_the_python_path(loader, tmp_path, monkeypatch):
    recorded = {**json.loads(build.MANIFEST.read_text()), "host_module": False}
    altered = tmp_path / "build.json"
    altered.write_text(json.dumps(recorded))
    monkeypatch.setattr(build, "MANIFEST", altered)
    assert _loader.is_available()
    host = _loader.host()
    assert host.int8_gemm(1, 2, 3) is None and host.quantize_rows(1, 2) is None
    assert host.route_topk_routes(1) is None and host.moe_ffn() is None
