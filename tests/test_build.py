"""What the build records and what the loader refuses: the library by its sources, the host path by
the torch and Python it was compiled against."""

import json

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
