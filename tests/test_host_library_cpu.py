"""The C++ host side of eager calls is a short cut: without one that fits the installed PyTorch the Python path serves
every call, and the kernel library alone is enough."""
import os
import warnings

import pytest
import torch

from parallax_b200 import _cabi, build, ops
from parallax_b200._paths import host_path


@pytest.fixture
def fresh(monkeypatch):
    _cabi.lib()
    monkeypatch.setattr(_cabi, "_host", None)
    return monkeypatch


def said_once():
    with pytest.warns(RuntimeWarning, match="Python path"):
        assert ops.eager_host() is None
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert ops.eager_host() is None


def test_a_built_module_is_used(fresh):
    assert ops.eager_host() is not None


@pytest.mark.parametrize("content", [None, b"not a library"])
def test_without_a_module_that_loads(fresh, tmp_path, content):
    path = tmp_path / "_plx_host.so"
    if content is not None:
        path.write_bytes(content)
    fresh.setattr(_cabi, "host_path", lambda: str(path))
    said_once()


def test_a_module_of_another_abi_version(fresh):
    fresh.setattr(_cabi, "ABI_VERSION", _cabi.ABI_VERSION + 1)
    said_once()


def test_another_pytorch_asks_for_another_module(fresh):
    assert os.path.exists(host_path())
    fresh.setattr(torch, "__version__", "9.9.9")
    assert not os.path.exists(host_path()) and build.is_stale()
    said_once()


def test_the_kernels_are_built_before_the_host_side(fresh):
    done = []
    fresh.setattr(build, "_build_library", lambda verbose: done.append("library"))
    fresh.setattr(build, "_build_host", lambda: done.append("host"))
    build.build(force=True)
    assert done == ["library", "host"]


def test_argument_errors_come_before_a_missing_library(monkeypatch):
    import parallax_b200 as plx

    monkeypatch.setattr(_cabi, "_lib", None)
    monkeypatch.setattr(_cabi, "_host", None)
    monkeypatch.setattr(_cabi, "LIB_PATH", "/nonexistent/libplx_sm100.so")
    x = torch.zeros(1, 1, 8, 64)
    with pytest.raises(TypeError, match="bf16 or fp16"):
        plx.parallax_func(x, x, x, x)
    with pytest.raises(TypeError, match="bf16 or fp16"):
        plx.parallax_decode(x, x, x, x)
    with pytest.raises(ValueError, match="single query"):
        plx.parallax_decode(*[torch.zeros(1, 2, 8, 64, dtype=torch.bfloat16)] * 4)
    with pytest.raises(RuntimeError, match="is missing"):
        _cabi.lib()
