"""The native host path is used with the Python, the torch and the argument blocks that it was built for, or not at all."""
import importlib.util
import os
import runpy
import struct
import sysconfig

import pytest
import torch

from conftest import PKG

ext = pytest.importorskip("flash_attn_legacy_cuda")


@pytest.fixture()
def build():
    spec = importlib.util.spec_from_file_location("fal_b200_build_h", os.path.join(PKG, "build.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


@pytest.fixture()
def built(build):
    if build.build_host() is None:
        pytest.skip("no compiler or headers for the host path")
    assert ext._load_host() is not None


def test_a_file_of_another_torch_or_python_is_not_loaded(built, monkeypatch):
    with monkeypatch.context() as mp:
        mp.setattr(torch, "__version__", "0.0.0")
        assert ext._load_host() is None
    with monkeypatch.context() as mp:
        get = sysconfig.get_config_var
        mp.setattr(sysconfig, "get_config_var", lambda name: "cpython-399" if name == "SOABI" else get(name))
        assert ext._load_host() is None
    assert ext._load_host() is not None


@pytest.mark.parametrize("block", ["_FWD_ARGS", "_DECODE_ARGS"])
def test_a_file_of_other_argument_blocks_is_not_used(built, monkeypatch, block):
    monkeypatch.setattr(ext, block, struct.Struct(getattr(ext, block).format + "Q"))
    assert ext._load_host() is None


@pytest.mark.parametrize("compiler", ["false", "/nonexistent"])
def test_a_file_of_older_sources_goes_when_it_cannot_be_built_again(build, monkeypatch, tmp_path, compiler):
    monkeypatch.setattr(build, "LIB_DIR", str(tmp_path))
    monkeypatch.setenv("CXX", compiler)
    assert build.build_host() is None and not list(tmp_path.iterdir())
    old = tmp_path / os.path.basename(runpy.run_path(os.path.join(PKG, "fal_host_file.py"))["host_path"](""))
    old.write_bytes(b"")
    assert build.build_host() == str(old)  # newer than its sources: taken as it is
    assert build.build_host(force=True) is None and old.exists()
    os.utime(old, (0, 0))
    assert build.build_host() is None and not list(tmp_path.iterdir())

