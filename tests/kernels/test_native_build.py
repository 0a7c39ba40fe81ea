"""The C++ binding belongs to one torch and one interpreter: what the build and the loader make of another one, or of none. No GPU."""

import subprocess

import pytest
import torch

from nanonemo_b200.csrc import build
from nanonemo_b200.ops import _lib


def test_the_binding_is_built_again_for_another_torch(monkeypatch, tmp_path):
    runs = []

    def compiler(cmd, **_):
        runs.append(cmd)
        (tmp_path / "_native.so").write_text("")
        return subprocess.CompletedProcess(cmd, 0, "", "")

    (tmp_path / "binding.cpp").write_text("")
    monkeypatch.setattr(build, "HERE", tmp_path)
    monkeypatch.setattr(build, "NATIVE", tmp_path / "_native.so")
    monkeypatch.setattr(build.subprocess, "run", compiler)
    build.build_native()
    build.build_native()
    assert len(runs) == 1
    monkeypatch.setattr(torch, "__version__", "0.0.0")
    build.build_native()
    build.build_native()
    assert len(runs) == 2


def test_a_binding_that_does_not_load_says_how_to_build_it(monkeypatch):
    if not build.LIB.exists():
        pytest.skip("kernel library not built")
    real = _lib.importlib.import_module

    def broken(name, *a):
        if name.endswith("._native"):
            raise ImportError("undefined symbol")
        return real(name, *a)

    monkeypatch.setattr(_lib.importlib, "import_module", broken)
    _lib.native.cache_clear()
    try:
        with pytest.raises(RuntimeError, match="undefined symbol.*nanonemo_b200.csrc.build"):
            _lib.native()
    finally:
        _lib.native.cache_clear()
