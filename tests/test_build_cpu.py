"""What the build asks of a machine: nothing where the binaries are current, no torch for the C library."""
import importlib.util
import os
import shutil

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture
def build():
    spec = importlib.util.spec_from_file_location("_build_under_test", os.path.join(ROOT, "inference.rs_b200", "build.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def no_toolkit():
    raise RuntimeError("nvcc not found")


def test_current_binaries_are_used_without_a_toolkit(build, monkeypatch):
    build.build()  # whatever is not current
    monkeypatch.setattr(build, "_nvcc", no_toolkit)
    assert build.build() == build.LIB and build.build_host() == build.HOST_LIB


def test_the_library_comes_first_and_needs_no_torch(build, monkeypatch):
    calls = []
    monkeypatch.setattr(build, "build_library", lambda *a: calls.append("library") or build.LIB)
    find = importlib.util.find_spec
    monkeypatch.setattr(importlib.util, "find_spec", lambda name, *a: None if name == "torch" else find(name, *a))
    assert build.build_host(force=True) is None
    assert build.build(force=True) == build.LIB and calls == ["library"]
    monkeypatch.setattr(build, "build_host", lambda *a: calls.append("host"))
    build.build()
    assert calls == ["library", "library", "host"]


def test_a_machine_that_cannot_compile_extensions_builds_the_library(build, monkeypatch, tmp_path):
    monkeypatch.setattr(build, "HOST_LIB", str(tmp_path / "host.so"))
    monkeypatch.setattr(shutil, "which", lambda name: None)
    assert build.build_host() is None
