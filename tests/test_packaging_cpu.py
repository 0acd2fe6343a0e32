"""What a container image, a wheel and an installed package need to build and load the native code."""
import ctypes
import os
import re

import pytest

from fastfold_b200 import _build
from fastfold_b200.ops import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_container_image_has_the_headers_of_the_extension_module():
    """csrc/host includes torch/extension.h and with it Python.h, which Debian-style images ship in python3-dev."""
    with open(os.path.join(ROOT, "docker", "Dockerfile")) as fh:
        installed = re.search(r"apt-get install (.*?)&& rm", fh.read(), re.S).group(1).split()
    assert "python3-dev" in installed


def _distribution():
    import setuptools  # noqa: F401  (brings distutils)
    from distutils.core import run_setup
    cwd = os.getcwd()
    os.chdir(ROOT)
    try:
        return run_setup("setup.py", stop_after="init")
    finally:
        os.chdir(cwd)


def test_wheel_carries_every_native_source():
    """An installed package rebuilds from, and checks its libraries against, the sources it carries."""
    from glob import glob
    package = os.path.join(ROOT, "fastfold_b200")
    carried = {os.path.realpath(f) for g in _distribution().package_data["fastfold_b200"] for f in glob(os.path.join(package, g))}
    sources = {os.path.realpath(f) for ext in ("cu", "cuh", "h", "cpp") for f in glob(os.path.join(package, "csrc", "**", "*." + ext), recursive=True)}
    assert sources and sources <= carried, sources - carried


def test_wheel_is_tagged_for_one_interpreter_and_platform():
    assert _distribution().has_ext_modules()


@pytest.fixture
def built(tmp_path, monkeypatch):
    """A library folder with both files and their stamps, and nothing loaded yet; loading or building is recorded."""
    for name in (_build.LIBNAME, _build.DISPATCH + ".so"):
        (tmp_path / name).write_bytes(b"not a library")
    monkeypatch.setattr(_build, "LIBDIR", str(tmp_path))
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "_native", None)
    (tmp_path / "build.stamp").write_text(_build._digest())
    (tmp_path / "dispatch.stamp").write_text(_build._dispatch_digest())
    calls = []
    monkeypatch.setattr(_build, "build", lambda **kw: calls.append("build"))
    monkeypatch.setattr(ctypes, "CDLL", lambda path: calls.append("load") or object())
    return tmp_path, calls


def test_current_files_are_loaded_as_they_are(built):
    _lib.get()
    assert built[1] == ["load"]


@pytest.mark.parametrize("spoil", ["build.stamp", "dispatch.stamp", _build.LIBNAME, _build.DISPATCH + ".so"])
def test_stale_or_missing_files_are_rebuilt_before_anything_is_loaded(built, spoil):
    folder, calls = built
    if spoil.endswith("stamp"):
        (folder / spoil).write_text("built from something else")
    else:
        (folder / spoil).unlink()
    _lib.get()
    assert calls == ["build", "load"]


def test_another_pytorch_makes_the_extension_module_stale(built, monkeypatch):
    import torch
    monkeypatch.setattr(torch, "__version__", "1.0")
    assert "another PyTorch" in _build.stale() and _build.DISPATCH in _build.stale()


def test_files_without_stamps_are_taken_as_they_are(built):
    folder, calls = built
    (folder / "build.stamp").unlink()
    (folder / "dispatch.stamp").unlink()
    _lib.get()
    assert calls == ["load"]


def test_a_stale_file_that_cannot_be_rebuilt_is_an_error(built, monkeypatch):
    folder, calls = built
    (folder / "dispatch.stamp").write_text("built from something else")

    def fail(**kw):
        raise OSError("no compiler")
    monkeypatch.setattr(_build, "build", fail)
    with pytest.raises(RuntimeError, match="another PyTorch.*no compiler"):
        _lib.get()
    assert calls == []


def test_an_extension_module_that_does_not_load_says_what_to_do(built):
    with pytest.raises(RuntimeError, match="Rebuild it"):
        _lib.native()
    assert _lib._native is None
