"""What a container image, a wheel and an installed package need to build and load the native code."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_container_image_has_the_headers_of_the_extension_module():
    """csrc/host includes torch/extension.h and with it Python.h, which Debian-style images ship in python3-dev."""
    with open(os.path.join(ROOT, "docker", "Dockerfile")) as fh:
        installed = re.search(r"apt-get install (.*?)&& rm", fh.read(), re.S).group(1).split()
    assert "python3-dev" in installed


def _distribution():
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
