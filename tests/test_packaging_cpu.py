"""What a container image, a wheel and an installed package need to build and load the native code."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_container_image_has_the_headers_of_the_extension_module():
    """csrc/host includes torch/extension.h and with it Python.h, which Debian-style images ship in python3-dev."""
    with open(os.path.join(ROOT, "docker", "Dockerfile")) as fh:
        installed = re.search(r"apt-get install (.*?)&& rm", fh.read(), re.S).group(1).split()
    assert "python3-dev" in installed
