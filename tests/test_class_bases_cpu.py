"""The class starts of a sector's down words, read back with the stride of a class:
any number of words a class (8x4 (0, 16) has 601,080,390) on the CPU."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "ftlm_extended_hubbard_development_b200")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("strided") / "strided")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(PKG, "csrc"), "-I" + os.path.join(CUDA, "include"),
                    os.path.join(HERE, "native", "strided.cpp"), "-o", out], check=True)
    return out


@pytest.mark.parametrize("stride", [1, 12870, (1 << 28) - 1, 1 << 28, 601080390])
@pytest.mark.parametrize("count", [0, 1, 7])
def test_class_starts_of_any_class_size(exe, stride, count):
    out = subprocess.run([exe, str(stride), str(count)], check=True, capture_output=True, text=True, timeout=60)
    assert int(out.stdout) == 0
