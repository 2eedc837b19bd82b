"""Device buffers on slabs (dbuf.h) against a counting driver on the CPU."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "ftlm_extended_hubbard_development_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("slabs") / "slabs")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CSRC, "-I" + os.path.join(CUDA, "include"),
                    os.path.join(HERE, "native", "slabs.cpp"), "-o", out], check=True)
    return out


def _run(*args):
    return int(subprocess.run(args, check=True, capture_output=True, text=True, timeout=60).stdout)


@pytest.mark.parametrize("how", [[], ["keep"]])
def test_growing_in_small_steps_holds_a_bounded_amount(exe, how):
    """A buffer on a slab at least doubles (ensure_keep: by half), so the regions it has left
    are at most 2 (3) times the largest one, 32 MB, and slabs round up to 64 MB: below
    3 slabs and the buffer's own last allocation with its predecessor (2 x 60 MB)."""
    assert _run(exe, "grow", *how) <= (3 * 64 + 2 * 60) << 20


def test_a_small_request_does_not_need_a_whole_slab(exe):
    assert _run(exe, "full") == 1
